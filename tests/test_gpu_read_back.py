"""Rows read into page-locked arrays (written there by a kernel) against pageable ones (packed and
copied): equal bit for bit, whatever fields are wanted, with every particle alive or not."""
import numpy as np
import pytest

import scenarios as S
from conftest import gpu_available

pytestmark = pytest.mark.gpu

FIELDS = (("pos", 3), ("vel", 3), ("angvel", 3), ("quat", 4), ("force", 3), ("moment", 3))


@pytest.fixture(scope="module")
def gpu(dem_lib):
    if not gpu_available():
        pytest.skip("no GPU")
    from esys.lsm import _capi

    return lambda *a: _capi.DemSim(*a)


def _leaving(make):
    """A packing one of whose particles leaves the grid."""
    s = S.friction_pack(make, nx=5, ny=4, nz=5)
    v = s.particles(sort=False)["vel"]
    v[7] = (0.0, 0.0, -4e4)
    s.set_particles(vel=v)
    s.step(40)
    return s


CASES = [("one", lambda m: S.friction_pack(m, nx=1, ny=1, nz=1)), ("rot", lambda m: S.friction_pack(m, nx=7, ny=6, nz=9)),
         ("nrot", lambda m: S.gravity_box(m, n_side=8)), ("dead", _leaving),
         ("large", lambda m: S.friction_pack(m, nx=42, ny=40, nz=40))]  # beyond the rows written directly


@pytest.mark.parametrize("name,build", CASES, ids=[c[0] for c in CASES])
def test_pinned_equals_pageable(gpu, name, build):
    import torch

    s = build(gpu)
    s.step(3)
    want = s.particles(sort=False)
    n = len(want["id"])
    for skip in ((), ("id", "vel"), ("pos", "quat", "moment")):
        ids = torch.full((n + 1,), -7, dtype=torch.int32, pin_memory=True)
        out = {k: torch.full((n + 1, d), -7.0, dtype=torch.float64, pin_memory=True) for k, d in FIELDS}
        got = s.get_particles_raw(*[0 if k in skip else a.data_ptr() for k, a in (("id", ids), *out.items())])
        assert got == n
        for k, a in (("id", ids), *out.items()):
            a = a.numpy()
            if k in skip:
                assert (a == -7).all(), k
            else:
                assert np.array_equal(a[:n], want[k]) and (a[n] == -7).all(), k
    if name == "dead":
        assert n == 99


def test_rows_behind_a_header(gpu):
    """Page-locked arrays that start 4 bytes off a multiple of 8 (rows behind a message's header): a
    copy takes any address, a kernel's stores do not."""
    import torch

    s = S.friction_pack(gpu, nx=7, ny=6, nz=9)
    s.step(3)
    want = s.particles(sort=False)
    n = len(want["id"])
    bufs = {k: torch.zeros(4 + 8 * n * d, dtype=torch.uint8, pin_memory=True) for k, d in FIELDS}
    ids = torch.zeros(4 + 4 * n, dtype=torch.uint8, pin_memory=True)
    assert s.get_particles_raw(ids.data_ptr() + 4, *[b.data_ptr() + 4 for b in bufs.values()]) == n
    assert np.array_equal(np.frombuffer(ids.numpy()[4:].tobytes(), np.int32), want["id"])
    for k, d in FIELDS:
        assert np.array_equal(np.frombuffer(bufs[k].numpy()[4:].tobytes()).reshape(n, d), want[k]), k


def test_rule_of_the_rows_written_directly(gpu, dem_lib):
    """The rule alone, no launch: whole page-locked arrays only, at multiples of 8 bytes."""
    import ctypes as C

    import torch

    rule = lambda address, count: dem_lib.dem_rows_mapped(C.c_void_p(address), C.c_size_t(count))
    torch.cuda.init()
    pinned = torch.zeros(1000, dtype=torch.float64, pin_memory=True)
    at = pinned.data_ptr()
    assert rule(at, 1000) and rule(at + 8, 999)
    assert not rule(at + 4, 999)
    assert not rule(at, 1 << 24)                      # beyond the allocation, whatever it was rounded up to
    plain = np.zeros(2 * 65536 // 8)            # 64 KB of it registered
    assert not rule(plain.ctypes.data, 8)
    page = (plain.ctypes.data + 4095) // 4096 * 4096
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(page, 65536, 0)) == 0
    try:
        assert rule(page, 8192)
        assert not rule(page, 8193) and not rule(page + 65528, 2)   # the tail is pageable
        assert not rule(page - 8, 8)                                # and so is the head
        assert not rule(page + 4, 8)
    finally:
        assert int(rt.cudaHostUnregister(page)) == 0
