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
