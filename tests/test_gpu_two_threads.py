"""Two handles stepped by two host threads at once: a handle is single-threaded, several run side by
side.  Bar: no call fails, and each specimen's state equals the one it reaches when stepped alone.
All tests need a GPU.
"""
import threading

import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_small_and_large_specimen_side_by_side(dem_lib, precision):
    """Launches of one kernel with unlike shares of a block's shared memory."""
    from esys.lsm import _capi

    def build(n):
        s = S.friction_pack(lambda *a: _capi.DemSim(*a), nx=n, ny=n, nz=n)
        s.set_option("precision", precision)
        return s

    sizes, calls, failed = (3, 26), 400, []
    alone = [build(n) for n in sizes]
    for s in alone:
        for _ in range(calls):
            s.step(2)
    both = [build(n) for n in sizes]
    start = threading.Barrier(2)

    def work(s):
        try:
            start.wait(60)
            for _ in range(calls):
                s.step(2)
        except Exception as e:  # noqa: BLE001 - the error is the finding
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in both]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for a, b in zip(alone, both):
        pa, pb = a.particles(), b.particles()
        for k in ("pos", "vel", "angvel", "quat"):
            assert np.array_equal(pa[k], pb[k]), k
