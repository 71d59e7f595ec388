"""Device bond hand-off against the host hand-off, whose lists leave the held pairs out, at each
number of lanes while no bond fails, and at one lane across failures with a change of the precision
form and back in between (which rounds both sides' histories alike).

Bar: bit equality.  At several lanes it holds because the block's only contacts are its bonds and
the platens: the held entries contribute nothing, wherever they fall.  All tests need a GPU.
"""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu

KEYS = ("id", "pos", "vel", "angvel", "quat", "force", "moment")


def _both(dem_lib, precision, tpp, strength):
    from esys.lsm import _capi

    sims = []
    for on in (0, 1):
        s = S.bonded_block(lambda *a: _capi.DemSim(*a), strength=strength)
        s.set_option("precision", precision)
        s.set_option("threads_per_particle", tpp)
        s.set_option("bond_handoff", on)
        sims.append(s)
    return sims


def _same(host, dev):
    ph, pd = host.particles(), dev.particles()
    for k in KEYS:
        assert np.array_equal(ph[k], pd[k]), k


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("tpp", [1, 2, 4, 8])
def test_no_failures_equal_host_handoff(dem_lib, precision, tpp):
    host, dev = _both(dem_lib, precision, tpp, (1e9, 1e9, 1e9, 1e9))
    for s in (host, dev):
        S.run_loaded(s, 60, 0.002)
        assert len(s.breaks()[0]) == 0
    _same(host, dev)


@pytest.mark.parametrize("precision", [64, 32])
def test_change_of_form_between_failures(dem_lib, precision):
    host, dev = _both(dem_lib, precision, 1, (0.3, 0.6, 0.6, 0.3))
    for s in (host, dev):
        S.run_loaded(s, 100, 0.002)
        s.set_option("precision", 96 - precision)
        s.step(3)
        s.set_option("precision", precision)
        S.run_loaded(s, 50, 0.002)
    assert len(host.breaks()[0]) > 0
    for u, v in zip(host.breaks(), dev.breaks()):
        assert np.array_equal(u, v)
    _same(host, dev)
