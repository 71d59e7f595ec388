"""Order of summation of bonded specimens under the device bond hand-off.

A particle's entries of the pair list, held or free, keep their lanes whatever fails and whichever
kernel walks them, so (a) a window's recomputed steps repeat its forward's bit for bit, at every
number of lanes, (b) runs with failures repeat bit for bit also where the bonds are evaluated within
the step kernel, and (c) the automatic number of lanes is the one that the whole list's mean length
gives.  The specimen is a bonded block cut by an unbonded plane: the particles beside the cut have
contacts that no bond holds, bonds that none of them has lost, and listed pairs that bonds hold.
All tests need a GPU.
"""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "angvel", "quat")
GRAD = ("params", "vel", "angvel", "pos", "quat")


@pytest.fixture(scope="module")
def gpu(dem_lib):
    from esys.lsm import _capi

    return lambda *a: _capi.DemSim(*a)


def _cut_block(gpu, lanes, strength=3000.0, n=(6, 8, 6)):
    """window_block's law and loading on a jittered lattice in contact, unbonded across two planes."""
    rng = np.random.default_rng(21)
    g = np.stack(np.meshgrid(*(np.arange(k) for k in n), indexing="ij"), -1).reshape(-1, 3)
    pos = g * 0.97 + rng.uniform(-0.02, 0.02, size=g.shape) + 1.0
    rad = rng.uniform(0.48, 0.5, size=len(g))
    d = np.linalg.norm(pos[:, None] - pos[None], axis=-1)
    np.fill_diagonal(d, np.inf)
    i, j = np.nonzero(np.triu(d - rad[:, None] - rad[None] <= 0.03, 1))
    same = ((g[i, 0] < n[0] // 2) == (g[j, 0] < n[0] // 2)) & ((g[i, 2] < n[2] // 2) == (g[j, 2] < n[2] // 2))
    top = pos.max(axis=0) + 1.0
    sim = gpu("RotSphere", 1.25, 0.2, (0, 0, 0), tuple(float(x) for x in top), (0, 0, 0), 1e-4)
    sim.add_particles(np.arange(len(g)), pos, rad, S.sphere_mass(rad), tag=np.zeros(len(g), np.int32),
                      vel=rng.normal(0, 1.0, size=pos.shape), angvel=rng.normal(0, 1.0, size=pos.shape))
    sim.add_connections(np.ones(same.sum(), np.int32), i[same], j[same])
    sim.add_rot_bond_group("bonds", 1, 1e5, 1e5, 1e5, 1e5, strength, strength, strength, strength, True, True, 1.0)
    sim.add_rot_friction_group("friction", 1e5, 0.6, 0.6, 1e5, 1e-4, True, True)
    sim.add_exclusion("bonds", "friction")
    sim.add_wall("bottom", (0, float((pos[:, 1] - rad).min()), 0), (0, 1, 0))
    sim.add_wall("top", (0, float((pos[:, 1] + rad).max()), 0), (0, -1, 0))
    for w in ("bottom", "top"):
        sim.add_wall_group(w + "_w", w, 1e5)
    sim.add_damping(0, 0.5, 50)
    sim.add_damping(1, 0.5, 50)
    sim.set_wall_velocity("bottom", (0, 0.2, 0))
    sim.set_wall_velocity("top", (0, -0.2, 0))
    sim.set_option("bond_handoff", 1)
    if lanes is not None:
        sim.set_option("threads_per_particle", lanes)
    return sim


def _free_contacts(sim):
    """Touching pairs between particles that have lost no bond."""
    a, b, st = sim.pairs("friction")
    lost = set(np.concatenate(sim.breaks()[:2]).tolist())
    return sum(1 for x, y, r in zip(a, b, st) if r[4] != 0 and int(x) not in lost and int(y) not in lost)


T = 60


@pytest.mark.parametrize("precision,lanes", [(64, 1), (64, 2), (64, 4), (64, 8), (64, None), (32, 2), (32, 4), (32, 8)])
def test_window_recompute_repeats_the_forward(gpu, precision, lanes):
    out = []
    for K in (1, 13, T):
        s = _cut_block(gpu, lanes)
        s.set_option("precision", precision)
        R = s.window_forward(T, K)
        out.append(s.window_adjoint(S.mse_grad(R, S.mse_target(R))))
        assert len(s.breaks()[0]) > 0 and _free_contacts(s) > 20
    for o in out[1:]:
        for k in GRAD:
            assert np.array_equal(o[k], out[0][k]), (k, np.abs(o[k] - out[0][k]).max())


def test_ensemble_window_recompute_repeats_the_forward(gpu):
    from esys.lsm import _capi

    out = []
    for K in (1, 13, T):
        e = _capi.Ensemble([_cut_block(gpu, None, n=(6, 8 + k, 6)) for k in range(2)])
        e.set_option("threads_per_particle", 4)
        R = e.window_forward(T, K)
        out.append(e.window_adjoint([S.mse_grad(r, S.mse_target(r)) for r in R]))
        e.close()
    for o in out[1:]:
        for x, y in zip(o, out[0]):
            for k in ("params", "vel", "angvel"):
                assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("lanes", [2, 4, 8])
def test_bonds_in_the_step_kernel_equal_the_bond_pass(gpu, lanes):
    """Without the bond pass the failure flags are raised by the launch that walks the lists: the
    order of a sum may not follow them.  The same bond forces in the same order either way."""
    out = []
    for bond_pass in (1, 0, 0):
        s = _cut_block(gpu, lanes)
        s.set_option("bond_pass", bond_pass)
        s.step(T)
        assert len(s.breaks()[0]) > 0
        out.append(s.particles())
    for o in out[1:]:
        for k in STATE:
            assert np.array_equal(o[k], out[0][k]), k


def test_automatic_lanes_follow_the_whole_list(gpu):
    """5.1 entries of the pair list, held ones included, and 4.4 bonds a particle: 4 lanes (6 to 12)."""
    a, b = _cut_block(gpu, None), _cut_block(gpu, 4)
    for s in (a, b):
        s.step(T)
        assert s.counters()["threads_per_particle"] == 4
    pa, pb = a.particles(), b.particles()
    for k in STATE + ("force", "moment"):
        assert np.array_equal(pa[k], pb[k]), k
