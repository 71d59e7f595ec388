"""The neighbour search with several lanes per particle: the list of a pair group against all pairs
tested on the host, at particle counts on either side of its warps and of the one-block scan, with a
particle that has more neighbours than the kernel collects in shared memory, through a periodic face;
and tangential histories carried over a second search.  All tests need a GPU.
"""
import numpy as np
import pytest

import scenarios as S

pytestmark = pytest.mark.gpu

SKIN = 0.2


def _pairs(sim):
    a, b, st = sim.pairs("friction")
    return {(int(min(x, y)), int(max(x, y))): tuple(r) for x, y, r in zip(a, b, st)}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nx,ny,nz,crowd", [(1, 1, 1, 0), (2, 2, 1, 0), (5, 3, 3, 60), (4, 4, 33, 0), (21, 20, 21, 90)])
def test_list_is_every_near_pair(dem_lib, precision, nx, ny, nz, crowd):
    from esys.lsm import _capi

    rng = np.random.default_rng(11)
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5) * 1.0 + rng.uniform(-0.05, 0.05, size=g.shape)
    rad = rng.uniform(0.4, 0.5, size=len(g))
    if crowd:  # small particles around one point: each the other's neighbour
        pos = np.concatenate([pos, np.array([0.9, 1.0, 1.0]) + rng.uniform(-0.1, 0.1, size=(crowd, 3))])
        rad = np.concatenate([rad, np.full(crowd, 0.05)])
    n, L = len(pos), float(max(nx, 4))
    sim = _capi.DemSim("RotSphere", 1.2, SKIN, (0, -1, -1), (L, ny + 1.0, nz + 1.0), (1, 0, 0), 1e-7)
    ids = np.arange(n)[::-1].copy()
    sim.add_particles(ids, pos, rad, S.sphere_mass(rad), vel=rng.normal(0, 0.5, size=(n, 3)))
    sim.set_option("precision", precision)
    sim.add_rot_friction_group("friction", 1e3, 0.6, 0.6, 1e3, 1e-7, True, True)
    sim.step(6)
    p = sim.particles()
    order = np.argsort(p["id"])
    x, r = p["pos"][order], rad[::-1]
    want = set()
    for i in range(n - 1):
        d = x[i + 1:] - x[i]
        d[:, 0] -= L * np.round(d[:, 0] / L)
        for j in np.nonzero((d * d).sum(1) < (r[i] + r[i + 1:] + SKIN) ** 2)[0]:
            want.add((i, i + 1 + int(j)))
    before = _pairs(sim)
    sim.search_neighbors()
    sim.step(1)
    after = _pairs(sim)
    # positions move by 1e-7 a step: a pair that near to the cutoff would be an accident of the seed
    assert set(before) == want
    assert set(after) == want
    if crowd:
        assert max(np.bincount([k[0] for k in want])) > 32
    for k, b in before.items():
        if b[4] != 0.0:  # in contact: a rigid step more of the same sliding, not a fresh start
            for c in range(3):
                assert abs(after[k][c] - b[c]) <= 0.5 * max(abs(v) for v in b[:3]) + 1e-12, k
