"""The multi-step kernel (bond-free specimens) against single-step launches of the same timesteps.

Both form every particle's sums in the same order, so the FP64 states are equal bit for bit,
whatever the block's share of particles, its pruned lists, their refreshes and the neighbour
searches in between.  Wall reactions are summed over blocks of different sizes: each is compared
within n * 2^-52 of the sum's scale.  The FP32-force form differs by FMA contraction only: its
rounding (2^-24 per operation, about 40 operations and 20 contributions a force) stays below 1e-5
of the largest force.
"""
import numpy as np
import pytest

import scenarios as S
from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(dem_lib):
    if not gpu_available():
        pytest.skip("no GPU")
    from esys.lsm import _capi

    return lambda *a: _capi.DemSim(*a)


def _pair(gpu, build, kw, steps, prec=64):  # the specimen in the multi-step kernel and in single steps
    out = []
    for single in (False, True):
        s = build(gpu, **kw)
        if prec != 64:
            s.set_option("precision", prec)
        if single:
            s.set_option("split", 1)  # two single-step kernels a step (one where the law has no split form)
        for k in steps:
            s.step(k)
        out.append(s)
    return out


def _equal(a, b, groups, walls):
    pa, pb = a.particles(), b.particles()
    for k in pa:
        assert np.array_equal(pa[k], pb[k]), (k, np.abs(pa[k] - pb[k]).max())
    for g in groups:
        for x, y in zip(a.pairs(g), b.pairs(g)):
            assert np.array_equal(x, y), g
    assert a.counters()["rebuilds"] == b.counters()["rebuilds"]
    n = len(pa["id"])
    for w in walls:
        (xa, fa), (xb, fb) = a.wall(w), b.wall(w)
        assert np.array_equal(xa, xb)
        assert np.abs(fa - fb).max() <= n * 2.0 ** -52 * max(np.abs(fb).max(), 1e-300)


FR = (["friction"], ["floor", "roof"])


def _skin(gpu, v):
    """The same scenario with another search skin (verletDist)."""
    return lambda pt, gs, vd, *rest: gpu(pt, gs, v, *rest)


def _thin(build, v):
    return lambda gpu, **kw: build(_skin(gpu, v), **kw)


def _closing(gpu, speed, **kw):
    """A frictional packing between platens that the native loader closes (and slides) every step."""
    s = S.friction_pack(gpu, **kw)
    s.set_wall_velocity("floor", (3.0, speed, 0.0))
    s.set_wall_velocity("roof", (0.0, -speed, 1.0))
    return s


def _two_groups(gpu, **kw):
    """RotFriction and elastic groups on the same pairs, viscous and local dampings of both motions, a third
    of the particles held still, not turning, or both."""
    class Held:
        def __init__(self, *a):
            self.sim = gpu(*a)

        def __getattr__(self, k):
            return getattr(self.sim, k)

        def add_particles(self, ids, *a, **k):
            self.sim.add_particles(ids, *a, flags=np.where(np.arange(len(ids)) % 3 == 0, np.arange(len(ids)) // 3 % 4, 0), **k)

    s = S.friction_pack(Held, **kw).sim
    s.add_elastic_group("elastic", 500.0, True)
    s.add_local_damping("ALocal", 0, 0.2)
    s.add_local_damping("rotlocal", 1, 0.2)
    return s


# name, scenario, its arguments, steps of each call, what to compare, whether the multi-step kernel takes them
# (a dense frictional packing in FP64 whose records do not fit a block's shared memory takes single steps)
CASES = [
    # one particle; fewer particles than a block's groups; a ragged count over many blocks
    ("one", S.friction_pack, dict(nx=1, ny=1, nz=1), (5,), FR, True),
    ("seven", S.friction_pack, dict(nx=7, ny=1, nz=1), (1, 2, 30), FR, True),
    ("ragged", S.friction_pack, dict(nx=13, ny=11, nz=12), (60,), FR, True),
    ("periodic", S.friction_pack, dict(nx=9, ny=6, nz=7, periodic=True, vscale=30.0), (90, 1, 40), FR, True),
    # fast: the lists are pruned again and neighbour searches stop the launch every few steps
    ("fast", S.friction_pack, dict(nx=10, ny=9, nz=8, vscale=250.0), (64,), FR, True),
    ("elastic", S.gravity_box, dict(n_side=9), (120,), (["elastic"], ["xlo", "zlo", "zhi"]), True),
    ("nrot_friction", S.nrot_friction_pack, dict(n_side=7, vscale=20.0), (80,), (["friction"], []), True),
    ("rot_nrot_friction", S.nrot_friction_pack, dict(rot=True, n_side=5), (50,), (["friction"], []), True),
    ("hertz", S.hertz_mindlin_pack, dict(n_side=6, vscale=20.0), (80,), ([], []), True),
    # every law's and damping's place in a step at once
    ("two_groups", _two_groups, dict(nx=13, ny=11, nz=12), (50, 3, 20), (["friction", "elastic"], FR[1]), True),
    # planes that move every step: their forces, their reactions and the searches in between
    ("closing", _closing, dict(nx=13, ny=11, nz=12, speed=40.0), (1, 2, 25, 3, 60), FR, True),
    ("closing_periodic", _closing, dict(nx=12, ny=9, nz=7, speed=40.0, periodic=True), (40, 7), FR, True),
    # two halves of a block no longer hold the particles (more than 256 a block)
    ("block_256_up", S.friction_pack, dict(nx=36, ny=34, nz=35, squeeze=1.1), (30,), FR, False),
    ("block_256_up_touching", _thin(S.friction_pack, 0.02), dict(nx=36, ny=34, nz=35, squeeze=0.96), (30,), FR, True),
    # records read back from L2: results all at once, in several parts, and nothing in contact
    ("parts", S.friction_pack, dict(nx=44, ny=40, nz=40), (12,), FR, False),
    ("at_once_touching", _thin(S.friction_pack, 0.01), dict(nx=42, ny=40, nz=40, squeeze=0.96), (40,), FR, True),
    ("parts_touching", _thin(S.friction_pack, 0.01), dict(nx=60, ny=50, nz=50, squeeze=0.96), (30, 5), FR, True),
    ("parts_closing", _thin(_closing, 0.01), dict(nx=60, ny=50, nz=50, squeeze=0.96, speed=150.0), (5, 20), FR, True),
    ("parts_nrot_friction", _thin(S.nrot_friction_pack, 0.01), dict(n_side=46), (30,), (["friction"], ["zlo"]), True),
    ("parts_rot_nrot_friction", _thin(S.nrot_friction_pack, 0.01), dict(n_side=46, rot=True), (30,), (["friction"], []), True),
    ("parts_hertz", _thin(S.hertz_mindlin_pack, 0.01), dict(n_side=46), (30,), ([], []), True),
    ("at_once_two_groups", _thin(_two_groups, 0.002), dict(nx=44, ny=40, nz=40, squeeze=0.99), (30,),
     (["friction", "elastic"], FR[1]), True),
    ("loose", S.friction_pack, dict(nx=70, ny=50, nz=50, squeeze=1.14), (12,), FR, True),
    ("beyond", S.friction_pack, dict(nx=64, ny=44, nz=44, squeeze=0.8), (8,), FR, False),
]


@pytest.mark.parametrize("name,build,kw,steps,what,multi", CASES, ids=[c[0] for c in CASES])
def test_equals_single_steps(gpu, name, build, kw, steps, what, multi):
    a, b = _pair(gpu, build, kw, steps)
    _equal(a, b, *what)
    runs, full = (a.counters()[k] for k in ("multi_step_launches", "multi_step_full"))
    assert full == 0 and (runs > 0) == multi and runs < a.counters()["steps"]
    assert b.counters()["multi_step_launches"] == 0
    if "closing" in name:
        assert all(np.abs(a.wall(w)[1]).max() > 0 for w in what[1])


def test_lists_that_outgrow_a_block_in_mid_launch(gpu):
    """The launch leaves before the step whose pruned lists do not fit, the call goes on singly, and the
    multi-step kernel is tried again after the next neighbour search."""
    def build(make):
        s = S.gravity_box(make, n_side=60)
        s.add_gravity("pull", (0.0, 0.0, -2000.0))
        return s

    a, b = _pair(gpu, lambda g: build(g), {}, (90,))
    c = a.counters()
    assert c["multi_step_launches"] == 1 and c["multi_step_full"] == 1 and c["rebuilds"] == b.counters()["rebuilds"]
    _equal(a, b, ["elastic"], ["zlo"])
    for s in (a, b):
        s.step(60)
    c = a.counters()
    assert c["multi_step_launches"] > 1
    _equal(a, b, ["elastic"], ["zlo"])


# shape, squeeze, steps, launches of the multi-step kernel that its lists did not fit
FP32 = [(dict(nx=13, ny=11, nz=12), 40, 0), (dict(nx=36, ny=34, nz=35), 30, 0), (dict(nx=44, ny=40, nz=40), 12, 0),
        (dict(nx=70, ny=50, nz=50, squeeze=1.14), 12, 0),
        (dict(nx=64, ny=44, nz=44, squeeze=0.8), 8, 1)]  # full before the first step


@pytest.mark.parametrize("kw,steps,full", FP32)
def test_fp32_form_equals_single_steps(gpu, kw, steps, full):
    a, b = _pair(gpu, S.friction_pack, kw, (steps,), prec=32)
    pa, pb = a.particles(), b.particles()
    for k in ("pos", "vel", "angvel", "force", "moment"):
        assert np.abs(pa[k] - pb[k]).max() <= 1e-5 * np.abs(pb[k]).max(), k
    for x, y in zip(a.pairs("friction")[:2], b.pairs("friction")[:2]):
        assert np.array_equal(x, y)
    assert a.counters()["multi_step_launches"] >= 1 and a.counters()["multi_step_full"] == full


def test_a_barrier_that_gives_up_loses_the_handle(gpu):
    """A wait that runs out (here at once: no poll at all) ends the launch with blocks at unlike steps.
    The call reports it and the handle refuses everything that follows; others are unaffected."""
    from esys.lsm._capi import DemError, Ensemble

    s, other = (S.friction_pack(gpu, nx=13, ny=11, nz=12) for _ in range(2))
    for x in (s, other):
        x.step(3)
    s.set_option("barrier_polls", 0)
    with pytest.raises(DemError, match="timed out"):
        s.step(5)
    e = Ensemble([s, other])
    for call in (lambda: s.step(1), s.particles, lambda: s.wall("roof"), lambda: s.set_particles(vel=np.zeros((1, 3))),
                 lambda: s.window_forward(2, 2), lambda: s.set_option("precision", 32), lambda: e.step(1)):
        with pytest.raises(DemError, match="state was lost"):
            call()
    e.close()
    other.step(5)
    assert other.timestep == 8


@pytest.mark.parametrize("blocks,launches", [(11, 1), (37, 1), (65535, 10)])
def test_number_of_blocks(gpu, blocks, launches):
    """Any number of blocks that the GPU holds at once gives the same states; more than that is refused
    by the launch and the call goes on in single steps (as where a process may use a part of the GPU)."""
    a, b = (S.friction_pack(gpu, nx=13, ny=11, nz=12) for _ in range(2))
    a.set_option("run_blocks", blocks)
    b.set_option("split", 1)
    for s in (a, b):
        s.step(2)
    before = a.counters()["launches"]
    for s in (a, b):
        s.step(10)
    assert a.counters()["launches"] - before == launches
    _equal(a, b, ["friction"], ["floor", "roof"])


@pytest.mark.parametrize("shape,squeeze,launches", [((13, 11, 12), 0.93, (1, 1, 1, 1)), ((32, 32, 32), 1.04, (1, 2, 1, 1)),
                                                    ((42, 40, 40), 1.14, (1, 2, 3, 1))])
def test_short_calls(gpu, shape, squeeze, launches):
    """Calls of one to four steps: singly where the multi-step kernel's first prune costs more than the
    launches it saves (few and many particles a block, records in L2), and the same states."""
    kw = dict(zip(("nx", "ny", "nz"), shape), squeeze=squeeze)
    a, b = (S.friction_pack(gpu, **kw) for _ in range(2))
    b.set_option("split", 1)
    for s in (a, b):
        s.step(1)
    for k, want in zip((1, 2, 3, 4), launches):
        before = a.counters()["launches"]
        a.step(k)
        assert a.counters()["launches"] - before == want, k
        b.step(k)
    _equal(a, b, ["friction"], ["floor", "roof"])


@pytest.mark.parametrize("precision,lanes", [(64, 1), (32, 2)])
def test_lanes_of_single_steps(gpu, precision, lanes):
    """5.2 entries of the pair list a particle: one lane in FP64 (the states do not depend on how the steps
    are dealt to calls), two by the mean in the FP32 form."""
    a, b, c = (S.friction_pack(gpu, nx=9, ny=6, nz=7, vscale=5.0) for _ in range(3))
    for s in (a, b, c):
        s.set_option("precision", precision)
    b.set_option("threads_per_particle", lanes)
    for _ in range(20):
        a.step(1)
        b.step(1)
    c.step(20)
    pa, pb, pc = a.particles(), b.particles(), c.particles()
    for k in ("pos", "vel", "angvel", "quat"):
        assert np.array_equal(pa[k], pb[k]), k
        assert precision == 32 or np.array_equal(pa[k], pc[k]), k
