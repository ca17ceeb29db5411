"""The grid engine's rule kernels at the edges of their tiles: crowds of one
boid, of a warp's 32 and an item's 32 plus or minus one, of the shared list's
512 candidates plus or minus one and beyond, in one cell and across the
periodic corner, each bit for bit against the oracle (one update, its rule
forces, and the neighbour sets)."""
import numpy as np
import pytest

from conftest import assert_bits_equal, make_params, make_sim

pytestmark = pytest.mark.gpu

FIELD = 0.7  # 13 device cells per axis with marun2019's radii


def crowd_state(m, others, centre, seed):
    """m boids in a ball of radius 0.018 around the centre (periodic), the
    others uniform; ids shuffled, so that the crowd's are spread."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(m, 3))
    d *= 0.018 * rng.uniform(0, 1, (m, 1)) ** (1 / 3) / np.linalg.norm(d, axis=1, keepdims=True)
    pos = np.concatenate([np.mod(centre + d, FIELD), rng.uniform(0, FIELD, (others, 3))])
    v = rng.normal(size=pos.shape)
    v *= rng.uniform(0.001, 0.005, (len(v), 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    perm = rng.permutation(len(pos))
    return pos[perm].astype(np.float32).reshape(-1), v[perm].astype(np.float32).reshape(-1)


def check(B, O, pos, vel, tuning):
    prm, n = O.MARUN2019, len(pos) // 3
    p = make_params(O, n, FIELD, prm)
    op, ov = pos.copy(), vel.copy()
    of = O.GridPort(p, op).step(op, ov, 1, forces=True)
    sim = make_sim(B, "grid", n, FIELD, prm)
    if tuning:
        sim.set_tuning(*tuning)
    sim.set_state(pos, vel)
    c, h = sim.neighbor_sets()
    oc, oh = O.neighbor_sets(p, pos, vel)
    assert np.array_equal(c, oc) and np.array_equal(h, oh)
    sim.update(1)
    gp, gv = sim.state()
    assert_bits_equal(gp, op, "positions")
    assert_bits_equal(gv, ov, "velocities")
    assert_bits_equal(sim.forces(), of, "forces")
    sim.close()
    return c


@pytest.mark.parametrize("corner", [False, True])
@pytest.mark.parametrize("tuning", [None, (1, 1, 0, 0), (1 << 30,) * 4])
@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 129, 256, 511, 512, 513, 1100])
def test_crowds_at_tile_edges(boids_lib, oracle_mod, m, tuning, corner):
    pos, vel = crowd_state(m, 40, 0.0 if corner else 6.5 * FIELD / 13, 1000 + m)
    check(boids_lib, oracle_mod, pos, vel, tuning)


@pytest.mark.parametrize("others", [8192 - 700, 8193 - 700, 17000])
def test_crowds_over_the_list_across_id_windows(boids_lib, oracle_mod, others):
    """More accepted neighbours than a warp's list holds, with ids over one,
    just over one and three windows of its bit map."""
    pos, vel = crowd_state(700, others, 0.0, others)
    c = check(boids_lib, oracle_mod, pos, vel, None)
    assert c.max() > 256


@pytest.mark.parametrize("density,share", [(16, 0.0), (22, 0.0), (44, 0.0), (6, 1.0)])
def test_items_done_together(boids_lib, density, share):
    """So many dense-cell items that a CTA takes several at once, of cells with
    a remainder to share among their items (34, 47 and 94 boids a cell) and of
    clusters, against the thread-per-boid kernel alone."""
    B = boids_lib
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    n = 300001
    field = (n / (16384 * density)) ** (1 / 3)
    pos, vel = gathered(n, field, share, density, 90)
    a, b = make_sim(B, "grid", n, field, prm), make_sim(B, "grid", n, field, prm)
    b.set_tuning(*(1 << 30,) * 4)
    for s in (a, b):
        s.set_state(pos, vel)
    for x, y in zip(a.neighbor_sets(), b.neighbor_sets()):
        assert np.array_equal(x, y)
    for s in (a, b):
        s.update(1)
    for x, y in zip(a.state(), b.state()):
        assert_bits_equal(x, y, "state")
    assert_bits_equal(a.forces(), b.forces(), "forces")
    for s in (a, b):
        s.close()


@pytest.mark.parametrize("spread", [True, False])  # the crowd's ids over all, or the lowest
@pytest.mark.parametrize("m", [16000, 17000, 36000])
def test_crowds_over_one_plan_of_id_windows(boids_lib, m, spread):
    """More candidates than the 32 id windows that the dense-cell kernel plans
    at once: the next ones planned behind them, in a handle (files candidates
    by window) and in an ensemble, against a warp per boid."""
    B = boids_lib
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    pos, vel = crowd_state(m, 2000, 0.0, m)
    n = len(pos) // 3
    if not spread:
        far = np.abs(np.mod(pos.reshape(n, 3) + FIELD / 2, FIELD) - FIELD / 2).max(1) > 0.02
        order = np.argsort(far, kind="stable")
        pos, vel = (np.ascontiguousarray(x.reshape(n, 3)[order]).reshape(-1) for x in (pos, vel))
    a, b = make_sim(B, "grid", n, FIELD, prm), make_sim(B, "grid", n, FIELD, prm)
    b.set_tuning(*b.tuning())
    for s in (a, b):
        s.set_state(pos, vel)
    for x, y in zip(a.neighbor_sets(), b.neighbor_sets()):
        assert np.array_equal(x, y)
    for s in (a, b):
        s.update(2)
    for x, y in zip(a.state(), b.state()):
        assert_bits_equal(x, y, "state")
    assert_bits_equal(a.forces(), b.forces(), "forces")
    p = B.flock_params(n, FIELD, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"])
    e = B.Ensemble([(p, B.INIT_RANDOM_UNIFORM, 1)])
    e.init()
    e.set_tuning(*e.tuning())
    e.set_state(0, pos, vel)
    e.step(2)
    for x, y in zip(a.state(), e.state(0)):
        assert_bits_equal(x, y, "ensemble")
    for s in (a, b, e):
        s.close()


def test_ensemble_tuned_between_statistics_and_step(boids_lib):
    """Thresholds set while the statistics' binning waits for its step: that
    step runs on what was classified, the later ones by the thresholds."""
    B = boids_lib
    m = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008))
    flocks = [(B.flock_params(n, (n / 16384) ** (1 / 3), m["sep"], m["ali"], m["coh"], 0.005, 0.001),
               B.INIT_RANDOM_UNIFORM, 5 + n) for n in (1000, 3000)]
    a, b = B.Ensemble(flocks), B.Ensemble(flocks)
    for e in (a, b):
        e.init()
        e.step(60)
    a.stats()
    a.set_tuning(4, 2, 64, 32)
    for e in (a, b):
        e.step(3)
    for f in range(len(flocks)):
        for x, y in zip(a.state(f), b.state(f)):
            assert_bits_equal(x, y, "flock %d" % f)
        assert a.tuning() == (4, 2, 64, 32)
    a.close()
    b.close()


@pytest.mark.parametrize("field", [0.7, 0.13])  # 0.13: every pair is near the radius, no device cells
@pytest.mark.parametrize("n", [1, 2, 15, 17, 63, 64, 65, 255, 257, 1023, 1025, 1041])
def test_all_pairs_at_tile_edges(boids_lib, oracle_mod, n, field):
    """The N^2 kernels at the edges of their 8, 16, 64, 256 and 1024 boid
    tiles, some boids outside the field and beyond the distance up to which
    the filter's angles are used."""
    O, prm = oracle_mod, oracle_mod.MARUN2019
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, field, (n, 3))
    out = rng.random(n) < 0.2
    pos[out] += field * rng.integers(-6, 7, (out.sum(), 3))
    v = rng.normal(size=(n, 3))
    v *= rng.uniform(0.001, 0.005, (n, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    pos, vel = pos.astype(np.float32).reshape(-1), v.astype(np.float32).reshape(-1)
    p = make_params(O, n, field, prm)
    op, ov = pos.copy(), vel.copy()
    of = O.step_allpairs(p, op, ov, 2, forces=True)
    sim = make_sim(boids_lib, "pairs", n, field, prm)
    sim.set_state(pos, vel)
    sim.update(2)
    gp, gv = sim.state()
    assert_bits_equal(gp, op, "positions")
    assert_bits_equal(gv, ov, "velocities")
    assert_bits_equal(sim.forces(), of, "forces")
    sim.close()


@pytest.mark.parametrize("field", [0.02, 0.0008, 1e-6])
def test_all_pairs_with_sight_of_many_fields(boids_lib, oracle_mod, field):
    """Radii of 2.5, 62 and 50 000 fields: every pair is in reach of the N^2 kernels' filter."""
    O, prm, n = oracle_mod, dict(oracle_mod.MARUN2019), 300
    prm["vmax"], prm["vmin"] = field / 10, field / 50
    rng = np.random.default_rng(3)
    pos = rng.uniform(0, field, 3 * n).astype(np.float32)
    vel = (rng.normal(size=3 * n) * field / 50).astype(np.float32)
    op, ov = pos.copy(), vel.copy()
    O.step_allpairs(make_params(O, n, field, prm), op, ov, 2)
    sim = make_sim(boids_lib, "pairs", n, field, prm)
    sim.set_state(pos, vel)
    sim.update(2)
    gp, gv = sim.state()
    assert_bits_equal(gp, op, "positions")
    assert_bits_equal(gv, ov, "velocities")
    sim.close()


@pytest.mark.parametrize("n", [4863, 4864, 4865, 9729])
def test_all_pairs_with_one_boid_a_warp_and_more(boids_lib, n):
    """The N^2 kernels where their last one's 4864 warps have one boid each,
    or go on to another: the neighbour counts that it clears are those it has
    read, update after update (against the same engine on device cells)."""
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    field = (n / 16384) ** (1 / 3)
    pos, vel = gathered(n, field, 0.5, n)
    a, b = make_sim(boids_lib, "pairs", n, field, prm), make_sim(boids_lib, "allpairs", n, field, prm)
    for s in (a, b):
        s.set_state(pos, vel)
    for _ in range(3):
        for s in (a, b):
            s.update(1)
        for x, y in zip(a.state(), b.state()):
            assert_bits_equal(x, y, "state")
    a.close()
    b.close()


@pytest.mark.parametrize("n,field", [(1, 0.7), (1023, 0.7), (8191, 0.7), (8193, 0.7), (16384, 0.7), (16385, 0.7),
                                     (3000, 1.33), (3000, 1.4), (40960, 0.7), (40961, 0.7)])
def test_allocation_free_step_at_its_kernels_limits(boids_lib, oracle_mod, n, field):
    """The allocation-free step on both sides of the lines between its
    one-kernel sort (16384 boids, 65536 cells), the warp-per-boid rules (40960
    boids) and the general path, twice in a row on the same scratch."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    B, O, prm = boids_lib, oracle_mod, oracle_mod.MARUN2019
    p = make_params(O, n, field, prm)
    op, ov = O.init_state(p, "random_uniform", True, 7)
    op, ov = op.reshape(-1).copy(), ov.reshape(-1).copy()
    prms = B.flock_params(n, field, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"])
    a = [torch.from_numpy(x.copy()).cuda() for x in (op, ov)]
    b = [torch.empty_like(x) for x in a]
    port = O.GridPort(p, op)
    for call in range(2):
        rc = B.lib().boids_step_noalloc(C.byref(prms), a[0].data_ptr(), a[1].data_ptr(), b[0].data_ptr(),
                                        b[1].data_ptr(), None)
        assert rc == 0, B.lib().boids_last_error().decode()
        torch.cuda.synchronize()
        port.step(op, ov, 1)
        assert_bits_equal(b[0].cpu().numpy(), op, "positions, call %d" % call)
        assert_bits_equal(b[1].cpu().numpy(), ov, "velocities, call %d" % call)
        a, b = b, a


def gathered(n, field, share, seed, cluster=64):
    """A state of n boids, that share of them in clusters of about so many, the others uniform."""
    rng = np.random.default_rng(seed)
    m = int(n * share)
    centre = rng.uniform(0, field, (m // cluster + 1, 3))
    pos = np.concatenate([np.mod(centre[rng.integers(0, len(centre), m)] + rng.normal(0, 0.012, (m, 3)), field),
                          rng.uniform(0, field, (n - m, 3))])
    v = rng.normal(size=pos.shape)
    v *= rng.uniform(0.001, 0.005, (n, 1)) / np.linalg.norm(v, axis=1, keepdims=True)
    perm = rng.permutation(n)
    return pos[perm].astype(np.float32).reshape(-1), v[perm].astype(np.float32).reshape(-1)


# pairs sharing an x cell: below, about and over the lower line, over the upper one
@pytest.mark.parametrize("share,cluster", [(0.0, 64), (0.06, 64), (0.12, 64), (1.0, 64), (0.5, 1000)])
@pytest.mark.parametrize("n", [40961, 65537, 262144, 262145])
def test_route_by_crowding(boids_lib, n, share, cluster):
    """Flocks over 40960 boids, whose steps go a warp per boid or by the cells'
    split as the scan's measure has it (up to 262144 boids), against the split
    alone: state, forces and neighbour sets, over updates that cross the line,
    and the allocation-free step."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    B = boids_lib
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    field = (n / 16384) ** (1 / 3)
    pos, vel = gathered(n, field, share, n, cluster)
    a, b = make_sim(B, "grid", n, field, prm), make_sim(B, "grid", n, field, prm)
    b.set_tuning(*b.tuning())
    for s in (a, b):
        s.set_state(pos, vel)
    for x, y in zip(a.neighbor_sets(), b.neighbor_sets()):
        assert np.array_equal(x, y)
    for steps in (1, 33):
        for s in (a, b):
            s.update(steps)
        for x, y in zip(a.state(), b.state()):
            assert_bits_equal(x, y, "state")
        assert_bits_equal(a.forces(), b.forces(), "forces")
    q = [torch.from_numpy(np.ascontiguousarray(x).reshape(-1).copy()).cuda() for x in a.state()]
    r = [torch.empty_like(x) for x in q]
    prms = B.flock_params(n, field, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"])
    rc = B.lib().boids_step_noalloc(C.byref(prms), q[0].data_ptr(), q[1].data_ptr(), r[0].data_ptr(), r[1].data_ptr(),
                                    None)
    assert rc == 0, B.lib().boids_last_error().decode()
    torch.cuda.synchronize()
    b.update(1)
    for x, y in zip(r, b.state()):
        assert_bits_equal(x.cpu().numpy(), np.asarray(y).reshape(-1), "allocation-free step")
    a.close()
    b.close()


def test_ensemble_route_by_crowding(boids_lib):
    """An ensemble over 40960 slots whose uniform and gathered flocks (one of a
    single boid, one of an odd size) go a warp per boid, against the split."""
    B = boids_lib
    m = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008))
    sizes = (30001, 1, 129, 16384, 5000)
    flocks = [(B.flock_params(n, max(0.7, (n / 16384) ** (1 / 3)), m["sep"], m["ali"], m["coh"], 0.005, 0.001),
               B.INIT_RANDOM_UNIFORM, n) for n in sizes]
    a, b = B.Ensemble(flocks), B.Ensemble(flocks)
    b.set_tuning(*b.tuning())
    for e in (a, b):
        e.init()
        for f in (0, 4):
            e.set_state(f, *gathered(sizes[f], flocks[f][0].field_size, 1.0, f))
    for steps in (1, 17, 40):
        for e in (a, b):
            e.step(steps)
        for f in range(len(sizes)):
            for x, y in zip(a.state(f), b.state(f)):
                assert_bits_equal(x, y, "flock %d" % f)
    for e in (a, b):
        e.stats()  # bins the state; the step goes on from there
        e.step(1)
    for f in range(len(sizes)):
        for x, y in zip(a.state(f), b.state(f)):
            assert_bits_equal(x, y, "flock %d" % f)
    a.close()
    b.close()


@pytest.mark.parametrize("batch", [False, True])  # a handle, an ensemble
@pytest.mark.parametrize("collapsed", [False, True])
@pytest.mark.parametrize("n", [3000, 50000])
def test_autotuned_flock_keeps_its_route(boids_lib, n, collapsed, batch):
    """Thresholds that an autotuner chose on a uniform or a collapsed flock
    take no route away from it: a gathered state has the kernels of an untuned
    flock, and the same bits."""
    B = boids_lib
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    field = max(0.7, (n / 16384) ** (1 / 3))

    def flock():
        if not batch:
            s = make_sim(B, "grid", n, field, prm, record_forces=False)
            return s, s.set_state, s.update, s.state
        p = B.flock_params(n, field, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"])
        e = B.Ensemble([(p, B.INIT_RANDOM_UNIFORM, 1)])
        e.init()
        return e, lambda *s: e.set_state(0, *s), e.step, lambda: e.state(0)

    crowd, loose = gathered(n, field, float(collapsed), 1, 1000), gathered(n, field, 1.0, 2, 64)
    seen = []
    for tune in (True, False):
        h, put, step, get = flock()
        put(*crowd)
        if tune:
            h.autotune(2)
        put(*loose)
        step(1)
        before = h.kernel_launches()
        step(1)
        seen.append((h.kernel_launches() - before, *get()))
        h.close()
    assert seen[0][0] == seen[1][0]
    for x, y in zip(seen[0][1:], seen[1][1:]):
        assert_bits_equal(x, y, "state")


def test_ensemble_initial_states(boids_lib, oracle_mod):
    """Flocks drawn side by side (more than 8192 boids in all), of both
    placements and odd sizes, against the oracle's sequence for each alone."""
    B, O, prm = boids_lib, oracle_mod, oracle_mod.MARUN2019
    sizes = (16385, 1, 127, 129, 8000, 30000)
    flocks = [(B.flock_params(n, 1.3, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"]),
               B.INIT_TEST if f % 2 else B.INIT_RANDOM_UNIFORM, 11 * f + 3) for f, n in enumerate(sizes)]
    e = B.Ensemble(flocks)
    for _ in range(2):
        e.init()
        for f, n in enumerate(sizes):
            op, ov = O.init_state(make_params(O, n, 1.3, prm), "test" if f % 2 else "random_uniform", True, 11 * f + 3)
            p, v = e.state(f)
            assert_bits_equal(p.reshape(-1), op.reshape(-1), "positions of flock %d" % f)
            assert_bits_equal(v.reshape(-1), ov.reshape(-1), "velocities of flock %d" % f)
    e.close()


@pytest.mark.parametrize("field", [0.21, 0.52, 0.57])  # 4, 10 and 11 cells per axis: 256, 4000 and 5324 in all
@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025])
def test_one_block_sort_at_its_limits(boids_lib, oracle_mod, n, field):
    """Flocks on both sides of the one-block counting sort's 1024 boids and
    4096 cells: a handle's updates and the allocation-free step, twice."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    B, O, prm = boids_lib, oracle_mod, oracle_mod.MARUN2019
    p = make_params(O, n, field, prm)
    op, ov = (x.reshape(-1).copy() for x in O.init_state(p, "random_uniform", True, 3))
    sim = make_sim(B, "grid", n, field, prm)
    sim.set_state(op, ov)
    c, h = sim.neighbor_sets()
    oc, oh = O.neighbor_sets(p, op, ov)
    assert np.array_equal(c, oc) and np.array_equal(h, oh)
    prms = B.flock_params(n, field, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"])
    a = [torch.from_numpy(x.copy()).cuda() for x in (op, ov)]
    b = [torch.empty_like(x) for x in a]
    port = O.GridPort(p, op)
    for call in range(2):
        rc = B.lib().boids_step_noalloc(C.byref(prms), a[0].data_ptr(), a[1].data_ptr(), b[0].data_ptr(),
                                        b[1].data_ptr(), None)
        assert rc == 0, B.lib().boids_last_error().decode()
        torch.cuda.synchronize()
        sim.update(1)
        port.step(op, ov, 1)
        for got in ([x.cpu().numpy() for x in b], [np.asarray(x).reshape(-1) for x in sim.state()]):
            assert_bits_equal(got[0], op, "positions, call %d" % call)
            assert_bits_equal(got[1], ov, "velocities, call %d" % call)
        a, b = b, a
    sim.close()


@pytest.mark.parametrize("n", [1, 1025, 786432, 786433, (1 << 21) + 1])
def test_state_round_trip_in_pieces(boids_lib, n):
    """set_state and get_state on both sides of the sizes at which they move
    the state in one, two and four pieces, the bad coordinate in the last
    piece included."""
    B = boids_lib
    prm = dict(sep=(0.01, 0.5, 0.002), ali=(0.05, 1 / 3, 0.06), coh=(0.05, 0.5, 0.008), vmax=0.005, vmin=0.001)
    field = max(0.3, (n / 16384) ** (1 / 3))
    rng = np.random.default_rng(n)
    pos = rng.uniform(0, field * 0.999, 3 * n).astype(np.float32)
    vel = rng.uniform(-0.003, 0.003, 3 * n).astype(np.float32)
    sim = make_sim(B, "grid", n, field, prm, record_forces=False)
    sim.set_state(pos, vel)
    p, v = sim.state()
    assert_bits_equal(np.asarray(p).reshape(-1), pos, "positions")
    assert_bits_equal(np.asarray(v).reshape(-1), vel, "velocities")
    bad = pos.copy()
    bad[-1] = field * 1.5
    with pytest.raises(B.BoidsError):
        sim.set_state(bad, vel)
    sim.close()


@pytest.mark.parametrize("m", [254, 257, 600])
def test_long_segments_thread_per_boid(boids_lib, oracle_mod, m):
    """Runs of candidates longer than a buffer entry's offset, several passes
    per boid, in an ensemble (whose passes follow one another in one kernel)."""
    B, O, prm = boids_lib, oracle_mod, oracle_mod.MARUN2019
    sizes = (m + 40, 200)
    flocks = [(B.flock_params(n, FIELD, prm["sep"], prm["ali"], prm["coh"], prm["vmax"], prm["vmin"]),
               B.INIT_RANDOM_UNIFORM, 1) for n in sizes]
    e = B.Ensemble(flocks)
    e.init()
    e.set_tuning(*(1 << 30,) * 4)
    want = []
    for f, n in enumerate(sizes):
        pos, vel = crowd_state(m if f == 0 else 100, n - (m if f == 0 else 100), 0.35, f)
        e.set_state(f, pos, vel)
        p = make_params(O, n, FIELD, prm)
        O.GridPort(p, pos).step(pos, vel, 1)
        want.append((pos, vel))
    e.step(1)
    for f in range(len(sizes)):
        for x, y in zip(e.state(f), want[f]):
            assert_bits_equal(x.reshape(-1), y, "flock %d" % f)
    e.close()
