"""The walk's lists and rounds at the sizes where they are cut: group sizes
around 32 and 64, flush thresholds, long leaf runs, few particles.  With OldAcc
0 the relative criterion opens every node, so the walk is a direct sum: each
target meets every other particle once, and forces and potentials agree with
the FP64 sum to FP32 rounding."""
import numpy as np
import pytest

import ggb200
import oracle

pytestmark = pytest.mark.gpu


def _system(n, softening, seed):
    rng = np.random.default_rng(seed)
    pos = rng.normal(size=(n, 3)) * np.array([1.0, 1.0, 0.2])
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32).astype(np.float64)
    h = np.full(n, {"none": 0.0, "one": 0.4, "two": 0.4}[softening])
    if softening == "two":
        h[::3] = 0.15
    return pos, mass, h.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("softening", ["none", "one", "two"])
@pytest.mark.parametrize("group_size,flush,leaf_size", [(1, 128, 1), (2, 32, 8), (31, 64, 8), (32, 128, 32), (33, 96, 8),
                                                        (63, 32, 32), (64, 128, 8)])
@pytest.mark.parametrize("n", [2, 33, 65, 700, 3001])
def test_opening_every_node_is_the_direct_sum(n, group_size, flush, leaf_size, softening):
    pos, mass, h = _system(n, softening, n)
    with ggb200.GravityTree(group_size=group_size, flush=flush, leaf_size=leaf_size) as t:
        t.load(pos, mass, h)
        t.build()
        zero = np.zeros(n)
        acc, pot, nint, st = t.evaluate(old_acc=zero, err_tol_force_acc=0.001, want_ninter=True)
        only, _ = t.evaluate_potential(old_acc=zero, err_tol_force_acc=0.001)
    assert st["error_word"] == 0
    assert np.all(nint == n - 1)
    want, wpot = oracle.direct_sum(pos, mass, h)
    # a pair's FP32 offset, 1/r and force factor carry about ten roundings of
    # 6e-8; the spline's corrections cancel to a few times that near u = 1
    assert np.linalg.norm(acc - want) < 3e-6 * np.linalg.norm(want)
    assert np.linalg.norm(pot - wpot) < 2e-6 * np.linalg.norm(wpot)
    if softening != "none":     # the potential walk's self term is infinite without softening
        # it adds each target's own term, 2.8 m / h, in FP32 and takes it out
        # again: up to four roundings of 6e-8 of it stay behind per target
        own = 4 * 6e-8 * np.linalg.norm(2.8 * mass / h)
        assert np.linalg.norm(only - wpot) < 2e-6 * np.linalg.norm(wpot) + own


# (box half-width, kernel radius, particle mass); a pair's force factor m/r^3 has to be an FP32 number
@pytest.mark.parametrize("scale,h,m", [(1.0, 0.0, 1.0), (1e-8, 0.0, 1e-8), (1e8, 0.0, 1.0), (1.0, 1e-14, 1.0),
                                       (1e8, 1e-6, 1.0), (1.0, 1e-25, 1e-6), (1e-8, 4e-9, 1.0), (1e8, 4e7, 1.0),
                                       (1e13, 4e12, 1e30)])
@pytest.mark.parametrize("group_size", [1, 32, 64])
def test_close_pairs_at_any_scale(group_size, scale, h, m):
    """One group's worth of particles in a box around the origin, two of them
    1e-7 box widths apart at its centre (where the walk's FP32 offsets resolve
    them), with and without softening, the kernel radius far below or near the
    box."""
    n = 32
    rng = np.random.default_rng(11)
    pos = rng.uniform(-0.9, 0.9, (n, 3))
    pos[0], pos[1] = [-1.0, -1.0, -1.0], [1.0, 1.0, 1.0]       # the box, centred on the origin
    pos[2], pos[3] = [5e-8, 2e-8, -3e-8], [-5e-8, -2e-8, 3e-8]
    pos *= scale
    mass, hh = np.full(n, m), np.full(n, h)
    with ggb200.GravityTree(group_size=group_size) as t:
        t.load(pos, mass, hh)
        t.build()
        acc, pot, nint, st = t.evaluate(old_acc=np.zeros(n), err_tol_force_acc=0.001, want_ninter=True)
    assert st["error_word"] == 0 and np.all(nint == n - 1)
    want, wpot = oracle.direct_sum(pos, mass.astype(np.float32), hh.astype(np.float32))
    # each pair carries about ten roundings of 6e-8, relative to its own size; the
    # Newtonian pair bounds the softened one
    d = pos[None] - pos[:, None]
    r = np.sqrt((d ** 2).sum(-1)) + np.where(np.eye(n) > 0, np.inf, 0.0)
    r = np.maximum(r, 0.3 * h)
    assert np.all(np.linalg.norm(acc - want, axis=1) < 2e-6 * (m / r ** 2).sum(1))
    assert np.all(np.abs(pot - wpot) < 2e-6 * (m / r).sum(1))


@pytest.mark.parametrize("every_node", [False, True])
def test_cut_walks_give_the_same_bits_alone_and_in_a_batch(every_node):
    """A system in the range of sizes whose long walks are cut, opening every
    node: its sub-walks run as tasks when it is alone, and as each warp's own
    work in a batch too large for that.  Same interactions, same bits.  (A strict
    Barnes-Hut pass has long walks too, but none longer than the work of a cut.)"""
    n = 98304
    pos, mass, h = _system(n, "one", 5)
    big = 400001 - n
    rng = np.random.default_rng(6)
    more, mm = rng.normal(size=(big, 3)), np.full(big, 1.0)
    theta = dict(err_tol_theta=0.15)     # a Barnes-Hut pass strict enough for long walks
    old, both = None, None
    if every_node:
        theta = dict(err_tol_force_acc=0.001)
        old = np.full(n, 1e-30)
        both = np.concatenate([old, np.full(big, 1e30)])
    with ggb200.GravityTree() as t:
        t.load(pos, mass, h)
        t.build()
        alone = t.evaluate(old_acc=old, want_ninter=True, **theta)
        cuts = [t.last_cuts()]
        t.load(np.concatenate([pos, more]), np.concatenate([mass, mm]), np.concatenate([h, np.full(big, h[0])]),
               counts=[n, big])
        t.build()
        batch = t.evaluate(old_acc=both, want_ninter=True, **theta)
        cuts.append(t.last_cuts())
    assert cuts[0] == cuts[1] and (cuts[0] > 0) == every_node
    assert alone[3]["error_word"] == 0 and batch[3]["error_word"] == 0
    assert alone[2].mean() > 8192        # long enough to be cut
    for a, b in zip(alone[:3], batch[:3]):
        assert np.array_equal(a, b[:n])


# one system as tasks (98,304 and 131,072 + 1 targets: both work limits) and, past the
# records of tasks or beside a second system, each warp its own sub-walks
@pytest.mark.parametrize("n,other", [(98304, 0), (131073, 0), (98304, 302000)])
@pytest.mark.parametrize("group_size,staging", [(32, 0), (32, 1), (64, 0), (64, 1)])
def test_cut_walks_that_open_every_node_are_the_direct_sum(n, other, group_size, staging):
    pos, mass, h = _system(n, "one", 8)
    if other:
        rng = np.random.default_rng(9)
        pos = np.concatenate([pos, rng.normal(size=(other, 3))])
        mass, h = np.concatenate([mass, np.ones(other)]), np.full(n + other, h[0])
    counts = [n, other] if other else [n]
    old = np.full(n + other, 1e-30)    # opens every node; no walk is cut with an OldAcc of 0
    old[n:] = 1e30                     # the other system's nodes are used whole
    with ggb200.GravityTree(group_size=group_size, node_staging=staging) as t:
        t.load(pos, mass, h, counts=counts)
        t.build()
        acc, pot, nint, st = t.evaluate(old_acc=old, err_tol_force_acc=0.001, want_ninter=True)
        # every group meets n - 1 particles, far beyond the work of a cut
        assert t.last_cuts() > 0.5 * (n // group_size)
        only, _ = t.evaluate_potential(old_acc=old, err_tol_force_acc=0.001)
        assert t.last_cuts() > 0.5 * (n // group_size)
    assert st["error_word"] == 0
    assert np.all(nint[:n] == n - 1)
    tg = np.arange(0, n, 401).astype(np.int32)
    want, wpot = oracle.direct_sum(pos[:n], mass[:n], h[:n], targets=tg)
    # as above: about ten roundings of 6e-8 per pair
    assert np.linalg.norm(acc[tg] - want) < 3e-6 * np.linalg.norm(want)
    assert np.linalg.norm(pot[tg] - wpot) < 2e-6 * np.linalg.norm(wpot)
    own = 4 * 6e-8 * np.linalg.norm(2.8 * mass[tg] / h[tg])
    assert np.linalg.norm(only[tg] - wpot) < 2e-6 * np.linalg.norm(wpot) + own


@pytest.mark.parametrize("group_size", [32, 64])
def test_cut_walks_of_a_subset_and_after_a_stack_overflow(group_size):
    """An active subset inside the window, in an order of its own, and the same
    with a node stack that overflows before and after cuts: the walk runs again
    with a larger one and gives the same bits."""
    n = 200000
    pos, mass, h = _system(n, "two", 10)
    act = np.random.default_rng(11).permutation(n)[:99000].astype(np.int32)
    out = []
    for entries in (0, 64):
        with ggb200.GravityTree(group_size=group_size, walk_stack_entries=entries) as t:
            t.load(pos, mass, h)
            t.build()
            out.append(t.evaluate(active=act, old_acc=np.full(n, 1e-30), err_tol_force_acc=0.001, want_ninter=True))
            assert t.last_cuts() > 0
    assert out[0][3]["error_word"] == 0 and out[1][3]["error_word"] == 0
    for a, b in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(a, b)
    assert np.all(out[0][2] == n - 1)
    few = np.arange(0, act.size, 997)
    want, wpot = oracle.direct_sum(pos, mass, h, targets=act[few])
    assert np.linalg.norm(out[0][0][few] - want) < 3e-6 * np.linalg.norm(want)
    assert np.linalg.norm(out[0][1][few] - wpot) < 2e-6 * np.linalg.norm(wpot)


@pytest.mark.parametrize("criterion", ["strict", "all"])
@pytest.mark.parametrize("group_size", [32, 64])
def test_cuts_do_not_lengthen_walks_that_are_all_long(group_size, criterion):
    """300,000 targets are the most a system is cut with.  Where a strict criterion
    (or an OldAcc of 0) makes every walk long, one more target, which switches cuts
    off, changes the time by little (cuts of most walks made it 1.3 to 1.8)."""
    import torch
    rng = np.random.default_rng(13)
    pos = rng.normal(size=(300001, 3)) * (0.05 + rng.random((300001, 1)) ** 4)
    best = {}
    for n in (300000, 300001):
        rec = torch.from_numpy(ggb200.make_records(pos[:n], np.ones(n), np.full(n, 1e-3)).view(np.uint8)).cuda()
        acc = torch.empty((n, 3), dtype=torch.float64, device="cuda")
        with ggb200.GravityTree(group_size=group_size, timing=True) as t:
            t.set_stream(torch.cuda.current_stream().cuda_stream)
            t.load_device(rec, [n])
            t.build()
            t.evaluate_device(acc, err_tol_theta=0.7)
            old = acc.norm(dim=1) if criterion == "strict" else torch.zeros(n, dtype=torch.float64, device="cuda")
            times = []
            for _ in range(5):
                t.evaluate_device(acc, d_old_acc=old, err_tol_force_acc=1e-5)
                times.append(t.last_stats()["ms_walk"])
            best[n] = min(times)
    assert best[300000] < 1.15 * best[300001], best


def test_small_subsets_of_a_large_system_are_not_prepared_for_cuts():
    """A subset walk pays for cuts (41 MB of records) only with as many targets as a
    cut takes; the records of a later, larger one do not make a
    captured step stale."""
    import torch
    n, small = 350000, 98303
    rng = np.random.default_rng(12)
    rec = torch.from_numpy(ggb200.make_records(rng.normal(size=(n, 3)), np.ones(n), np.full(n, 1e-3)).view(np.uint8))
    rec = rec.cuda()
    stream = torch.cuda.Stream()
    acc = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    acc2 = torch.empty_like(acc)
    act = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    walks = dict(err_tol_theta=0.7)
    with ggb200.GravityTree() as t:
        t.set_stream(stream.cuda_stream)
        t.load_device(rec, [n])
        t.build()
        t.evaluate_device(acc, **walks)
        t.evaluate_device(acc2, d_active=act, n_active=1000, **walks)     # allocates what any subset takes
        t.evaluate_device(acc2, d_active=act, n_active=small, **walks)
        t.evaluate_device(acc2, d_active=act, n_active=n, **walks)
        before, launches = t.device_bytes(), []
        for k in (1000, small, n, n, small + 1):     # (the last is the first that may be cut)
            l0 = ggb200.kernel_launches()
            t.evaluate_device(acc2, d_active=act, n_active=k, **walks)
            launches.append(ggb200.kernel_launches() - l0)
            if k == n:
                assert t.device_bytes() == before
                t.capture_step(acc, **walks)
        stream.synchronize()
        assert t.device_bytes() > before + (30 << 20)
        assert launches[1] == launches[2] == launches[3] == launches[4]
        t.launch_step()
        stream.synchronize()
        assert t.last_stats()["error_word"] == 0
