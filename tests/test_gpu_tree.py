"""The tree kernels at the sizes where their work split changes: one block or
several, whole and partial blocks of nodes, chunked full-depth cells, empty
systems.  A walk that opens every node must meet each particle exactly once; a
Barnes-Hut walk with a huge opening angle must see each system's own total
mass at its centre of mass."""
import numpy as np
import pytest

import ggb200

pytestmark = pytest.mark.gpu


def _system(n, seed, duplicates):
    rng = np.random.default_rng(seed)
    pos = rng.normal(size=(n, 3))
    if duplicates and n > 3:
        pos[1: n // 2] = pos[n // 2]      # one full-depth cell, split into chunks
    pos[:1] = [100.0, 1.0, -2.0]          # the far target
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32).astype(np.float64)
    return pos, mass, np.full(n, 1e-3)


@pytest.mark.parametrize("duplicates", [False, True])
@pytest.mark.parametrize("sizes", [[1], [2], [8], [9], [63, 65], [1023], [1024], [1025], [5, 0, 700, 3000], [2049],
                                   [33000]])
def test_every_particle_is_in_the_tree_once(sizes, duplicates):
    parts = [_system(n, 10 + i, duplicates) for i, n in enumerate(sizes)]
    pos, mass, h = (np.concatenate([p[k] for p in parts]) for k in range(3))
    off = np.concatenate([[0], np.cumsum(sizes)])
    with ggb200.GravityTree() as t:
        t.load(pos, mass, h, counts=sizes)
        t.build()
        _, _, nint, st = t.evaluate(old_acc=np.zeros(len(mass)), err_tol_force_acc=0.001, want_ninter=True)
        assert st["error_word"] == 0
        first = np.array([off[i] for i, n in enumerate(sizes) if n > 8], dtype=np.int32)
        mono = t.evaluate(active=first, err_tol_theta=1e9)[0] if len(first) else []
    for s, n in enumerate(sizes):
        # pairs at r = 0 are not counted: the particle itself and its duplicates
        same = np.ones(n)
        if duplicates and n > 3:
            same[1: n // 2 + 1] = n // 2
        assert np.array_equal(nint[off[s]:off[s + 1]], n - same)
    # a root of more than one leaf bucket is used whole at this opening angle
    for got, a in zip(mono, first):
        b = off[np.searchsorted(off, a, side="right")]
        com = (mass[a:b, None] * pos[a:b]).sum(0) / mass[a:b].sum()
        d = com - pos[a]
        want = mass[a:b].sum() * d / np.linalg.norm(d) ** 3
        # FP32 offset, 1/r and mass: a few roundings of 6e-8
        assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("sizes", [[300], [3000, 0, 40000]])
@pytest.mark.parametrize("group_size", [1, 32])
@pytest.mark.parametrize("kernel", [0, 1])
def test_a_build_whose_waits_give_up_leaves_no_tree(kernel, group_size, sizes):
    """The node kernel's (0) or the moments kernel's (1) blocks wait for one
    block more than there are.  Nothing reads the unfinished tree, neither in a
    context's first build nor over an earlier tree, and the next build is
    whole again."""
    import ctypes

    import torch
    parts = [_system(n, 50 + i, False) for i, n in enumerate(sizes)]
    pos, mass, h = (np.concatenate([p[k] for p in parts]) for k in range(3))
    n = len(mass)
    with ggb200.GravityTree(group_size=group_size) as t:
        t.load(pos, mass, h, counts=sizes)
        t.build()
        want = t.evaluate(err_tol_theta=0.7)[0]

    def status(t):
        st = ggb200.Stats()
        return t._lib.gg_last_stats(t._h, ctypes.byref(st)), st

    with ggb200.GravityTree(group_size=group_size) as t:
        for first in (True, False):
            t.load(pos, mass, h, counts=sizes)
            t.load_velocities(np.ones((n, 3)))
            assert t._lib.gg_selftest_tree_wait(t._h, kernel) == -5      # GG_ERR_TIMEOUT
            if not first:      # a resident tree is moved by the drift; one that is not whole is left alone
                t.drift(1e-3)
            acc = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
            pot = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            t.evaluate_device(acc, pot, err_tol_theta=0.7)
            t.evaluate_potential_device(pot, err_tol_theta=0.7)
            code, st = status(t)
            assert code == -5 and st.n_nodes == 0 and st.interactions == 0 and st.nodes_tested == 0
            assert bool((acc == 7.0).all()) and bool((pot == 7.0).all())
            t.load(pos, mass, h, counts=sizes)
            t.build()
            got = t.evaluate(err_tol_theta=0.7)[0]
            assert np.array_equal(got, want)


def test_a_build_does_not_wait_for_other_kernels_to_end():
    """A build large enough to take every thread slot of the GPU, next to a
    kernel of another stream that holds one for about a second: the build ends
    first, on the slots that are left."""
    import torch
    n = 800000
    rng = np.random.default_rng(60)
    rec = torch.from_numpy(ggb200.make_records(rng.normal(size=(n, 3)), np.ones(n), np.full(n, 1e-3)).view(np.uint8))
    rec = rec.cuda()
    mine, other, done = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event()
    acc = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    with ggb200.GravityTree() as t:
        t.set_stream(mine.cuda_stream)
        t.load_device(rec, [n])
        t.build()
        t.evaluate_device(acc, err_tol_theta=0.7)
        torch.cuda.synchronize()
        want = acc.clone()
        with torch.cuda.stream(other):
            torch.cuda._sleep(2 * 10 ** 9)
            done.record()
        t.build()
        mine.synchronize()
        assert not done.query()
        t.evaluate_device(acc, err_tol_theta=0.7)
        torch.cuda.synchronize()
        assert t.last_stats()["error_word"] == 0
    assert torch.equal(acc, want)


@pytest.mark.parametrize("S", [1, 255, 256, 257, 5000])
def test_root_cubes_of_many_systems(S):
    """Up to 256 systems' root cubes are formed by the extent kernel's last block,
    more by a launch of their own: the FP64 expressions of the extent, to the bit,
    empty systems and single particles included."""
    rng = np.random.default_rng(S)
    sizes = rng.integers(0, 9, S)
    sizes[-1] = 3
    n = int(sizes.sum())
    pos = rng.normal(size=(n, 3)) * 10.0 ** rng.integers(-3, 4, (n, 1))
    with ggb200.GravityTree() as t:
        t.load(pos, np.ones(n), np.full(n, 1e-3), counts=sizes.tolist())
        t.build()
        got = t.domains()
    off = np.concatenate([[0], np.cumsum(sizes)])
    for s in range(S):
        p = pos[off[s]:off[s + 1]]
        mn, mx = (p.min(0), p.max(0)) if len(p) else (np.zeros(3), np.zeros(3))
        length = 1.001 * (mx - mn).max()
        if length <= 0:
            length = 1.0
        mid = 0.5 * (mn + mx)
        assert got[s]["len"] == length
        assert np.array_equal(got[s]["center"], mid) and np.array_equal(got[s]["corner"], mid - 0.5 * length)


def test_root_cubes_of_many_systems_are_no_serial_tail():
    """2,097,152 particles as 262,144 systems of 8: the keys stage takes the time of
    many blocks, not of one that forms every root cube (which took 30 times the
    stage of 256 systems)."""
    import torch
    n = 1 << 21
    rng = np.random.default_rng(61)
    rec = torch.from_numpy(ggb200.make_records(rng.normal(size=(n, 3)), np.ones(n), np.full(n, 1e-3)).view(np.uint8))
    rec = rec.cuda()
    ms = {}
    for S in (256, 262144):
        with ggb200.GravityTree(timing=True) as t:
            t.load_device(rec, [n // S] * S)
            times = []
            for _ in range(6):
                t.build()
                times.append(t.last_stats()["ms_keys"])
        ms[S] = min(times)
    print(ms)
    assert ms[262144] < 12 * ms[256], ms


def test_contexts_on_several_streams_build_beside_a_walk():
    """Four contexts on four streams rebuild and walk while a fifth one's walks
    keep the GPU busy: each gets the bits it gets alone."""
    import torch
    sizes = [1000, 40000, 150000, 700000]
    busy_n = 300000

    def records(n, seed):
        rng = np.random.default_rng(seed)
        r = ggb200.make_records(rng.normal(size=(n, 3)), np.ones(n), np.full(n, 1e-2))
        return torch.from_numpy(r.view(np.uint8)).cuda()

    trees, accs, recs, want = [], [], [], []
    for i, n in enumerate(sizes + [busy_n]):
        t = ggb200.GravityTree()
        s = torch.cuda.Stream()
        t.set_stream(s.cuda_stream)
        recs.append(records(n, 80 + i))
        accs.append(torch.empty((n, 3), dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
        t.load_device(recs[-1], [n])
        t.build()
        t.evaluate_device(accs[-1], err_tol_theta=0.7)
        t.synchronize()
        want.append(accs[-1].clone())
        trees.append(t)
    torch.cuda.synchronize()
    for _ in range(10):
        trees[-1].evaluate_device(accs[-1], err_tol_theta=0.3)
        for t, r, a, n in zip(trees[:-1], recs, accs, sizes):
            a.zero_()
        torch.cuda.current_stream().synchronize()
        for t, r, a, n in zip(trees[:-1], recs, accs, sizes):
            t.load_device(r, [n])
            t.build()
            t.evaluate_device(a, err_tol_theta=0.7)
        for t, a, w in zip(trees[:-1], accs, want):
            t.synchronize()
            assert t.last_stats()["error_word"] == 0
            assert torch.equal(a, w)
    torch.cuda.synchronize()
    for t in trees:
        t.close()
