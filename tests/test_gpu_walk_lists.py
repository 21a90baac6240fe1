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


def test_cut_walks_give_the_same_bits_alone_and_in_a_batch():
    """A system in the range of sizes whose long walks are cut, opening every
    node: its sub-walks run as tasks when it is alone, and as each warp's own
    work in a batch too large for that.  Same interactions, same bits."""
    n = 98304
    pos, mass, h = _system(n, "one", 5)
    big = 400001 - n
    rng = np.random.default_rng(6)
    more, mm = rng.normal(size=(big, 3)), np.full(big, 1.0)
    theta = dict(err_tol_theta=0.15)     # a Barnes-Hut pass strict enough for long walks
    with ggb200.GravityTree() as t:
        t.load(pos, mass, h)
        t.build()
        alone = t.evaluate(want_ninter=True, **theta)
        t.load(np.concatenate([pos, more]), np.concatenate([mass, mm]), np.concatenate([h, np.full(big, h[0])]),
               counts=[n, big])
        t.build()
        batch = t.evaluate(want_ninter=True, **theta)
    assert alone[3]["error_word"] == 0 and batch[3]["error_word"] == 0
    assert alone[2].mean() > 8192        # long enough to be cut
    for a, b in zip(alone[:3], batch[:3]):
        assert np.array_equal(a, b[:n])
