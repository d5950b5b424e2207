"""Small batches run whole iterations in one launch (k_iterate); with option use_graph 0
the same steps are launched one by one.  Both take the same sums in the same order,
so every result is the same bits: one tile and many, 2-D and 3-D, odd and even
line lengths, deflated and cyclic systems, exits on ITMAX and on convergence."""
import numpy as np
import pytest

from mfix_b200 import leq
from mfix_b200 import systems as S

pytestmark = pytest.mark.gpu


def _launched(solve):
    assert leq.set_option("use_graph", 0) == 0
    try:
        return solve()
    finally:
        leq.set_option("use_graph", 1)


CASES = {
    "one_tile_2d": lambda: S.conv_diff(20, 30, 1, seed=1, do_k=False),
    "even_2d": lambda: S.conv_diff(64, 64, 1, seed=2, do_k=False),
    "odd_2d": lambda: S.conv_diff(61, 47, 1, seed=3, do_k=False),
    "odd_3d": lambda: S.conv_diff(19, 25, 17, seed=4),
    "even_3d": lambda: S.conv_diff(40, 64, 33, seed=5),
    "most_tiles": lambda: S.conv_diff(89, 70, 90, seed=6),  # 148 tiles: one per SM
    "capped": lambda: S.conv_diff(24, 30, 22, seed=7, itmax=5, tol=1e-10),
    "deflated": lambda: S.pressure_scaled(24, 30, 22, seed=8, tol=1e-6),
    "cyclic": lambda: S.conv_diff_cyclic(12, 16, 10, seed=9, cyc=5),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", sorted(CASES))
def test_same_bits_as_launches(cuda, case, precision):
    s = CASES[case]()

    def solve():
        w = s.copy()
        assert leq.set_option("precision", precision) == 0
        try:
            ier = leq.solve_system(w)
        finally:
            leq.set_option("precision", 0)
        st = leq.last_stats()
        return ier, w, {k: st[k] for k in ("iterations", "outer_steps", "exit_kind", "rnorm", "rnorm0", "deflated",
                                           "fp64_fallback", "line_skips", "line_fallbacks")}, st["kernel_launches"]

    solve()  # the line shapes are tuned now
    i1, w1, s1, n1 = solve()
    i2, w2, s2, n2 = _launched(solve)
    assert i1 == i2 and s1 == s2
    assert n2 - n1 > 8 * s1["iterations"]  # k_iterate took the iterations of the first solve
    assert np.array_equal(w1.x, w2.x) and np.array_equal(w1.a, w2.a) and np.array_equal(w1.b, w2.b)


@pytest.mark.parametrize("precision", [0, 1])
def test_one_tile_too_many_is_launched(cuda, precision):
    """149 tiles on 148 SMs: every kernel of an iteration is launched by itself."""
    s = S.conv_diff(90, 70, 90, seed=6, itmax=5, tol=1e-30)
    rc, res = leq.batch_solve([s], precision=precision)
    assert rc == 0 and leq.last_stats()["kernel_launches"] > 8 * 5


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_same_bits_as_launches(cuda, precision):
    sysm = [S.conv_diff(*d, seed=q, do_k=d[2] > 1) for q, d in
            enumerate([(16, 18, 16), (30, 31, 1), (12, 64, 9), (5, 6, 7), (33, 20, 12)])]

    def solve():
        batch = [s.copy() for s in sysm]
        rc, res = leq.batch_solve(batch, precision=precision)
        assert rc == 0
        return batch, [(r.ier, r.iterations, r.rnorm) for r in res]

    solve()
    b1, r1 = solve()
    b2, r2 = _launched(solve)
    assert r1 == r2
    assert all(np.array_equal(u.x, v.x) for u, v in zip(b1, b2))


@pytest.mark.parametrize("precision", [0, 1])
def test_expired_wait_ends_its_system_alone(cuda, precision):
    """A barrier wait that runs out (a limit of no reads at all) ends that system with IER -15 in all
    its blocks; a system of one block, which waits for none, is solved, and so is the next batch."""
    one, many = S.conv_diff(4, 6, 3, seed=1), S.conv_diff(40, 64, 33, seed=5)

    def solve():
        batch = [one.copy(), many.copy()]
        _, res = leq.batch_solve(batch, precision=precision)
        return batch, [r.ier for r in res]

    want, ier = solve()
    assert ier == [0, 0]
    assert leq.set_option("wait_polls", 0) == 0
    try:
        got, ier = solve()
    finally:
        assert leq.set_option("wait_polls", 2 ** 22) == 0
    assert ier == [0, leq.IER_INCOMPLETE]
    assert np.array_equal(got[0].x, want[0].x)
    got, ier = solve()
    assert ier == [0, 0] and all(np.array_equal(u.x, v.x) for u, v in zip(got, want))
