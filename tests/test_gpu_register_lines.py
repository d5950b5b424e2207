"""J-line kernels around the edges of their shapes: chunk remainders, one and two
passes, widths that leave lanes idle, short and long lines, both precisions.

Each line is solved by LEQ_MSOLVE (model/leqsol_mod.f:286-598) through the GPU
and through the oracle; the recurrences are re-associated, so the results differ
by a few roundings of a diagonally dominant solve: 1e-12 in FP64.
"""
import numpy as np
import pytest

import oracle
from mfix_b200 import leq
from mfix_b200 import systems as S

pytestmark = pytest.mark.gpu


# interior J cells: L = J + 2; FP64 chunks are 4 rows, half chunks 2, FP32's 8 and 4
@pytest.mark.parametrize("jmax", [1, 2, 5, 6, 14, 16, 17, 30, 62, 64, 66, 126, 128, 130, 254, 256, 258, 300])
def test_msolve_line_lengths(cuda, jmax):
    s = S.conv_diff(5, jmax, 4, seed=jmax)
    dev = "cuda"
    a, b = cuda.from_numpy(s.a).to(dev), cuda.from_numpy(s.b).to(dev)
    x = cuda.zeros(s.n, dtype=cuda.float64, device=dev)
    cuda.cuda.synchronize()
    g = leq.geom(s.imax2, s.jmax2, s.kmax2, s.do_k)
    assert leq.leq_msolve(g, b.data_ptr(), a.data_ptr(), x.data_ptr(), "RSRS", "LINE") == 0
    want = oracle.msolve(s, s.b)[1]
    got = x.cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("jmax", [6, 30, 34, 62, 66, 126, 130, 254, 258, 262, 300])
@pytest.mark.parametrize("lanes", [4, 8, 16, 32])
def test_solve_line_lengths(cuda, precision, jmax, lanes):
    """Whole solves with a forced width: the true residual meets TOL, the mixed form without a hand-over."""
    s = S.conv_diff(6, jmax, 5, seed=jmax, tol=1e-8)
    w = s.copy()
    assert leq.set_option("line_lanes", lanes) == 0 and leq.set_option("precision", precision) == 0
    try:
        assert leq.solve_system(w) == 0
        assert leq.last_stats()["fp64_fallback"] == 0
    finally:
        leq.set_option("precision", 0)
        leq.set_option("line_lanes", 0)
    r = w.b - S.matvec_np(w.imax2, w.jmax2, w.kmax2, w.do_k, w.a, w.x)
    assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(w.b)


def _flag_lines(s, seed):
    """Five interior J-lines with one diagonal shrunk a hundredfold (DGTSV interchanges rows there) and
    one without a tridiagonal (INFO != 0: left as it was); the system still converges."""
    rng = np.random.default_rng(seed)
    lines = [(i + k * s.imax2) * s.jmax2 for i in range(1, s.imax2 - 1) for k in range(1, s.kmax2 - 1)]
    for base in rng.choice(lines, size=5, replace=False):
        s.a[3, base + int(rng.integers(2, s.jmax2 - 2))] *= 0.01
    base = lines[len(lines) // 2]
    s.a[np.ix_([1, 3, 5], range(base + 1, base + s.jmax2 - 1))] = 0.0
    return base


@pytest.mark.parametrize("jmax", [14, 62, 128, 190])  # 4, 16 and 32 lanes, half a chunk, two passes
def test_msolve_flagged_lines(cuda, jmax):
    """Lines that the register kernel hands to DGTSV.  The oracle's result moves by 1.2e-15 at most
    when each entry of A moves by an ulp; 1e-12 as for the lines without interchanges."""
    s = S.conv_diff(7, jmax, 6, seed=jmax)
    oracle.scale(s)
    base = _flag_lines(s, jmax)
    b = np.random.default_rng(4).standard_normal(s.n)
    _, want, skips = oracle.msolve(s, b, "RSRS", "LINE")
    assert skips > 0
    da, db = cuda.from_numpy(s.a).to("cuda"), cuda.from_numpy(b).to("cuda")
    x = cuda.zeros(s.n, dtype=cuda.float64, device="cuda")
    cuda.cuda.synchronize()
    g = leq.geom(s.imax2, s.jmax2, s.kmax2, s.do_k)
    assert leq.leq_msolve(g, db.data_ptr(), da.data_ptr(), x.data_ptr(), "RSRS", "LINE") == 0
    got = x.cpu().numpy()
    assert np.array_equal(got[base:base + s.jmax2], b[base:base + s.jmax2])
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("jmax", [14, 30, 66, 258])
def test_solve_flagged_lines(cuda, precision, jmax):
    """The same in whole solves, in k_iterate and launched (use_graph 0): equal bits, TOL met."""
    s = S.conv_diff(9, jmax, 8, seed=jmax, tol=1e-8)
    _flag_lines(s, jmax)
    out = []
    for graph in (1, 0):
        w = s.copy()
        assert leq.set_option("precision", precision) == 0 and leq.set_option("use_graph", graph) == 0
        try:
            assert leq.solve_system(w) == 0
        finally:
            leq.set_option("precision", 0)
            leq.set_option("use_graph", 1)
        st = leq.last_stats()
        assert st["fp64_fallback"] == 0 and st["line_fallbacks"] > st["line_skips"] > 0
        out.append((w.x, st["iterations"], st["line_fallbacks"], st["line_skips"]))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1:] == out[1][1:]
    r = w.b - S.matvec_np(w.imax2, w.jmax2, w.kmax2, w.do_k, w.a, w.x)
    assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(w.b)


def test_timed_sweeps_leave_the_counts(cuda):
    """The first solve of a line length times the line kernels; those sweeps' flagged lines are not the
    solve's.  JMAX2 = 87 (odd, FP64: a timed length) occurs in no other test."""
    s = S.conv_diff(9, 85, 8, seed=5, tol=1e-8)
    _flag_lines(s, 5)
    counts = []
    for _ in range(2):
        w = s.copy()
        assert leq.solve_system(w) == 0
        st = leq.last_stats()
        counts.append((st["line_skips"], st["line_fallbacks"]))
    assert counts[0] == counts[1] and counts[0][0] > 0


@pytest.mark.parametrize("scale", [1e36, 1e37, 1e38, 1e40])
@pytest.mark.parametrize("graph", [0, 1])
def test_fp32_overflow_is_no_answer(cuda, scale, graph):
    """Right-hand sides whose iteration overflows FP32 (and leaves NaN in the padded lines' pads): the
    FP64 form's verdict, not a wrong answer."""
    s = S.conv_diff(9, 171, 7, seed=6, tol=1e-8)
    s.b *= scale
    assert leq.set_option("precision", 1) == 0 and leq.set_option("use_graph", graph) == 0
    try:
        w = s.copy()
        assert leq.solve_system(w) == 0
    finally:
        leq.set_option("precision", 0)
        leq.set_option("use_graph", 1)
    if scale > 1e39:  # not even the right-hand side is an FP32 number
        assert leq.last_stats()["fp64_fallback"] == 1
    r = w.b - S.matvec_np(w.imax2, w.jmax2, w.kmax2, w.do_k, w.a, w.x)
    assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(w.b)


def _solved_with(tmp_path, s, precision, entry):
    """The solution after the choices file `entry` (None: no file) was read."""
    if entry is not None:
        path = tmp_path / "choices.json"
        path.write_text("[\n  {%s}\n]\n" % entry)
        assert leq.autotune_cache(str(path)) == 0
    w = s.copy()
    try:
        rc, res = leq.batch_solve([w], precision=precision)
    finally:
        leq.autotune_cache(None)
    assert rc == 0 and res[0].ier == 0
    return w.x


@pytest.mark.parametrize("precision,jmax", [(1, 74), (1, 171), (0, 98)])
def test_one_pass_lines_keep_their_shape(cuda, tmp_path, precision, jmax):
    """A length that the register kernel serves in one pass has one shape, whatever was chosen before
    (another batch size, another process): the same bits."""
    s = S.conv_diff(9, jmax, 7, seed=jmax)
    elem, L = (4 if precision else 8), jmax + 2
    want = _solved_with(tmp_path, s, precision, None)
    for lanes in (8, 16):
        entry = f'"elem": {elem}, "L": {L}, "lanes": {lanes}, "staged": 1'
        assert np.array_equal(_solved_with(tmp_path, s, precision, entry), want)


def test_choices_without_a_kernel_are_of_k_jline(cuda, tmp_path):
    """Files from before k_jline_reg name no kernel: their choices were timed on k_jline."""
    s = S.conv_diff(9, 198, 7, seed=4)
    entry = '"elem": 8, "L": 200, "lanes": 32'
    old = _solved_with(tmp_path, s, 0, entry)
    assert np.array_equal(old, _solved_with(tmp_path, s, 0, entry + ', "staged": 1'))
    assert not np.array_equal(old, _solved_with(tmp_path, s, 0, entry + ', "staged": 0'))


def test_batch_of_mixed_parities_equals_alone(cuda):
    """FP64 systems of even and odd JMAX2 in one batch (two line kernels): each as alone."""
    sysm = [S.conv_diff(9, j, 7, seed=j) for j in (20, 21, 62, 63, 128, 131, 10)]
    alone = []
    for s in sysm:
        w = s.copy()
        assert leq.solve_system(w) == 0
        alone.append(w)
    batch = [s.copy() for s in sysm]
    rc, res = leq.batch_solve(batch)
    assert rc == 0
    for w, v, r in zip(alone, batch, res):
        assert r.ier == 0 and np.array_equal(w.x, v.x)
