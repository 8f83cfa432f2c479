"""The FP64 contractions: the exact-slice products at the FP64 level and the
small DMMA kernel against quadruple-precision references, over ragged sizes,
index orders and wide dynamic ranges; neither may be less accurate than an
FP64 product is."""
import numpy as np
import pytest

from test_gpu_contract import CASES, _run

pytestmark = pytest.mark.gpu

TC, PIPE = 20, 21          # fcc_test_contract: tensor cores / FP64 pipe whatever the size


def _quad(A, B):
    """A @ B.T with ~106 bits: Dekker products accumulated by TwoSum (Ogita,
    Rump & Oishi, SIAM J. Sci. Comput. 26, 1955 (2005))."""
    def two_sum(a, b):
        s = a + b
        z = s - a
        return s, (a - (s - z)) + (b - z)

    def split(x):
        c = 134217729.0 * x
        h = c - (c - x)
        return h, x - h
    s = np.zeros((A.shape[0], B.shape[0]))
    lo = np.zeros_like(s)
    for k in range(A.shape[1]):
        a, b = A[:, k][:, None], B[:, k][None, :]
        p = a * b
        ah, al = split(a)
        bh, bl = split(b)
        e = al * bl - (((p - ah * bh) - al * bh) - ah * bl)
        s, q = two_sum(s, p)
        lo += q + e
    return s + lo


@pytest.mark.parametrize("prec", [TC, PIPE])
@pytest.mark.parametrize("spec,sa,sb,sc", CASES[:-2] + CASES[-1:])
def test_index_orders_and_scalings(prec, spec, sa, sb, sc):
    rng = np.random.default_rng(3)
    A, B, C = rng.standard_normal(sa), rng.standard_normal(sb), rng.standard_normal(sc)
    for alpha, beta in ((1.0, 0.0), (-0.5, 1.0), (0.7, -1.3)):
        rc, out = _run(prec, spec, A, B, C, alpha, beta)
        assert rc == 0
        ref = alpha * np.einsum(spec, A, B) + beta * C
        assert np.abs(out - ref).max() < 1e-13 * np.abs(ref).max()


# a contraction of integral- or amplitude-like rows spans decades; the error of
# an FP64 product of length K is about sqrt(K / 2) 2^-54.8 of |A_r| |B_c| / sqrt(K)
@pytest.mark.parametrize("M,N,K", [(8, 8, 5000), (130, 17, 700), (46, 46, 46), (200, 300, 129), (64, 64, 1500)])
@pytest.mark.parametrize("spread", [0.0, 3.0, 8.0])
def test_no_less_accurate_than_the_fp64_pipe(M, N, K, spread):
    rng = np.random.default_rng(M + K)
    A = rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-spread, 0, (M, K))
    B = rng.standard_normal((N, K)) * 10.0 ** rng.uniform(-spread, 0, (N, K))
    ref = _quad(A, B)
    err = {}
    for prec in (TC, PIPE):
        rc, out = _run(prec, "mk,nk->mn", A, B, np.zeros((M, N)))
        assert rc == 0
        err[prec] = np.linalg.norm(out - ref) / np.linalg.norm(ref)
    # both end with one rounding to FP64 (rms 2^-53 / sqrt(12) of an element)
    assert err[TC] <= max(err[PIPE], 2.0 ** -53), err


# Sums far below their terms: the leading groups of the exact-slice sums cancel
# and the rest decides.  Every operand is cut 2^-62 below its row's scale (up to
# twice the maximum) and pairs of weight 2^-76 of it are dropped, seven of 2^14
# at most per term: 2^-58 of the scales together, 2^-56 of the maxima.
@pytest.mark.parametrize("M,N,K", [(130, 400, 16), (300, 257, 64), (500, 260, 336), (260, 250, 1024), (250, 260, 1088)])
@pytest.mark.parametrize("level", [4, 13, 22, 30, 45])
def test_sums_that_cancel(M, N, K, level):
    rng = np.random.default_rng(K + level)
    a, b = rng.standard_normal((M, K // 2)), rng.standard_normal((N, K // 2))
    A = np.concatenate([a, -a * (1 + 2.0 ** -level * rng.standard_normal(a.shape))], 1)
    B = np.concatenate([b, b], 1)
    rc, out = _run(TC, "mk,nk->mn", A, B, np.zeros((M, N)))
    assert rc == 0
    ref = _quad(A, B)
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    assert np.all(np.abs(out - ref) <= K * 2.0 ** -56 * scale + 2.0 ** -53 * np.abs(ref))


# tiles of pairs of CTAs (even numbers of 128 rows, or eight and more), rows that
# leave the second CTA of a pair empty, and long products turned over; integers,
# so every digit and sum is exact
@pytest.mark.parametrize("M,N,K", [(256, 130, 70), (257, 129, 70), (129, 40, 64), (1025, 17, 65), (1153, 300, 130),
                                   (100, 1030, 2100), (300, 200, 2049), (90, 250, 4100)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-2.0, 1.0), (3.0, -0.5)])
def test_pair_tiles(M, N, K, alpha, beta):
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(-1000, 1000, (M, K)).astype(float)
    B = rng.integers(-1000, 1000, (N, K)).astype(float)
    C = 2.0 * rng.integers(-99, 99, (M, N)).astype(float)
    rc, out = _run(TC, "mk,nk->mn", A, B, C, alpha, beta)
    assert rc == 0
    assert np.array_equal(out, alpha * (A @ B.T) + beta * C)


def test_peaked_rows_against_a_metric():
    # rows with a few large entries against the inverse square root of a nearly
    # dependent metric: the largest entries of one side meet the smallest of the
    # other, and the sums are far below the product of the maxima
    rng = np.random.default_rng(7)
    n, K = 300, 500
    x = np.linspace(0, 30, K)
    S = np.exp(-0.5 * (x[:, None] - x[None, :]) ** 2) + 1e-9 * np.eye(K)
    w, U = np.linalg.eigh(S)
    J = (U / np.sqrt(w)) @ U.T
    A = np.exp(-2.0 * (30 * rng.random(n)[:, None] - x[None, :]) ** 2) * rng.standard_normal((n, K))
    ref = _quad(A, J)
    err = {}
    for prec in (TC, PIPE):
        rc, out = _run(prec, "mk,nk->mn", A, J, np.zeros((n, K)))
        assert rc == 0
        err[prec] = np.linalg.norm(out - ref) / np.linalg.norm(ref)
    assert err[TC] <= max(err[PIPE], 2.0 ** -53), err


@pytest.mark.parametrize("M,N,K", [(1, 5, 3), (7, 9, 1), (16, 17, 4), (33, 15, 130), (5, 5, 9000), (250, 250, 40), (9, 8, 1701), (1, 2, 4097), (64, 8, 31)])
def test_small_kernel_edges(M, N, K):
    rng = np.random.default_rng(M * N + K)
    A = rng.integers(-1000, 1000, (M, K)).astype(float)
    B = rng.integers(-1000, 1000, (N, K)).astype(float)
    C = rng.integers(-9, 9, (M, N)).astype(float)
    rc, out = _run(PIPE, "mk,nk->mn", A, B, C, -1.0, 2.0)
    assert rc == 0
    assert np.array_equal(out, 2.0 * C - A @ B.T)          # integers: exact in any order


@pytest.mark.parametrize("shape,spec,bspec", [((300, 70), "mk,k->m", "col"), ((70, 300), "km,k->m", "row"),
                                              ((12, 25, 40), "kab,k->ab", "row"), ((31, 200), "mk,k->m", "col")])
def test_matrix_vector_both_layouts(shape, spec, bspec):
    rng = np.random.default_rng(1)
    A = rng.integers(-99, 99, shape).astype(float)
    k = shape[-1] if bspec == "col" else shape[0]
    x = rng.integers(-99, 99, k).astype(float)
    ref = np.einsum(spec, A, x)
    rc, out = _run(0, spec, A, x, np.ones_like(ref), 2.0, -1.0)
    assert rc == 0
    assert np.array_equal(out, 2.0 * ref - 1.0)


@pytest.mark.parametrize("M,K", [(32, 31), (70, 300), (129, 33), (1000, 64)])
def test_matrix_vector_bits_do_not_depend_on_the_layout(M, K):
    rng = np.random.default_rng(M + K)
    A, x = rng.standard_normal((M, K)), rng.standard_normal(K)
    rc, rows = _run(PIPE, "mk,k->m", A, x, np.zeros(M))
    rc2, cols = _run(PIPE, "km,k->m", np.ascontiguousarray(A.T), x, np.zeros(M))
    assert rc == 0 and rc2 == 0
    assert np.array_equal(rows, cols)


def test_results_repeat_bit_for_bit():
    rng = np.random.default_rng(2)
    for M, N, K in ((40, 30, 20000), (300, 300, 300)):
        A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
        one, two = (_run(TC, "mk,nk->mn", A, B, np.zeros((M, N)))[1] for _ in range(2))
        assert np.array_equal(one, two)


def test_triples_pack_by_runs_gives_the_same_energy():
    # runs of three, each packed when it is used: the same products, so only the
    # split of a product into jobs (one rounding of an element of W) can differ
    from conftest import inputs
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    inp = inputs(2)
    Options.reset()
    Options.set("cc_max_iter", 2)
    ctx = Context(inp)
    RCCSD.compute(inp, context=ctx)
    lib = _lib.load()
    whole = ctx.triples(_lib.FCC_PREC_FP64)
    assert lib.fcc_test_set_t3_kc(ctx.h, 3) == 0
    runs = ctx.triples(_lib.FCC_PREC_FP64)
    assert lib.fcc_test_set_t3_kc(ctx.h, 0) == 0
    ctx.close()
    Options.reset()
    assert abs(runs - whole) < 1e-13 * abs(whole), (runs, whole)


def test_triples_small_and_sliced_forms_agree():
    # a size on either side of the rule o^3 v^3 (v + o) < 1e8 against the oracle's
    # sum over all triples is in test_gpu_triples.py; here the same amplitudes
    # triple by triple against the whole
    from conftest import inputs
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    import ctypes
    inp = inputs(1)
    Options.reset()
    Options.set("cc_max_iter", 2)
    ctx = Context(inp)
    RCCSD.compute(inp, context=ctx)
    lib = _lib.load()
    whole = ctx.triples(_lib.FCC_PREC_FP64)
    o = inp.o
    ijk = np.array([(i, j, k) for i in range(o) for j in range(i + 1) for k in range(j + 1) if not i == j == k], np.int32)
    each = np.zeros(len(ijk))
    assert lib.fcc_test_triples_subset(ctx.h, ijk.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), len(ijk),
                                       each.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    ctx.close()
    Options.reset()
    assert abs(each.sum() - whole) < 1e-12 * abs(whole), (each.sum(), whole)


# the longest sums of an (H2O)8 iteration: the ladder's (columns c <= d) and the
# singles' (Q, d)
@pytest.mark.parametrize("M,N,K", [(130, 20, 11628), (40, 24, 102144)])
@pytest.mark.parametrize("spread", [0.0, 8.0])
def test_no_less_accurate_than_the_fp64_pipe_over_long_sums(M, N, K, spread):
    rng = np.random.default_rng(M + K)
    A = rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-spread, 0, (M, K))
    B = rng.standard_normal((N, K)) * 10.0 ** rng.uniform(-spread, 0, (N, K))
    ref = _quad(A, B)
    err = {}
    for prec in (TC, PIPE):
        rc, out = _run(prec, "mk,nk->mn", A, B, np.zeros((M, N)))
        assert rc == 0
        err[prec] = np.linalg.norm(out - ref) / np.linalg.norm(ref)
    assert err[TC] <= max(err[PIPE], 2.0 ** -53), err


# Elements of rows that span decades.  An operand is cut 2^-62 below its row's
# scale (up to twice the maximum), and pairs of weight 2^-76 of the scales are
# dropped, seven of 2^14 at most per term: 2^-56 K of the product of the maxima at
# most, whatever an element's own terms are.  (An FP64 product is within K 2^-53 of
# the sum of an element's own |a| |b|: nearer where that sum is below 2^-3 of the
# product of the maxima, as here.)
@pytest.mark.parametrize("M,N,K", [(300, 257, 64), (200, 300, 700), (130, 40, 5000)])
def test_elements_of_wide_rows(M, N, K):
    rng = np.random.default_rng(K)
    A = rng.standard_normal((M, K)) * 10.0 ** rng.uniform(-12, 0, (M, K))
    B = rng.standard_normal((N, K)) * 10.0 ** rng.uniform(-12, 0, (N, K))
    A[:, 0], B[:, 0] = 1.0, 0.0        # the row maxima do not meet
    A[:, 1], B[:, 1] = 0.0, 1.0
    rc, out = _run(TC, "mk,nk->mn", A, B, np.zeros((M, N)))
    assert rc == 0
    ref = _quad(A, B)
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    assert np.all(np.abs(out - ref) <= K * 2.0 ** -56 * scale + 2.0 ** -53 * np.abs(ref))
