"""The exact-slice kernel with 8-bit digits: the digit packing against an
integer model through each of its kernels, products whose accumulators reach
the 2^24 bound, and the edges of tiles, chunks and jobs."""
import ctypes
import struct

import numpy as np
import pytest

from oracle import ozaki
from test_gpu_contract import _run

pytestmark = pytest.mark.gpu


def _digits(x, e, S):
    """Balanced base-256 digits of x 2^-e: the integer nearest to |x| 2^(8S - e)
    with the sign of x, halves cut away from zero, carried digit by digit
    (S = 8: the digits of the magnitude with the sign of x)."""
    bits = struct.unpack("<Q", struct.pack("<d", x))[0]
    be, Z = (bits >> 52) & 0x7FF, 0
    if be:
        m = (bits & ((1 << 52) - 1)) | (1 << 52)
        sh = 1075 + e - 8 * S - be
        Z = m << -sh if sh <= 0 else ((m >> sh) + ((m >> (sh - 1)) & 1) if sh < 64 else 0)
    neg = bits >> 63
    if neg and S < 8:
        Z = -Z
    d = [0] * S
    for s in range(S - 1, 0, -1):
        r = (Z + 128) % 256 - 128
        Z = (Z - r) >> 8
        d[s] = r
    d[0] = Z
    return [-t for t in d] if neg and S == 8 else d


# K = 100 and 700: the one-pass row walk with one and several warps a row, the
# fused and the two-pass transposing walk; 4500: the two-pass row walk
@pytest.mark.parametrize("row_fastest,K", [(0, 100), (0, 700), (0, 4500), (0, 5000), (0, 14080), (1, 100), (1, 177),
                                           (1, 700), (1, 1530), (1, 1600)])
@pytest.mark.parametrize("S", [1, 4, 6, 7, 8])
def test_device_wide_digits_are_the_integer_model(row_fastest, K, S):
    from fermicc import _lib
    lib = _lib.load()
    rng = np.random.default_rng(5 + S + 10 * row_fastest + K)
    R = 310 if K >= 5000 else 70      # long rows go through shared memory from 304 rows on
    x = rng.standard_normal((R, K)) * 10.0 ** rng.uniform(-3, 3, (R, 1))
    x[2, :] *= 10.0 ** rng.uniform(-12, 0, K)
    x[3, :] = 0.0
    x[4, :6] = [1.0, -1.0, 0.5, -0.75, 255.5 / 256.0, 5e-324]
    x[5, :] = 2.0 ** 40 * np.sign(rng.standard_normal(K))
    Kpad = (K + 63) // 64 * 64
    src = np.ascontiguousarray(x.T if row_fastest else x)
    out = np.empty((R, S * Kpad), dtype=np.uint16)
    ex = np.empty(R, dtype=np.int32)
    rc = lib.fcc_test_pack_oz(src.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), R, K, row_fastest, 10 + S,
                              out.ctypes.data_as(ctypes.POINTER(ctypes.c_uint16)),
                              ex.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
    assert rc == 0
    mx = np.abs(x).max(axis=1)
    assert np.array_equal(ex, np.where(mx > 0, np.frexp(mx)[1] + 1022, 0))
    got = out.reshape(R, S, Kpad)
    assert not got[:, :, K:].any()
    rows = [0, 2, 3, 4, 5, 33, R - 1]
    want = np.array([[_digits(float(v), int(np.frexp(mx[r])[1]) if mx[r] else 0, S) for v in x[r]] for r in rows])
    f = want.astype(np.float32)
    assert np.array_equal(f.astype(int), want) and np.abs(want).max() <= 256
    bits = (f.view(np.uint32) >> 16).astype(np.uint16).transpose(0, 2, 1)
    have = np.where(got[rows][:, :, :K] == 0x8000, 0, got[rows][:, :, :K])      # a digit -0 is 0
    assert np.array_equal(have, bits)


@pytest.mark.parametrize("digits", [0xFF00, 0xFE80, 0xFEFF, 0x8080])
def test_wide_chunk_sums_stay_exact_at_the_bound(digits):
    # rows of one value whose digits are (255, 0), (255, -128), (255, -1) and
    # (129, -128): sums of one sign, up to 2^24 per accumulator
    M, N, K = 130, 129, 1030
    A = np.full((M, K), digits / 65536.0)
    B = np.full((N, K), -digits / 65536.0)
    rc, out = _run(3, "mk,nk->mn", A, B, np.zeros((M, N)))
    assert rc == 0
    assert np.array_equal(out, np.full((M, N), -K * digits * digits / 2.0 ** 32))


@pytest.mark.parametrize("M,N,K", [(16, 16, 1), (17, 129, 65), (128, 128, 257), (300, 40, 2000), (1300, 1290, 130),
                                   (40, 24, 30000)])
@pytest.mark.parametrize("groups", [6, 7, 9])
def test_exact_products_over_tiles_chunks_and_jobs(M, N, K, groups):
    # 15-bit integers: exact in two slices, so every level gives the exact
    # product, rounded once (|sum| < 2^53) whatever the number of jobs
    rng = np.random.default_rng(M + K + groups)
    Ai = rng.integers(-2**14, 2**14 + 1, size=(M, K))
    Bi = rng.integers(-2**14, 2**14 + 1, size=(N, K))
    C = rng.integers(-100, 100, size=(M, N)).astype(float)
    rc, out = _run(10 + groups, "mk,nk->mn", Ai / 2.0**14, Bi / 2.0**14, C, 2.0, -1.0)
    assert rc == 0
    want = 2.0 * (Ai.astype(float) @ Bi.T.astype(float)) / 2.0**28 - C
    assert np.array_equal(out, want)


def test_infinities_and_nans_reach_their_rows_and_columns_only():
    rng = np.random.default_rng(0)
    A, B = rng.standard_normal((40, 70)), rng.standard_normal((50, 70))
    A[3, 5], B[7, 9] = np.inf, np.nan
    rc, out = _run(3, "mk,nk->mn", A, B, np.zeros((40, 50)))
    assert rc == 0
    bad = np.zeros((40, 50), dtype=bool)
    bad[3, :], bad[:, 7] = True, True
    assert np.array_equal(~np.isfinite(out), bad)


def test_nine_groups_cut_what_the_integer_model_cuts():
    # Sums that cancel to 2^-40 of their terms, where what a level drops (2^-48 of
    # the row scales) is 2^-8 of the result: the finish of the mixed form has to
    # drop what eight 6-bit digits drop.  The leading digits cancel exactly, so
    # the running sums stay near the size of the result and add 8 2^-47 of it.
    rng = np.random.default_rng(11)
    M, N, K = 20, 17, 64
    a, b = rng.standard_normal((M, K // 2)), rng.standard_normal((N, K // 2))
    A = np.concatenate([a, -a * (1 + 2.0 ** -40 * rng.standard_normal(a.shape))], 1)
    B = np.concatenate([b, b], 1)
    rc, out = _run(19, "mk,nk->mn", A, B, np.zeros((M, N)))
    assert rc == 0
    want = ozaki.product(A, B, 9)
    assert np.abs(out - want).max() <= 2.0 ** -30 * np.abs(want).max()


def _base(x, bits, S):
    """Balanced digits of the integers x, those of |x| with its sign, most
    significant first."""
    sign, x, d = np.sign(x), np.abs(x), []
    for _ in range(S - 1):
        r = ((x + (1 << (bits - 1))) & ((1 << bits) - 1)) - (1 << (bits - 1))
        x = (x - r) >> bits
        d.append(r)
    return [(t * sign).astype(float) for t in [x] + d[::-1]]


def _group_sum(DA, DB, g, bits):
    """The pairs of weight 2^(-bits g), exact (integers below 2^53, then a power of two)."""
    S = len(DA)
    return sum(DA[s - 1] @ DB[g - s - 1].T for s in range(max(1, g - S), min(S, g - 1) + 1)).astype(np.longdouble) \
        * np.longdouble(2.0) ** (-bits * g)


# Running sums over the longest product of an (H2O)8 iteration (K = 11628, the
# ladder), in one job: the number of outputs leaves no room for partial results,
# so 130 copies of 32 rows and columns.  An addition rounds the error word, of the
# size of a last place of the sum's (24 bits), to 24 bits of itself, twice:
# sqrt(2 / 12) 2^-48 of the sum at most, 2^-49.5 in the mean over a binade, and n
# of them add up to sqrt(n) that.
_REP, _K = 130, 11628


def test_nine_group_sums_over_a_long_product():
    rng = np.random.default_rng(21)
    A = np.rint(np.clip(0.15 * rng.standard_normal((32, _K)), -0.7, 0.7) * 2.0 ** 48)
    B = np.rint(np.clip(0.15 * rng.standard_normal((32, _K)), -0.7, 0.7) * 2.0 ** 48)
    A[:, 0] = B[:, 0] = 0.75 * 2.0 ** 48                      # row scales 1
    DA, DB = _base(A.astype(np.int64), 6, 8), _base(B.astype(np.int64), 6, 8)
    want = sum(_group_sum(DA, DB, g, 6) for g in range(2, 10))
    M = 32 * _REP
    rc, out = _run(19, "mk,nk->mn", np.tile(A * 2.0 ** -48, (_REP, 1)), np.tile(B * 2.0 ** -48, (_REP, 1)), np.zeros((M, M)))
    assert rc == 0
    assert np.array_equal(out, np.tile(out[:32, :32], (_REP, _REP)))
    err = np.sqrt(np.mean((out[:32, :32] - want) ** 2) / np.mean(want ** 2))
    # 16 blocks of up to 12 k-blocks, a chunk for each of four bands of two groups
    assert err <= np.sqrt(16 * 4 * 2) * 2.0 ** -49.5, np.log2(float(err))


def test_lower_bands_of_the_fp64_level_over_a_long_product():
    # 30-bit operands (four digits: nothing is dropped), neighbouring columns
    # opposite to 2^-17, so that the first band (all but carries of a digit) cancels
    # chunk by chunk and the error of the others' sums shows in the result
    rng = np.random.default_rng(22)
    a = np.rint(np.clip(0.15 * rng.standard_normal((32, _K // 2)), -0.7, 0.7) * 2.0 ** 30)
    b = np.rint(np.clip(0.15 * rng.standard_normal((32, _K // 2)), -0.7, 0.7) * 2.0 ** 30)
    a[:, 0] = b[:, 0] = 0.75 * 2.0 ** 30
    A, B = np.repeat(a, 2, axis=1), np.repeat(b, 2, axis=1)
    A[:, 1::2] = -a + np.rint(0.2 * rng.standard_normal(a.shape) * 2.0 ** 13)
    DA, DB = _base(A.astype(np.int64), 8, 4), _base(B.astype(np.int64), 8, 4)   # of x 2^-2: 32 bits
    band = [_group_sum(DA, DB, g, 8) * 16 for g in range(2, 9)]
    want, lower = sum(band), sum(band[2:])
    M = 32 * _REP
    rc, out = _run(20, "mk,nk->mn", np.tile(A * 2.0 ** -30, (_REP, 1)), np.tile(B * 2.0 ** -30, (_REP, 1)), np.zeros((M, M)))
    assert rc == 0
    err = np.sqrt(np.mean((out[:32, :32] - want) ** 2) / np.mean(lower ** 2))
    # in each block chunks of 5, 3 and 2 k-blocks: 3 + 4 + 6 of them, two groups each
    assert err <= np.sqrt(16 * 13 * 2) * 2.0 ** -49.5, np.log2(float(err))
