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
