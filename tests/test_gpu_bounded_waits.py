"""The bounded waits of the exact-slice GEMM (single CTAs and pairs), of the
grouped (T) GEMM and of the (T) energy kernel: without loads nothing is in flight
and nothing arrives, the waits (2 s) give up, the kernel returns with the error
flag set, and the next call is as usual.  Nothing here faults the GPU."""
import numpy as np
import pytest

from conftest import inputs
from test_gpu_contract import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [100, 256])          # single CTAs, pairs
@pytest.mark.parametrize("silent,normal", [(30, 19), (31, 20)])
def test_exact_slice_gemm(M, silent, normal):
    from fermicc import _lib
    rng = np.random.default_rng(M)
    A, B, C = rng.standard_normal((M, 70)), rng.standard_normal((90, 70)), np.zeros((M, 90))
    rc, _ = _run(silent, "mk,nk->mn", A, B, C)
    assert rc == _lib.FCC_ERR_TIMEOUT
    rc, out = _run(normal, "mk,nk->mn", A, B, C)
    assert rc == 0 and np.abs(out - A @ B.T).max() < 1e-12 * np.abs(out).max()


@pytest.mark.parametrize("kind", ["T3", "ENERGY"])
def test_mixed_triples(kind):
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    import ctypes
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 2)
    ctx = Context(inputs(1))
    RCCSD.compute(inputs(1), context=ctx)
    want = ctx.triples(_lib.FCC_PREC_MIXED)
    assert lib.fcc_test_inject(ctx.h, getattr(_lib, "FCC_TEST_FAULT_NO_LOADS_" + kind)) == 0
    et = ctypes.c_double()
    assert lib.fcc_triples(ctx.h, _lib.FCC_PREC_MIXED, ctypes.byref(et)) == _lib.FCC_ERR_TIMEOUT
    assert ctx.triples(_lib.FCC_PREC_MIXED) == want
    ctx.close()
    Options.reset()
