"""The FP64 form where memory is short: its contractions run on the tensor cores
only while their packed operands can be had, and on the FP64 pipe otherwise, with
the same results."""
import numpy as np
import pytest

from conftest import inputs

pytestmark = pytest.mark.gpu


def _steps(limit, waters=4):
    """Two FP64 iterations on a new context that may hold `limit` bytes of packed operands."""
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 2)
    ctx = Context(inputs(waters))
    assert lib.fcc_test_set_scratch(ctx.h, limit) == 0
    r = RCCSD.compute(inputs(waters), context=ctx)
    Options.reset()
    return ctx, r, lib.fcc_test_products(ctx.h), lib.fcc_test_scratch_held(ctx.h)


def test_contractions_keep_to_the_scratch_there_is():
    ctx, ref, most, held = _steps(-1)
    ctx.close()
    assert most > 0 and held > 0
    for limit in (0, held // 7, held // 2, held):
        ctx, r, products, now = _steps(limit)
        ctx.close()
        assert now <= limit and products <= most, (limit, now)
        assert (products == 0) == (limit == 0) and (limit < held or products == most)
        # both routes are at the level of one FP64 rounding of sums of a few thousand terms
        assert np.abs(r.T1 - ref.T1).max() < 1e-13 and np.abs(r.T2 - ref.T2).max() < 1e-13
        assert abs(r.correlation - ref.correlation) < 1e-12


def test_kept_operands_count():
    # the ladder's A operands are packed once and kept beside the other packed
    # operands: limits all over the range, some of which only they exceed
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 1)
    held, energies = [], []
    for step in range(-1, 48):
        ctx = Context(inputs(4))
        limit = -1 if step < 0 else held[0] * step // 48
        assert lib.fcc_test_set_scratch(ctx.h, limit) == 0
        energies.append(RCCSD.compute(inputs(4), context=ctx).correlation)
        held.append(lib.fcc_test_scratch_held(ctx.h))
        ctx.close()
        assert limit < 0 or held[-1] <= limit, (limit, held[-1])
    Options.reset()
    assert np.ptp(energies) < 1e-12
