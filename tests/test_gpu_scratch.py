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


@pytest.mark.parametrize("waters", [1, 2])
def test_triples_forms_agree(waters):
    # the contractions of the joined operands, their slices (whole and by runs) and
    # the contractions that read the operands where they are, on one system; (T) is
    # a sum of about 1e5 to 1e7 terms with cancellations of a decade
    import ctypes
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    inp = inputs(waters)
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 2)
    ctx = Context(inp)
    RCCSD.compute(inp, context=ctx)
    ijk = np.array([(i, j, k) for i in range(inp.o) for j in range(i + 1) for k in range(j + 1) if not i == j == k][:7], np.int32)
    whole, each = {}, {}
    for form, kc in ((1, 0), (1, 3), (2, 0), (2, 3), (3, 0), (3, 3)):
        assert lib.fcc_test_set_t3_form(ctx.h, form) == 0 and lib.fcc_test_set_t3_kc(ctx.h, kc) == 0
        n0 = lib.fcc_stat_launches()
        whole[form, kc] = ctx.triples(_lib.FCC_PREC_FP64)
        e = np.zeros(len(ijk))
        assert lib.fcc_test_triples_subset(ctx.h, ijk.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), len(ijk),
                                           e.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
        each[form, kc] = e
        assert lib.fcc_stat_launches() > n0
    # without a hook a system that may hold no slices takes the third form
    assert lib.fcc_test_set_t3_form(ctx.h, 0) == 0 and lib.fcc_test_set_t3_kc(ctx.h, 0) == 0
    assert lib.fcc_test_set_scratch(ctx.h, 0) == 0
    whole["limit"] = ctx.triples(_lib.FCC_PREC_FP64)
    ctx.close()
    Options.reset()
    ref = whole[2, 0]
    assert all(abs(w - ref) < 1e-12 * abs(ref) for w in whole.values()), whole
    assert all(np.abs(e - each[2, 0]).max() < 1e-12 * abs(ref) for e in each.values()), each


def test_a_triples_without_room_for_slices_takes_none():
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    inp = inputs(2)
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 1)
    ctx = Context(inp)
    assert lib.fcc_test_set_scratch(ctx.h, 0) == 0
    RCCSD.compute(inp, context=ctx)
    prof = np.zeros(24)
    import ctypes
    lib.fcc_prof_enable(1)
    ctx.triples(_lib.FCC_PREC_FP64)
    lib.fcc_prof_enable(0)
    assert lib.fcc_prof_read(prof.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 6) == 0
    ctx.close()
    Options.reset()
    assert prof[4 * 5] == 0 and prof[4 * 2] == 0 and prof[4 * 0] > 0   # no exact-slice product, no packing


@pytest.mark.parametrize("precision", ["fp64", "exact", "mixed"])
def test_what_a_call_leaves_is_bounded_and_given_back(precision):
    from fermicc import Options, RCCSD, _lib
    from fermicc.rccsd import Context
    inp = inputs(4)
    lib = _lib.load()
    Options.reset()
    Options.set("cc_max_iter", 2)
    Options.set("cc_gpu_precision", precision)
    ctx = Context(inp)

    def steps():
        assert lib.fcc_set_guess(ctx.h, None, None) == 0
        return RCCSD.compute(inp, context=ctx).correlation, lib.fcc_test_scratch_held(ctx.h)
    e, held = steps()
    assert held > 0
    # an allocation that finds no memory gets it, but not from under a product
    assert lib.fcc_test_reclaim(ctx.h, 1) == 0 and lib.fcc_test_scratch_held(ctx.h) == held
    assert lib.fcc_test_reclaim(ctx.h, 0) == 1 and lib.fcc_test_scratch_held(ctx.h) == 0
    assert lib.fcc_test_reclaim(ctx.h, 0) == 0
    for keep in (0, held - 1, held):
        assert lib.fcc_test_set_scratch_keep(ctx.h, keep) == 0
        for _ in range(2):
            e2, now = steps()
            assert now <= keep and abs(e2 - e) < 1e-10
    assert lib.fcc_test_set_scratch_keep(ctx.h, -1) == 0
    ctx.close()
    Options.reset()
