"""How products are cut over their inner dimension (host code of the kernel library, no GPU): those of few tokens
(``cw_gemm_tc_plan``), and those of a few hundred whose splits are kept apart for the next norm to add up (``cw_gemm_tc_parts_plan``): splits cut the
inner dimension into equal runs of whole 64-element blocks, never shorter than eight blocks, at most eight
of them, and only for token counts that the CTA-pair kernel takes this way."""

import ctypes
import random
import shutil

import pytest

from clockwork_b200.ops.library import library


def kernel_library():
    try:
        return library()  # (built at first use; the plans are host code and need no GPU)
    except Exception as err:  # noqa: BLE001
        if shutil.which("nvcc") is None:
            pytest.skip(f"the kernel library is not built and there is no nvcc here: {err}")
        raise


def plan(t, n, k, sms=148):
    lib = kernel_library()
    lib.cw_gemm_tc_parts_plan.argtypes = [ctypes.c_int] * 4 + [ctypes.POINTER(ctypes.c_int)]
    lib.cw_gemm_tc_parts_plan.restype = ctypes.c_int
    splits = ctypes.c_int(-1)
    assert lib.cw_gemm_tc_parts_plan(t, n, k, sms, ctypes.byref(splits)) == 0
    return splits.value


def test_splits_are_equal_runs_of_whole_blocks():
    rng = random.Random(3)
    seen = set()
    for _ in range(2000):
        t = rng.choice([129, 130, 192, 256, 257, 300, 512, 700, 1000, 1024])
        n = rng.choice([256, 1536, 2048, 3584, 5120, 1000, 130 * 4])
        k = rng.choice([512, 1536, 8960, 18944, 27648, 3584, 5120, 200, 264, 72 * 8])
        splits = plan(t, n, k)
        blocks = -(-k // 64)
        assert 1 <= splits <= 8 and blocks % splits == 0 and (splits == 1 or blocks // splits >= 8), (t, n, k, splits)
        seen.add(splits)
    assert len(seen) > 2  # (the sizes above do get cut in several ways)
    assert plan(256, 1536, 8960) > 1  # the down projection of the 1.5B layer at a few hundred tokens


@pytest.mark.parametrize("t", [545, 600, 640, 700, 768])
def test_slabs_do_not_run_in_rounds_that_cost_more_than_they_save(t):
    """The down product of the 7B layer: its tiles fill most pairs once, and four splits of each would run in two rounds and more."""
    assert plan(t, 3584, 18944) == 1 and plan(t, 4096, 14336) == 1
    assert plan(t, 1536, 8960) > 1  # (few tiles, a long inner dimension)


def test_other_token_counts_are_not_cut():
    for t in (1, 8, 64, 128, 1025, 2048, 4096):
        assert plan(t, 1536, 8960) == 1
    assert plan(256, 1536, 8960, sms=1) == 1


def few_token_plan(t, n, k, swiglu=False, sms=148):
    """(splits, CTAs that share an SM) of a product of few tokens."""
    lib = kernel_library()
    lib.cw_gemm_tc_plan.argtypes = [ctypes.c_int] * 5 + [ctypes.POINTER(ctypes.c_int)] * 3
    lib.cw_gemm_tc_plan_per_sm.argtypes = [ctypes.c_int] * 5
    bn, splits, ctas = (ctypes.c_int() for _ in range(3))
    assert lib.cw_gemm_tc_plan(t, n, k, swiglu, sms, ctypes.byref(bn), ctypes.byref(splits), ctypes.byref(ctas)) == 0
    return splits.value, lib.cw_gemm_tc_plan_per_sm(t, n, k, swiglu, sms)


@pytest.mark.parametrize("t,n,k,swiglu,want", [
    (8, 2048, 2048, False, (8, 2)), (16, 3584, 18944, False, (5, 2)), (32, 4608, 3584, False, (4, 2)), (64, 3500, 3584, False, (5, 2)),
    (64, 1536, 8960, False, (8, 1)),                                     # twelve clusters of eight find a place each
    (65, 3584, 3584, False, (4, 1)), (128, 4608, 3584, False, (3, 1)),   # more tokens: fewer parts
    (8, 3584, 2048, True, (4, 1)), (64, 4608, 2048, True, (3, 1)),       # gated products as well, whatever the tokens
    (8, 9000, 2048, False, (2, 1)), (1, 17920, 1536, False, (1, 1)),
])
def test_splits_of_few_tokens_are_the_same_on_every_part(t, n, k, swiglu, want):
    """The order of a product's sums follows from its sizes and the number of SMs, not from what the driver of a machine (or one
    without a GPU) says about the places of clusters."""
    assert few_token_plan(t, n, k, swiglu) == want


def test_splits_of_few_tokens_find_a_place_at_once():
    places = {1: [0, 148, 74, 45, 33, 26, 22, 15, 15], 2: [0, 296, 148, 93, 71, 56, 45, 37, 33]}
    seen = set()
    for tiles in range(1, 75):
        for t in (1, 17, 33, 65):
            for swiglu in (False, True):
                splits, per_sm = few_token_plan(t, 128 * tiles, 8192, swiglu)
                if t == 65 and swiglu:
                    assert splits == 1  # (two accumulators of 128 tokens leave no room to exchange parts)
                assert tiles <= places[per_sm][splits]
                seen.add((t <= 64, swiglu, per_sm))
    assert seen == {(True, False, 1), (True, False, 2), (True, True, 1), (False, False, 1), (False, True, 1)}
