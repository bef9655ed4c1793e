"""What a fused product runs - kernel, tiles, pairs - for its sizes, asked of the library without a device."""
import ctypes

import pytest

from alpaca_lora_4bit_b200 import _lib

RESIDENT = (74, 74, 33, 22, 15)            # a B200: pairs of SMs; clusters of one to four pairs at once
SHAPES = [(4096, 4096), (4096, 1024), (4096, 11008), (11008, 4096), (5120, 5120), (5120, 15360), (5120, 27648), (13824, 5120), (8192, 28672),
          (28672, 8192), (2176, 256), (512, 512)]
ROWS = [1, 17, 32, 77, 128, 250, 256, 257, 270, 288, 289, 320, 321, 333, 352, 384, 385, 500, 512, 513, 700, 800, 1024, 1038, 1100, 1152, 1536, 2048, 4096]
KERNEL, TILE, PAIRS, CLUSTER, CUT, ACT, FIRST = range(7)


def plan(M, K, N, G, act_order, transpose=False, resident=RESIDENT, workspace=None):
    """``G`` groups; a sequential layer's forward comes with its table of zero terms and the promise of its group size."""
    L = _lib.lib()
    out = (ctypes.c_int * 7)()
    dev = None if resident is None else (ctypes.c_int * 5)(*resident)
    size = int(L.q4_gemm_workspace_bytes(K, N, G)) if workspace is None else workspace
    table = not act_order and not transpose
    _lib.check(L.q4_gemm_plan(int(transpose), M, K, N, G, K // G if table else 0, int(table), size, dev, out), "gemm_plan")
    return list(out)


@pytest.mark.parametrize("act_order", [False, True])
def test_tiles_have_heights_that_the_mma_takes(act_order):
    """An MMA of a CTA pair with A in tensor memory takes N in steps of 32, up to 256; tiles above 256 rows are two MMAs.
    (In halves, tiles of 288 and 352 rows came to N = 144 and 176.)"""
    tall = 0
    for K, N in SHAPES:
        for M in ROWS:
            p = plan(M, K, N, K // 128, act_order)
            if p[KERNEL] != 4:
                continue
            rows, first = p[TILE], p[FIRST]
            assert 0 < rows <= 384 and (first == rows if rows <= 256 else first >= rows - first > 0), (M, K, N, p)
            assert first % 32 == 0 and first <= 256 and (rows - first) % 32 == 0, (M, K, N, p)
            tall += rows > 256
    assert tall > 20


@pytest.mark.parametrize("resident", [(74, 70, 33, 20, 13), (74, 61, 30, 20, 15), (74, 0, 0, 0, 0), RESIDENT])
def test_pairs_that_wait_for_one_another_are_resident_together(resident):
    """A pair that adds a tile up waits for the sums of others: with more pairs in the launch than the device holds at once it
    can keep an SM from the one it waits for.  (The number of pairs was half the number of SMs, whatever fits.)"""
    cut = 0
    for act_order in (False, True):
        for K, N in SHAPES:
            for M in ROWS:
                p = plan(M, K, N, K // 128, act_order, resident=resident)
                if p[KERNEL] != 4 or not p[CUT]:
                    continue
                cut += 1
                held = resident[p[CLUSTER]] * p[CLUSTER]
                assert p[PAIRS] <= held, (M, K, N, p)
    assert (cut > 20) == (resident[1] > 0)


@pytest.mark.parametrize("M,K,N,act_order,transpose,want", [
    (257, 9728, 3584, False, True, dict(KERNEL=2)),               # 49 us in two 256-row tiles, 57 in one of 512
    (257, 3584, 9728, False, True, dict(KERNEL=2)),               # 56 and 78
    (1800, 2048, 5632, True, True, dict(KERNEL=3)),               # 66 us in 512-row tiles, 74 in 256
    (1600, 5120, 5120, False, True, dict(KERNEL=2)),              # 84 in 256, 93 in 512
    (4096, 8192, 1024, True, True, dict(KERNEL=3, CUT=0)),        # whole tiles 84 us, dealt 107
    (1100, 11008, 4096, False, False, dict(KERNEL=4, CUT=1)),     # 84 us dealt; 94 in whole tiles of 288 rows
    (2500, 8192, 8192, False, False, dict(KERNEL=4, CUT=1)),      # 267 us dealt; 306 in whole tiles of 288 rows
    (1200, 11008, 4096, True, False, dict(KERNEL=4, ACT=1)),      # 110 us; the pair kernel 129
    (128, 8192, 1024, True, False, dict(KERNEL=4, ACT=1)),        # 29 us; 18 pairs a tile of the pair kernel 100
])
def test_choices_that_were_measured(M, K, N, act_order, transpose, want):
    p = plan(M, K, N, K // 128, act_order, transpose)
    assert {k: p[globals()[k]] for k in want} == want, p
