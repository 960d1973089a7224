"""The plan of the W4 GEMM (make_plan), on the CPU: how the (tile, 256-input chunk) steps are dealt to pairs of SMs."""
import ctypes as C

import pytest

from llama_cu_awq_b200 import _lib

PAIRS = 74   # 148 SMs


def _plan(M, K, N):
    L = _lib.test_lib()
    mt, pairs = C.c_int(), C.c_int()
    assert L.q4_test_gemm_plan(M, K, N, 2 * PAIRS, C.byref(mt), C.byref(pairs)) == 0
    return mt.value, pairs.value


def _most_parts(tiles, chunks, pairs):
    """The most pairs that work on one tile: step c belongs to pair ((c + 1) * pairs - 1) / total (pair_of)."""
    total = tiles * chunks
    pair = lambda c: ((c + 1) * pairs - 1) // total
    return max(pair(t * chunks + chunks - 1) - pair(t * chunks) + 1 for t in range(tiles))


# the 11008-input projection has 43 chunks, a prime: no number of pairs deals out equal shares that are a whole part of a tile
@pytest.mark.parametrize("K,N", [(4096, 4096), (4096, 12288), (4096, 22016), (11008, 4096), (5120, 5120), (5120, 15360), (13824, 5120), (8192, 8192), (8192, 10240),
                                 (28672, 8192), (11008, 8192), (8192, 5120), (2944, 2504), (640, 264)])
def test_no_more_parts_than_the_longest_share_asks_for(K, N):
    """Of all numbers of pairs with the same longest share, the plan's cuts its tiles into the fewest parts."""
    up = lambda a, b: -(-a // b)
    for M in (17, 48, 64, 77, 128, 200, 256, 333, 512, 777, 1024, 2000):
        mt, pairs = _plan(M, K, N)
        tiles, chunks = up(N, 256) * up(M, mt), up(K, 256)
        total = tiles * chunks
        assert 1 <= pairs <= min(PAIRS, total) and mt % 32 == 0 and 32 <= mt <= 256
        same = [p for p in range(1, min(PAIRS, total) + 1) if up(total, p) == up(total, pairs)]
        assert _most_parts(tiles, chunks, pairs) == min(_most_parts(tiles, chunks, p) for p in same), (M, mt, pairs)


@pytest.mark.parametrize("M,K,N", [(700, 28672, 8192), (1200, 28672, 8192), (1200, 8192, 57344), (1200, 8192, 10240), (1200, 4096, 22016)])
def test_long_prompts_take_few_tall_tiles(M, K, N):
    """Rows in more tiles than they need cost the weights' conversion again: measured 2 to 7 % on these shapes."""
    mt, _ = _plan(M, K, N)
    assert -(-M // mt) == -(-M // 256), mt
