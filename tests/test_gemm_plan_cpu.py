"""Which cluster size shares the K range of a tile, and which launches merge row blocks (host-only queries; no GPU
needed when the residency is given)."""
import ctypes

import pytest

from flydsl_b200 import _lib

B200 = (148, 74, 33, 15)                    # clusters of 1, 2, 4 and 8 CTAs that ran at once on one B200


def ksplit(resident, tokens, n, k, *, topk=1, blocks=None, tile_m=64, stage=2):
    blocks = (tokens + tile_m - 1) // tile_m if blocks is None else blocks
    return _lib.load().flymoe_gemm_ksplit(stage, _lib.SCALE_BLOCK128, tokens, topk, n, k, blocks, tile_m,
                                          ctypes.cast((ctypes.c_int32 * 4)(*resident), ctypes.c_void_p))


def test_few_tiles_of_long_k_are_shared():
    assert ksplit(B200, 64, 2112, 7168) == 8                            # 9 tiles of 56 K blocks
    assert ksplit(B200, 64, 2112, 128) == 1                             # one K block: nothing to share
    assert ksplit(B200, 64, 2112, 7168, tile_m=128) == 1                # 128-row blocks run on one CTA
    assert ksplit(B200, 64 * 148, 2112, 7168) == 1                      # the tiles fill the GPU


@pytest.mark.parametrize("size", [8, 4, 2])
def test_a_size_that_cannot_run_is_not_chosen(size):
    resident = [n if (1 << i) < size else 0 for i, n in enumerate(B200)]
    assert ksplit(resident, 64, 2112, 7168) == size // 2


def test_the_plan_counts_the_clusters_that_run_at_once():
    # 18 tiles of 56 K blocks: one round of 18 clusters of 8, or two where only 15 run at once -- then one round of 4
    assert ksplit((148, 74, 37, 18), 64, 4608, 7168) == 8
    assert ksplit(B200, 64, 4608, 7168) == 4


def test_wait_accounting_is_not_read_for_the_cluster_kernel():
    import bench
    from flydsl_b200 import workloads as wl
    lib, res = _lib.load(), ctypes.cast((ctypes.c_int32 * 4)(*B200), ctypes.c_void_p)
    one_token = wl.MoEConfig("few tiles", 1, 4096, 14336, 8, 2, 0)
    prefill = wl.MoEConfig("many tiles", 4096, 7168, 2048, 256, 8, 0)
    assert "moe_gemm_split_kernel" in bench.shared_k_note(lib, one_token, 16, 2, res)
    assert bench.shared_k_note(lib, one_token, 16, 1, res) is None            # 224 tiles fill the GPU
    assert [bench.shared_k_note(lib, prefill, 128, s, res) for s in (1, 2)] == [None, None]


TINY, MID, WIDE, MANY = (1024, 512, 8, 2), (2048, 1024, 64, 6), (4096, 14336, 8, 2), (7168, 2048, 256, 8)


@pytest.mark.parametrize("dims,tokens,tile_m,merged", [
    # one or two rounds of row blocks: merged, they are one round of tiles several times as long (measured 1.2-1.6x slower)
    (TINY, 64, 16, (0, 0)), (TINY, 192, 16, (0, 0)), (TINY, 192, 32, (0, 0)), (TINY, 512, 16, (0, 0)), (TINY, 768, 64, (0, 0)),
    # several rounds become one
    (TINY, 1024, 16, (1, 1)), (TINY, 2048, 32, (1, 1)), (MID, 512, 16, (1, 1)), (MID, 1024, 64, (1, 1)), (WIDE, 128, 32, (1, 1)),
    # hardly an expert has a second block, and no round is saved
    (MID, 273, 32, (0, 0)), (MID, 546, 64, (0, 0)),
    # weight streaming: the busy experts of skewed routing
    (MANY, 777, 32, (1, 1)), (MANY, 1024, 64, (1, 1)),
    # nothing to merge
    (MANY, 4096, 128, (0, 0)),
])
def test_row_blocks_are_merged_where_it_saves_rounds(dims, tokens, tile_m, merged):
    H, I, E, k = dims
    blocks = (tokens * k + E * tile_m - k + tile_m - 1) // tile_m
    lib = _lib.load()
    got = (lib.flymoe_gemm_merges_blocks(1, tokens, k, E, I, H, blocks, tile_m,
                                         _lib.ROWS_BY_TOKEN if tile_m <= 32 else _lib.ROWS_SORTED, 148),
           lib.flymoe_gemm_merges_blocks(2, tokens, k, E, H, I, blocks, tile_m, _lib.ROWS_SORTED, 148))
    assert got == merged


def test_only_launches_that_the_tile_table_covers_are_merged():
    H, I, E, k = MANY
    lib = _lib.load()
    assert lib.flymoe_gemm_merges_blocks(2, 8192, k, E, H, I, 4096, 16, _lib.ROWS_SORTED, 148) == 1
    assert lib.flymoe_gemm_merges_blocks(2, 8192, k, E, H, I, 4097, 16, _lib.ROWS_SORTED, 148) == 0
    assert lib.flymoe_gemm_merges_blocks(2, 8192, 1, 1, H, I, 512, 16, _lib.ROWS_SORTED, 148) == 0      # one expert: dense
