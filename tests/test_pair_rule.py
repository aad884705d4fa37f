"""Which products of many rows go to pairs of SMs: gated ones by the fill of their waves of tiles of 256 rows by 128 features, experts'
by how their runs fill tiles of 256 rows."""
import pytest

PAIRS = 74


@pytest.mark.parametrize("rows,features,inner,want", [
    (1536, 128, 1024, False), (1536, 1024, 2048, False), (2048, 1024, 2048, False),      # parts of a wave
    (1536, 1536, 2048, True), (3000, 768, 1024, True),                                    # 72 tiles
    (2048, 1536, 2048, False), (3000, 1024, 1024, False),                                 # 96: a second wave that is mostly empty
    (2048, 2048, 2048, True), (4096, 1536, 1024, True),                                   # 128 and 192
    (2048, 1536, 4096, False), (2048, 6144, 4096, False), (1536, 12288, 4096, False),     # a large inner size takes many waves
    (4096, 6144, 4096, True), (2048, 12288, 4096, True), (8192, 12288, 4096, True),
    (1535, 12288, 2048, False), (8192, 12288, 4097, False), (8192, 17408, 5120, False)])
def test_pair_tiles_fill(rows, features, inner, want):
    from llmserver_b200.ops import gemm_bf16
    assert gemm_bf16.pair_tiles_fill(rows, features, inner, PAIRS) is want
    assert not gemm_bf16.pair_tiles_fill(rows, features, inner, 0)


@pytest.mark.parametrize("experts", [1, 64])
def test_expert_tiles(experts):
    from llmserver_b200.parts.moe import RoutedExperts
    large = {per: RoutedExperts.pair_tiles(per * experts, experts) for per in (1, 128, 159, 160, 192, 256, 257, 320, 383, 384, 512, 4096)}
    assert large == {per: per in (160, 192, 256, 384, 512, 4096) for per in large}
