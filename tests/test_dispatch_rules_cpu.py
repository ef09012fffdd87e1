"""Rules that choose a kernel or a tile by sizes, at the sizes where they turn.  The times beside them were measured on a B200."""
import types

import pytest

from atlas_b200.ops import cuda as K

SMS = 148


@pytest.mark.parametrize("M,N,Kd,want", [
    (1, 4096, 8192, (128, 4)), (128, 4096, 21504, (128, 4)), (32, 5120, 14336, (128, 3)), (8, 9216, 8192, (128, 2)),      # meet in a cluster
    (1, 512, 8192, (64, 16)), (32, 1024, 14336, (64, 9)), (128, 2048, 8192, (64, 4)), (8, 3072, 8192, (64, 3)),          # narrow: 64-wide tiles
    (32, 4096, 8191, (64, 2)), (129, 4096, 8192, (64, 1)),
])
def test_bf16_decode_products_of_long_k(M, N, Kd, want):
    assert K.gemm_plan(M, N, Kd, 0, SMS) == want


@pytest.mark.parametrize("M,N,Kd,want", [(8192, 12352, 128, 128), (8192, 12352, 136, 256), (8192, 12288, 64, 256), (8192, 1921, 4096, 128)])
def test_bf16_products_whose_last_wide_tile_is_cut_off(M, N, Kd, want):
    assert K.gemm_plan(M, N, Kd, 0, SMS)[0] == want


@pytest.mark.parametrize("M,N,Kd,want", [
    (4500, 12352, 1024, 128), (8192, 18560, 1536, 128),                     # a wide tile of short K costs more than two narrow ones
    (4500, 12352, 2048, 256), (8192, 12352, 2048, 128), (8192, 12352, 4096, 256), (2500, 4992, 2048, 256),
    (1024, 4992, 4096, 128), (300, 18560, 4096, 128), (1024, 6272, 8192, 128),     # two wide waves for three narrow ones
    (1024, 12352, 4096, 256), (517, 12352, 3072, 256),
    (4500, 12288, 1024, 256), (1024, 4864, 1024, 256),                      # whole tiles: as ever
    (500, 4992, 4096, 128),                                                  # fewer wide tiles than SMs
])
def test_fp8_products_whose_last_wide_tile_is_cut_off(M, N, Kd, want):
    assert K.gemm_plan(M, N, Kd, 1, SMS)[0] == want


@pytest.mark.parametrize("ctx,q,seqs,Hq,Hkv,D,most,want", [
    (0, 5, 32, 32, 8, 256, 16, True), (0, 16, 32, 32, 8, 256, 16, True), (0, 17, 32, 32, 8, 256, 16, False),
    (500, 5, 32, 32, 8, 256, 16, False), (0, 5, 32, 16, 2, 256, 16, False), (0, 5, 32, 32, 8, 128, 16, False),
    (0, 5, 32, 32, 16, 256, 8, True), (0, 9, 32, 32, 16, 256, 8, False),
])
def test_many_short_prompts_on_wide_heads(ctx, q, seqs, Hq, Hkv, D, most, want):
    batch = types.SimpleNamespace(seq_lens_host=[9000] + [ctx + q] * seqs, query_lens_host=[1] + [q] * seqs)        # one decode row in front
    assert K._short_prompts_fill_waves(batch, 1, Hq, Hkv, D, SMS, most) is want
