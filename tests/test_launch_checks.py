"""What is decided before a launch: arguments that are refused (plain integers stand for device pointers, so no GPU is needed, and
where one is there, nothing is launched) and choices by size."""
import pytest

from omegalax_b200.ops import lib

A = 1 << 20      # an aligned address that is never read


@pytest.mark.parametrize("h,out,D,code", [(A + 2, A, 64, 6002), (A, A + 8, 64, 6002), (A, A, 60, 6001)])
def test_row_gather_of_the_head_wants_16_byte_rows(h, out, D, code):
    """A contiguous view may start anywhere; the gather reads 16 bytes at a time, as the products it stands before do."""
    assert lib.load().ob_ce_gather(h, A, A, out, 128, D, None) == code


@pytest.mark.parametrize("batch,rows,H,G,hd,causal,least,most", [
    (7, 512, 32, 8, 128, True, 1, 1), (4, 800, 32, 8, 128, True, 1, 1), (7, 512, 32, 4, 128, False, 1, 1), (2, 1000, 16, 8, 128, False, 1, 1),
    (1, 4096, 32, 8, 128, True, 1, 1), (2, 4096, 32, 8, 128, True, 1, 1), (1, 128, 16, 8, 128, True, 1, 1),
    (1, 4096, 32, 4, 128, True, 2, 4), (1, 3001, 32, 2, 256, True, 4, 8), (1, 512, 64, 4, 128, False, 8, 8), (1, 1000, 16, 8, 128, True, 2, 2)])
def test_ctas_share_a_key_tile_only_where_that_saves(batch, rows, H, G, hd, causal, least, most):
    """Sizes at which sharing was measured to lose, and to win by the factors named in ``attn_bwd_splits``."""
    from omegalax_b200.ops import kernels as K

    tiles = min(-(-rows // 128) * batch, batch * rows // 128 + batch) * (hd // 128)
    assert least <= K.attn_bwd_splits(tiles, H, G, -(-rows // 64), causal, batch * rows * G * hd) <= most


@pytest.mark.parametrize("M,N,K,few", [(1, 8, 64, True), (64, 4096, 32, True), (65, 4096, 512, False), (2048, 1024, 768, False), (500, 6144, 768, True),
                                       (2048, 1024, 1024, True), (1000, 6144, 4096, False), (128, 151936, 4096, True)])
def test_products_of_few_rows_go_where_they_are_faster(M, N, K, few):
    from omegalax_b200.ops import kernels

    assert kernels._use_few(M, N, K) is few


@pytest.mark.parametrize("rows,tiles,chunk", [(8192, 4, 4096), (32768, 4, 8192), (16384, 16, 1024), (4096, 64, 1024), (3000, 8, 4096),
                                              (2559, 4, 1024), (100, 8, 1024), (24000, 12, 2000)])
def test_more_tiles_than_the_default_bound_the_memory_of_the_head(rows, tiles, chunk):
    from omegalax_b200.trainers.loss import chunk_rows

    assert chunk_rows(rows, tiles) == chunk
