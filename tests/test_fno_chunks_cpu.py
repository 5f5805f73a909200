"""How the learned guess splits its weight gradients.

The chunk divides a sample's points; problems too small to fill the GPU at
2048 points a product take smaller ones, the others keep 2048: the buffer of
partial sums grows with the number of products, and the FP32 GEMM takes 65535
of them at most."""
import pytest

from fortress_b200.fno import GRADIENT_PRODUCTS, gradient_chunk


@pytest.mark.parametrize("n,batch", [(16, 1), (32, 7), (64, 64), (100, 3), (96, 20), (128, 16), (256, 1), (256, 8), (256, 64),
                                     (256, 512), (256, 2000), (48, 5)])
def test_chunks(n, batch):
    points = n * n
    chunk = gradient_chunk(batch, points)
    assert points % chunk == 0
    products = batch * points // chunk
    coarse = points
    while coarse > 2048 and coarse % 2 == 0:
        coarse //= 2
    at_2048 = batch * points // coarse
    if at_2048 >= GRADIENT_PRODUCTS:
        assert chunk == coarse                  # already enough of them
    else:
        assert products < 2 * GRADIENT_PRODUCTS and chunk <= coarse
    if at_2048 <= 65535:
        assert products <= 65535


def test_small_problems_fill_the_gpu():
    assert gradient_chunk(64, 64 * 64) == 512
