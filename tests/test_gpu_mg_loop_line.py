"""The one-launch multigrid loop near its upper lines against the separate kernels: the largest volume with coarse levels, the
largest without, a long narrow one with more chunks of two layers than sums have parts, and one with water in few layers.
Tolerance as in test_gpu_mg_loop: only the order of the f64 sums differs."""
import pytest

from test_gpu_mg_loop import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(128, 64, 48), (96, 64, 64), (64, 128, 48), (100, 101, 100), (24, 160, 48), (24, 160, 96),
                                   (2, 4, 1000), (16, 2000, 8), (64, 8, 700)])
def test_one_launch_matches_the_separate_kernels(shape):
    compare(shape)
