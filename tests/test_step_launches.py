"""The benchmark's count of our kernel launches in a steady step follows the engine's choices."""
import pytest

import bench


@pytest.mark.parametrize("sizes,fft,count", [
    ([32], "native", 7),                      # node sums: no fix-up
    ([64], "native", 7),
    ([32] * 16, "native", 7),                 # 2^19 cells, the last that adds node sums
    ([32] * 17, "native", 8),
    ([64, 64], "native", 7),
    ([64, 64, 32], "native", 11),             # two mesh sizes and a fix-up
    ([32, 64], "native", 10),
    ([128], "native", 8),
    ([32, 128], "native", 11),
    ([256], "native", 10),
    ([512], "native", 10),
    ([32, 64, 128, 256], "native", 19),       # the batched ensemble
    ([16], "native", 6),                      # cuFFT (not ours) and the Green kernel
    ([16, 32], "native", 9),
    ([32], "cufft", 6),
    ([64, 256], "cufft", 6),
])
def test_launches_of_a_steady_step(sizes, fft, count):
    assert bench.step_launches(sizes, fft) == count
    assert bench.step_launches(sizes, fft, True) == count + 1
