"""Edges of the dispatch and of the kernels' partitions, against the CPU oracle on the same seeded inputs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from berth_b200 import kernels, synth   # noqa: E402
from tests.gpu_util import assert_close, run_linear   # noqa: E402


def test_integer_path_one_hot_blocks(oracle):
    """An input with one element per 128-block rotates to blocks whose values are all alike; a block's product with the
    weights' byte sums (128 x 510 x 32512 on average) then lies around 2^31."""
    K, N, bits, cb = 512, 2048, 4, 2
    w = synth.linear_weights(1234, "onehot", K, N, bits)
    x = np.zeros((1, K), np.float16)
    x[0, ::128] = [1.0, -2.0, 0.5, 3.0]
    c, _ = run_linear(x, w, bits, cb, True)
    assert "k_exl3_gemv_i8" in kernels.last_launch()
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, cb), "one-hot blocks")


@pytest.mark.parametrize("bits", [3, 4, 5, 6])
@pytest.mark.parametrize("K,N", [(128, 128 * 301), (384, 256 * 160 + 128)])
def test_integer_path_several_band_groups_per_cta(oracle, K, N, bits):
    """So many columns that a CTA holds whole band groups and meets every 128-block of the row again and again."""
    w = synth.linear_weights(1234, f"wide{K}{bits}", K, N, bits)
    x = synth.activations(1234, f"wide{K}.x", 1, K)
    c, _ = run_linear(x, w, bits, 2, True)
    assert "k_exl3_gemv_i8" in kernels.last_launch() and "fused" in kernels.last_launch()
    assert_close(c, oracle.linear_f64(x, w["trellis"], w["suh"], w["svh"], K, N, bits, 2), "wide")
    assert kernels.device_status(torch.cuda.current_device()) == 0
