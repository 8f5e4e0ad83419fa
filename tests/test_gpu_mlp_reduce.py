"""The sum of the gradient's per-CTA partials (k_mlp_reduce) where fewer bits or a smaller range than FP64's would
show: an infinite partial, partial sums beyond FP32's range that come back, and a cancellation that
leaves one bit 51 places below the largest partial.  The last layer's bias gradient is the sum
of dy, and a CTA takes 64 rows, so every partial is chosen here and the sum is exact in FP64.
"""
import numpy as np
import pytest
import torch

from cudaprotoplanetarydisks_gb300.learned import MLP, NIN
from oracle import mlp_ref

pytestmark = pytest.mark.gpu
TILES = 40


def bias_gradient(partials):
    """Gradient of the first output's bias, and of the second's, whose partials are all 1."""
    n = 64 * TILES
    dy = torch.zeros((n, 2))
    dy[::64, 1] = 1.0
    for tile, v in partials.items():
        dy[64 * tile, 0] = v
    m = MLP(n, seed=1)
    m.backward(torch.zeros((n, NIN), dtype=torch.bfloat16, device="cuda"), dy.cuda())
    g = m.grad()
    m.close()
    return g[mlp_ref.OFF_B3], g[mlp_ref.OFF_B3 + 1]


BIG = float(torch.tensor(2e38).bfloat16())  # what dy is rounded to


@pytest.mark.parametrize("partials,want", [
    ({3: np.inf}, np.inf), ({3: -np.inf, 11: 1.0}, -np.inf), ({0: np.inf, 9: -np.inf}, np.nan), ({5: np.nan}, np.nan),
    ({0: BIG, 8: BIG}, np.inf), ({0: BIG, 8: BIG, 16: -BIG}, BIG), ({0: BIG, 1: BIG, 2: -BIG}, BIG),
    ({0: 2.0 ** 20, 8: 2.0 ** -6, 16: 2.0 ** -31, 24: -2.0 ** 20, 32: -2.0 ** -6}, 2.0 ** -31),
    ({0: 2.0 ** 20, 1: 2.0 ** -6, 2: 2.0 ** -31, 3: -2.0 ** 20, 4: -2.0 ** -6}, 2.0 ** -31)])
def test_partials_are_summed_as_in_fp64(partials, want):
    got, other = bias_gradient(partials)
    assert got == np.float32(want) or (np.isnan(got) and np.isnan(want)), got
    assert other == TILES
