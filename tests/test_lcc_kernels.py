"""The learned network's gradient where its kernels' tiles end: grids smaller than a
brick along one axis, ragged rows, one and several samples, every number of channels
(the layers), against the mma.sync convolutions, which share neither the row blocks
nor the weight gradient's tap groups with the tcgen05 kernels."""
import numpy as np
import pytest

from falcon_gb300 import lcc
from oracle import lcc_oracle as oracle_lcc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,D,H,W", [(1, 8, 8, 8), (3, 8, 24, 8), (1, 16, 8, 40), (2, 24, 40, 56)])
def test_gradient_of_ragged_grids_matches_mma_sync(built_lib, n, D, H, W):
    rng = np.random.default_rng(7)
    x = rng.standard_normal((n, D, H, W, 8)).astype(np.float32)
    t = rng.standard_normal((n, D, H, W)).astype(np.float32)
    out = []
    for path in (lcc.MMA_SYNC, lcc.TCGEN05):
        net = lcc.LCC(device=0, seed=5)
        net.set_tensor_path(path)
        out.append(net.loss_grad(x, t))
        net.close()
    (l0, g0), (l1, g1) = out
    # the tolerances of the two paths' comparison on its own grid (BF16 roundings that
    # fall the other way after FP32 sums in another order), layer by layer
    assert abs(l1 - l0) <= 2e-3 * l0
    offs = np.cumsum([0] + [co * ci * 27 + co for ci, co in oracle_lcc.LAYERS])
    for l in range(len(oracle_lcc.LAYERS)):
        a, b = g0[offs[l]:offs[l + 1]], g1[offs[l]:offs[l + 1]]
        assert np.linalg.norm(b - a) <= 2e-2 * np.linalg.norm(a), l
