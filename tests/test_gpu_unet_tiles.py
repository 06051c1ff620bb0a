"""The network's forward and gradients at sizes whose levels do not fill the
tensor-core kernels' pixel tiles (8 -> 1 pixel at the lowest level, widths that
are not multiples of 8, 16 or 128), on the exactly representable case of
test_gpu_unet.py and with its tolerances."""
import numpy as np
import pytest

from test_gpu_unet import EXACT_GRAD_TOL, EXACT_TOL, _compare, _sparse_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,batch", [(8, 1), (40, 3), (72, 2), (136, 1), (256, 1)])
def test_ragged_sizes_match_oracle(gb, size, batch):
    from oracle import unet_ref

    layers, n = unet_ref.layer_table()
    rng = np.random.default_rng(size + 31)
    params = _sparse_params(layers, n, rng)
    x = rng.integers(0, 4, (batch, size, size)).astype(np.float64)
    dout = rng.integers(-1, 2, (batch, size, size)).astype(np.float64)
    e_fwd, errs = _compare(gb, size, batch, params, x, dout)
    assert e_fwd <= EXACT_TOL
    assert max(errs.values()) <= EXACT_GRAD_TOL, errs
