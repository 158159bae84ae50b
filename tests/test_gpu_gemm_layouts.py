"""The operand layouts of the training kernel's matrix products on one tile: a layer forward (both operands K-major),
dh = dz W (W read MN-major) and dW = dz^T h (both MN-major), against FP64 products of the same BF16 values: 128 products
of unit normals in FP32, 1e-5 relative and 1e-4 absolute as for the forward layout."""
import numpy as np
import pytest

from photonprop_b200 import _lib, surrogate as sg
from oracle import mlp as omlp
from test_gpu_surrogate import _bf16_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_layout(layout):
    rng = np.random.default_rng(layout + 10)
    a, b = rng.normal(size=(2, 128, 128)).astype(np.float32)
    c = sg.gemm_selftest(_bf16_bits(a), _bf16_bits(b), layout=layout)
    x, y = omlp.bf16(a), omlp.bf16(b)
    want = (x @ y.T, x @ y, x.T @ y)[layout]
    np.testing.assert_allclose(c, want, rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("layout", [-1, 3])
def test_unknown_layout_is_refused(layout):
    z = np.zeros((128, 128), dtype=np.uint16)
    with pytest.raises(_lib.PPError):
        sg.gemm_selftest(z, z, layout=layout)
