"""Convolution and weight-gradient kernels at the edges of their split into runs
of planes: fewer planes than CTAs, runs of one plane, runs that cross tile
boundaries and wrap the accumulator and plane rings.  Forward activations within
one BF16 ulp of the oracle's, gradients to 1e-4 of their largest magnitude (the
tolerances of test_gpu_closure.py)."""
import numpy as np
import pytest

from oracle import closure_oracle as co
from tests.test_gpu_closure import _bf16_close, _close, _closure, _rand_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 16, 1), (16, 32, 2), (48, 16, 3), (32, 48, 37), (80, 64, 19)],
                         ids=lambda n: "x".join(map(str, n)))
def test_layers_and_gradients(n):
    from multiphysics_fvm_b200 import closure as CL
    rng = np.random.default_rng(5)
    c = _closure(n)
    params = _rand_params(rng)
    c.set_weights(params)
    X0 = np.zeros((n[2], n[1], n[0], 16))
    X0[..., :5] = rng.normal(0, 1, (n[2], n[1], n[0], 5))
    X0 = co.bf16(X0)
    c.set_buffer(CL.CB_X0, X0)
    c.forward()
    (W1, b1), (W2, b2), (W3, b3) = [(co.bf16(w), b.astype(np.float64)) for w, b in params]
    A1, A2 = c.buffer(CL.CB_A1).astype(np.float64), c.buffer(CL.CB_A2).astype(np.float64)
    _bf16_close(A1, co.bf16(co.relu(co.conv3d(X0, W1, b1))), "A1")
    _bf16_close(A2, co.bf16(co.relu(co.conv3d(A1, W2, b2))), "A2")
    _close(c.buffer(CL.CB_Z3), co.conv3d(A2, W3, b3), "Z3")
    import torch
    D = rng.normal(0, 1e-3, (5, n[2], n[1], n[0])).astype(np.float32)
    c.backward(torch.from_numpy(D).cuda(), 2e-3, (1 / n[0], 1 / n[1], 1 / n[2]))
    G3, G2, G1 = (c.buffer(b).astype(np.float64) for b in (CL.CB_G3, CL.CB_G2, CL.CB_G1))
    _bf16_close(G2, co.bf16(co.conv3d_dgrad(G3, W3) * (A2 > 0)), "G2")
    _bf16_close(G1, co.bf16(co.conv3d_dgrad(G2, W2) * (A1 > 0)), "G1")
    for layer, ((dw, db), (X, G)) in enumerate(zip(c.get_grads(), [(X0, G1), (A1, G2), (A2, G3)]), start=1):
        _close(dw, co.conv3d_wgrad(X, G), f"dW{layer}")
        scale = np.abs(G).sum(axis=(0, 1, 2)).max()
        assert np.abs(db - G.sum(axis=(0, 1, 2))).max() <= 1e-6 * scale, f"db{layer}"
