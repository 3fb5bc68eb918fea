"""The weight gradients' FP32 sums over the nodes of a large mesh, on a network
whose activations are the same at every node: each entry of the last layer's
gradients is then one product times the number of nodes."""
import numpy as np
import pytest

from proteuscfd_gb300 import SolutionSpace, cases
from proteuscfd_gb300 import _native as N

pytestmark = pytest.mark.gpu

L0, LAYER, H = 768, 8576, 64                  # first layer's offset, a layer's length, channels
CE, WS, WM, B = 256, 320, 4416, 8512          # a layer's gate constants, matrices and bias
WOUT = L0 + 3 * LAYER


def bf16(a):
    """float32 rounded to bfloat16 (to nearest, ties to even)"""
    u = np.asarray(a, np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7fff + ((u >> 16) & 1)) & 0xffff0000).astype(np.uint32).view(np.float32)


def test_weight_gradient_sums_of_a_large_mesh():
    """Zero matrices and positive biases: every node has the layers' biases as its
    activations, gates of 1 make the gathered mean the same, and only the first
    output reads them.  A product of two BF16 values has 16 significant bits, so
    a run of 256 nodes sums without a rounding; after it come at most 6 additions
    of runs in a block of 403,200 / 304 nodes and 38 + 8 of blocks, all of one
    sign: (6 + 38 + 8) * 2^-24 = 3.1e-6 of the entry."""
    c = cases.ns_flatplate(80, 72, 70, seed=3)
    m = cases.build_mesh(c)
    n = m.nnode
    S = SolutionSpace(m, c.param)
    S.lp_init(3)
    rng = np.random.default_rng(4)
    w = np.zeros(N.LP_NPARAM, np.float32)
    w[704:768] = bf16(rng.uniform(1, 2, H))
    for k in range(3):
        o = L0 + k * LAYER
        w[o + CE:o + WS] = 1.0
        w[o + B:o + LAYER] = bf16(rng.uniform(1, 2, H))
    w[WOUT:WOUT + H] = bf16(rng.uniform(0.1, 1, H))
    S.lp_set_params(w)
    x = rng.normal(size=(n, N.LP_NIN)).astype(np.float32)
    out = S.lp_forward(x)
    assert np.all(out == out[0])
    t = np.tile(out[0] - np.float32(3.0), (n, 1)).astype(np.float32)
    _, g = S.lp_loss_grad(x, t)
    d = np.float32(np.float32(2.0) / (np.float32(5.0) * np.float32(n))) * (out[0, 0] - t[0, 0])
    dz = bf16(w[WOUT:WOUT + H] * d).astype(np.float64)
    h = w[L0 + LAYER + B:L0 + 2 * LAYER].astype(np.float64)
    exact = n * np.outer(dz, h)
    last = g[L0 + 2 * LAYER:L0 + 3 * LAYER].astype(np.float64)
    for o in (WS, WM):
        got = last[o:o + H * H].reshape(H, H)
        assert np.abs(got / exact - 1.0).max() <= 3.1e-6
    assert np.abs(last[B:] / (n * dz) - 1.0).max() <= 3.1e-6
    S.close()
