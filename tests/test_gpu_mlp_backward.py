"""The backward pass at the edges of its 128-row tiles, 32-row column sums and
split-K shares, and its operands off the 16-byte alignment that its vector
loads want (they are then read element by element, to the same bits)."""

import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import mlp_oracle as mo  # noqa: E402
from tests.test_gpu_mlp import DEVICE, bf16_tensor, network, random_batch  # noqa: E402

pytestmark = pytest.mark.gpu


def blocks():
    return [(mo.W_OFFSETS[i], mo.W_OFFSETS[i + 1]) for i in range(4)] + [
        (mo.B_OFFSETS[i], mo.B_OFFSETS[i + 1]) for i in range(4)]


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 8193, 16385])
def test_rows_around_tile_edges(backend, n):
    net, p = network(3, backend._lib)
    x = random_batch(n, 4)
    dy = np.random.default_rng(5).normal(0, 1, (n, mo.OUTPUTS)).astype(np.float32) / n
    xt = bf16_tensor(x)
    _, act = net.forward(xt, keep=True)
    g = net.backward(xt, act, torch.from_numpy(dy).to(DEVICE)).cpu().numpy().astype(np.float64)
    _, cache = mo.forward(p, x, round_like_kernels=True)
    ref = mo.backward(cache, dy.astype(np.float64))
    for lo, hi in blocks():
        # bf16 output and hidden gradients (2^-9 relative each) feed four layers.
        err = np.linalg.norm(g[lo:hi] - ref[lo:hi]) / max(np.linalg.norm(ref[lo:hi]), 1e-30)
        assert err < 2e-2, (lo, hi, err)
    # The output layer's bias gradient is a plain FP32 sum of the gradients.
    got = g[mo.B_OFFSETS[3]:mo.B_OFFSETS[3] + mo.OUTPUTS]
    assert np.allclose(got, dy.astype(np.float64).sum(axis=0), rtol=0, atol=1e-6 * np.abs(dy).sum(axis=0).max())


def test_unaligned_operands_give_the_same_bits(backend):
    n = 300
    net, _ = network(3, backend._lib)
    xt = bf16_tensor(random_batch(n, 4))
    dy = torch.from_numpy(np.random.default_rng(5).normal(0, 1, (n, mo.OUTPUTS)).astype(np.float32)).to(DEVICE)
    _, act = net.forward(xt, keep=True)
    expected = net.backward(xt, act, dy).clone()
    lib = net._lib
    shifted = torch.empty(xt.numel() + 1, dtype=torch.int16, device=DEVICE)
    shifted[1:] = xt.reshape(-1)
    weights = torch.empty(net.weights.numel() + 1, dtype=torch.int16, device=DEVICE)
    weights[1:] = net.weights
    activations = torch.empty(act.numel() + 4, dtype=torch.uint8, device=DEVICE)
    activations[4:] = act
    scratch = torch.empty(int(lib.msb_mlp_backward_scratch_bytes(n)) + 4, dtype=torch.uint8, device=DEVICE)
    grads = torch.zeros_like(net.grads)
    stream = ctypes.c_void_p(torch.cuda.current_stream(DEVICE).cuda_stream)
    net._check(lib.msb_mlp_backward(
        ctypes.c_void_p(weights.data_ptr() + 2), ctypes.c_void_p(shifted.data_ptr() + 2), n,
        ctypes.c_void_p(activations.data_ptr() + 4), ctypes.c_void_p(dy.data_ptr()), ctypes.c_void_p(grads.data_ptr()),
        ctypes.c_void_p(scratch.data_ptr() + 4), stream))
    assert torch.equal(grads, expected)
