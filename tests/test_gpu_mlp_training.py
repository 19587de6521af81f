"""The one-pass training kernel at the edges of its tiles and of its grid (128 samples per tile, at
most 148 CTAs): loss and gradients against an FP64 restatement on the kernel's own BF16 operands."""

import ctypes

import pytest
import torch

from newton_b200 import _lib
from newton_b200 import learned as L

pytestmark = pytest.mark.gpu


def _fp64(mlp, X, T):
    p = mlp.params.double().clone()
    b16 = lambda t: t.float().bfloat16().double()  # noqa: E731
    W1, W2 = p[L.OFF_W1:L.OFF_B1].reshape(L.IN, L.HID), p[L.OFF_W2:L.OFF_B2].reshape(L.HID, L.HID)
    W3 = p[L.OFF_W3:L.OFF_B3].reshape(L.HID, L.OUTP)
    W1, W2, W3 = b16(W1), b16(W2), b16(W3)
    x = b16(X)
    silu = torch.nn.functional.silu
    dsilu = lambda z: torch.sigmoid(z) * (1 + z * (1 - torch.sigmoid(z)))  # noqa: E731
    z1 = x @ W1 + p[L.OFF_B1:L.OFF_W2]
    h1 = b16(silu(z1))
    z2 = h1 @ W2 + p[L.OFF_B2:L.OFF_W3]
    h2 = b16(silu(z2))
    e = (h2 @ W3 + p[L.OFF_B3:])[:, :3] - T.double()
    dy = torch.zeros(len(X), L.OUTP, dtype=torch.float64, device=X.device)
    dy[:, :3] = b16(2.0 * e / len(X))
    dz2 = b16((dy @ W3.T) * dsilu(b16(z2)))
    dz1 = b16((dz2 @ W2.T) * dsilu(b16(z1)))
    g = torch.cat([v.reshape(-1) for v in (x.T @ dz1, dz1.sum(0), h1.T @ dz2, dz2.sum(0), h2.T @ dy, dy.sum(0))])
    return (e * e).sum(), g


@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 128, 148 * 128 + 1, 40000])
def test_training_pass_matches_fp64_on_the_same_operands(n):
    lib = _lib.load()
    cnt = ctypes.c_uint32()
    _lib.check(lib.vbd_mlp_timeouts(ctypes.byref(cnt), 1))
    mlp = L.WarmStartMLP("cuda:0", seed=11)
    gen = torch.Generator(device="cuda").manual_seed(n)
    X = torch.randn(n, L.IN, generator=gen, device="cuda")
    T = torch.randn(n, 3, generator=gen, device="cuda")
    loss = mlp.gradients(X, T)
    again = mlp.grads.clone()
    loss2 = mlp.gradients(X, T)
    assert torch.equal(again, mlp.grads) and torch.equal(loss, loss2)  # fixed summation order
    ref_loss, ref = _fp64(mlp, X, T)
    # same operands, FP32 accumulation: what is left are operands that round the other way, where a
    # pre-rounding value differs in its last FP32 bits: a 2^-9 step on a small share of them, far
    # below the 2^-9 of one rounding in the 2-norm
    assert abs(float(loss) - float(ref_loss)) <= 1e-4 * float(ref_loss)
    for a, b in ((L.OFF_W1, L.OFF_B1), (L.OFF_B1, L.OFF_W2), (L.OFF_W2, L.OFF_B2), (L.OFF_B2, L.OFF_W3),
                 (L.OFF_W3, L.OFF_B3), (L.OFF_B3, L.N_PARAMS)):
        d = (mlp.grads[a:b].double() - ref[a:b]).norm() / ref[a:b].norm()
        assert float(d) <= 2.0 ** -9, (a, float(d))
    _lib.check(lib.vbd_mlp_timeouts(ctypes.byref(cnt), 0))
    assert cnt.value == 0


def test_training_pass_accepts_rows_that_are_not_16_byte_aligned():
    mlp = L.WarmStartMLP("cuda:0", seed=12)
    flat = torch.randn(300 * L.IN + 1, device="cuda")
    T = torch.randn(300, 3, device="cuda")
    X = flat[1:].reshape(300, L.IN)
    assert X.data_ptr() % 16 != 0
    mlp.gradients(X, T)
    a = mlp.grads.clone()
    mlp.gradients(X.clone(), T)
    assert torch.equal(a, mlp.grads)
