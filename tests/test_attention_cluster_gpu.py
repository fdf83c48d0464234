"""dK and dV of the near-fp32 attention, summed over the CTAs of a cluster: one, two, four and eight of them, ranks
without a query tile, ragged last tiles. Reference: the same backward in 64 bits; tolerance as for the other sizes of this
mode (three TF32 products keep about 2^-21 of an operand, sums over a few hundred terms)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,Hk,D", [(1, 40, 3, 3, 64), (1, 100, 1, 1, 64), (3, 301, 9, 3, 64), (1, 513, 4, 1, 64), (1, 200, 2, 1, 128),
                                        (16, 300, 6, 3, 64)])
def test_backward(B, T, H, Hk, D):
    import torch

    from emberlm_b200 import lib, ops

    gen = torch.Generator("cuda").manual_seed(1)
    qkv = torch.empty(B * T, (H + 2 * Hk) * D, device="cuda").uniform_(-1.5, 1.5, generator=gen)
    dout = torch.empty(B * T, H * D, device="cuda").uniform_(-1, 1, generator=gen)
    x = qkv.double().reshape(B, T, H + 2 * Hk, D).requires_grad_()
    q, k, v = x[:, :, :H], x[:, :, H:H + Hk].repeat_interleave(H // Hk, 2), x[:, :, H + Hk:].repeat_interleave(H // Hk, 2)
    s = torch.einsum("bihd,bjhd->bhij", q, k) * D ** -0.5
    p = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf")).softmax(-1)
    torch.einsum("bhij,bjhd->bihd", p, v).reshape(B * T, -1).backward(dout.double())
    want = x.grad.reshape(B * T, -1)
    out, lse = ops.attention(qkv, B, T, H, Hk, D, precision=lib.GEMM_3XTF32)
    runs = [ops.attention_backward(qkv, out, dout, lse, B, T, H, Hk, D, precision=lib.GEMM_3XTF32) for _ in range(2)]
    assert torch.equal(*runs)
    assert float((runs[0].double() - want).abs().max() / want.abs().max()) < 5e-5
