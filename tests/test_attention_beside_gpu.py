"""dQ beside dK and dV: the two kernels of the attention backward run at the same time. Their inputs come from the kernel
right before them and the kernel right behind them reads both results, over and over without a pause; every pass gives the
bits of a pass with the device idle before and after it. Fewer and more dK/dV items than SMs, both head sizes, both precisions."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x3", [False, True])
@pytest.mark.parametrize("B,T,H,Hk,D", [(1, 127, 9, 3, 64), (2, 300, 3, 3, 64), (16, 513, 9, 3, 64), (2, 300, 4, 2, 128), (8, 700, 16, 8, 128)])
def test_backward_without_a_pause(B, T, H, Hk, D, x3):
    import torch

    from emberlm_b200 import lib, ops

    precision = lib.GEMM_3XTF32 if x3 else lib.GEMM_TF32
    gen = torch.Generator("cuda").manual_seed(2)
    base = torch.empty(B * T, (H + 2 * Hk) * D, device="cuda").uniform_(-1.5, 1.5, generator=gen)
    douts = [torch.empty(B * T, H * D, device="cuda").uniform_(-1, 1, generator=gen) for _ in range(4)]

    def run(i, dout, pause):
        qkv = base * (1.0 + 0.1 * i)
        out, lse = ops.attention(qkv, B, T, H, Hk, D, precision=precision)
        dout.copy_(douts[i])
        if pause:
            torch.cuda.synchronize()
        got = ops.attention_backward(qkv, out, dout, lse, B, T, H, Hk, D, precision=precision)
        if pause:
            torch.cuda.synchronize()
        return got * 2.0

    dout = torch.empty_like(douts[0])
    want = [run(i, dout, True) for i in range(4)]
    got = [run(i % 4, dout, False) for i in range(24)]
    assert all(torch.equal(g, want[i % 4]) for i, g in enumerate(got))
