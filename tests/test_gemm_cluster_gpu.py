"""Products with few tiles: K split over the CTAs of a cluster. Small integers are exact in TF32, so a wrong tile, range
or column exchange shows as a wrong integer. The parts are added in a fixed order, so runs on random values agree bit for
bit."""
import pytest

pytestmark = pytest.mark.gpu


def _ints(shape, seed):
    import torch

    return torch.randint(-3, 4, shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda").float()


# one and several rows of tiles, ragged edges (N = 130: rows that cannot be stored in fours), the shortest K of each cluster
# size (2, 4 and 8 CTAs: 128, 256 and 512), a K that leaves ranges of different lengths, two rows of tiles on clusters of
# 4 and 2, more tiles than clusters (another kernel's)
SHAPES = [(1, 576, 576), (127, 960, 576), (37, 576, 1536), (129, 130, 1000), (300, 3072, 576), (5, 64, 512), (64, 192, 256), (128, 8, 128),
          (200, 2048, 2052), (127, 1024, 3072), (255, 960, 960), (250, 2048, 1024), (130, 1024, 64)]


@pytest.mark.parametrize("epilogue", ["store", "accumulate", "residual"])
@pytest.mark.parametrize("ta,tb", [(0, 1), (0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("precision", ["tf32", "3xtf32"])
def test_exact(precision, M, N, K, ta, tb, epilogue):
    import torch

    from emberlm_b200 import lib, ops

    if (ta and M % 4) or (not tb and N % 4):
        pytest.skip("rows of the operand are not 16-byte aligned: another kernel's")
    a, b, c = _ints((K, M) if ta else (M, K), 1), _ints((N, K) if tb else (K, N), 2), _ints((M, N), 3)
    want = ((a.T if ta else a).double() @ (b.T if tb else b).double() + (0 if epilogue == "store" else c.double())).float()
    p = lib.GEMM_TF32 if precision == "tf32" else lib.GEMM_3XTF32
    got = []
    for _ in range(2):
        if epilogue == "accumulate":
            got.append(ops.matmul(a, b, bool(ta), bool(tb), p, out=c.clone(), epilogue=lib.EPI_ACCUMULATE))
        elif epilogue == "residual":
            got.append(ops.matmul(a, b, bool(ta), bool(tb), p, epilogue=lib.EPI_RESIDUAL, aux=c))
        else:
            got.append(ops.matmul(a, b, bool(ta), bool(tb), p))
    assert torch.equal(got[0], want) and torch.equal(got[1], want)


@pytest.mark.parametrize("epilogue", ["store", "accumulate", "residual"])
@pytest.mark.parametrize("ta,tb", [(0, 1), (0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(904, 576, 1536), (1000, 3000, 100), (576, 1536, 904), (260, 100, 6000), (1200, 4096, 32)])
def test_three_products_in_one_launch(M, N, K, ta, tb, epilogue):
    """Operands of 12 significant bits have a low part, so the ranges of all three products count; sums stay exact."""
    import torch

    from emberlm_b200 import lib, ops

    gen = torch.Generator("cuda").manual_seed(5)
    a, b = (torch.randint(-1, 2, s, generator=gen, device="cuda").float() for s in ((K, M) if ta else (M, K), (N, K) if tb else (K, N)))
    a[::3] *= 2049.0     # TF32 holds 2048: one more bit than it has
    c = _ints((M, N), 3)
    want = ((a.T if ta else a).double() @ (b.T if tb else b).double() + (0 if epilogue == "store" else c.double())).float()
    if epilogue == "accumulate":
        got = ops.matmul(a, b, bool(ta), bool(tb), lib.GEMM_3XTF32, out=c.clone(), epilogue=lib.EPI_ACCUMULATE)
    else:
        got = ops.matmul(a, b, bool(ta), bool(tb), lib.GEMM_3XTF32, epilogue=lib.EPI_RESIDUAL if epilogue == "residual" else lib.EPI_STORE,
                         aux=c if epilogue == "residual" else None)
    assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K", [(127, 960, 576), (903, 3072, 576), (576, 1536, 903)])
def test_random_products(M, N, K):
    """TF32 rounds each operand by at most 2^-11: a product of independent values errs by about 2^-11 sqrt(2 / 3) of its
    size, well under 1e-3 in the 2-norm. 3xTF32 leaves 2^-21 an operand and fp32 sums: 2e-6."""
    import torch

    from emberlm_b200 import lib, ops

    gen = torch.Generator("cuda").manual_seed(4)
    a, b = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K)))
    want = a.double() @ b.double().T
    for p, limit in ((lib.GEMM_TF32, 1e-3), (lib.GEMM_3XTF32, 2e-6)):
        err = (ops.matmul(a, b, False, True, p).double() - want).norm() / want.norm()
        assert err < limit, (p, float(err))


# a cluster; units of two runs on one range (K <= 512) and two, 128 and 256 wide
@pytest.mark.parametrize("epilogue", ["store", "residual", "accumulate"])
@pytest.mark.parametrize("M,N,K", [(127, 960, 576), (200, 960, 960), (903, 576, 576), (903, 3072, 576), (1000, 1536, 1000), (600, 2000, 500), (1100, 2048, 96)])
def test_same_bits_each_time(M, N, K, epilogue):
    """3xTF32 products of random values, and TF32 ones on a cluster. (Off clusters the ranges of K > 512 that are
    accumulated, and those of K > 1024, are added in the order of their arrival.) Against 64 bits as test_random_products."""
    import torch

    from emberlm_b200 import lib, ops

    gen = torch.Generator("cuda").manual_seed(6)
    a, b, c = (torch.randn(s, generator=gen, device="cuda") for s in ((M, K), (N, K), (M, N)))
    if epilogue == "accumulate" and K > 512 and M > 256:
        pytest.skip("added in the order of arrival")

    def once(p):
        if epilogue == "accumulate":
            return ops.matmul(a, b, False, True, p, out=c.clone(), epilogue=lib.EPI_ACCUMULATE)
        return ops.matmul(a, b, False, True, p, epilogue=lib.EPI_RESIDUAL if epilogue == "residual" else lib.EPI_STORE,
                          aux=c if epilogue == "residual" else None)

    want = a.double() @ b.double().T + (0 if epilogue == "store" else c.double())
    for p, limit in ((lib.GEMM_3XTF32, 2e-6), (lib.GEMM_TF32, 1e-3)):
        if p == lib.GEMM_TF32 and M >= 256:
            continue
        first = once(p)
        assert (first.double() - want).norm() / want.norm() < limit
        for _ in range(5):
            assert torch.equal(once(p), first)
