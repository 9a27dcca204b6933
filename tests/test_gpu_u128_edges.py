"""u128 products at the edges of the integer conversions, the fused kernel, the cluster kernel and the five launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _coefficients(kind, count, N):
    rng = np.random.default_rng(N + count)
    a = rng.integers(0, 2 ** 64, (count, N, 2), dtype=np.uint64)
    top = np.uint64(2 ** 63)
    if kind == "zeros":
        a[:] = 0
    elif kind == "sparse":
        a[:, 1::3] = 0
    elif kind == "small":  # results below 2^53, where the high words have fractions
        a[:, :, 0] = rng.integers(0, 5, (count, N)).astype(np.uint64)
        a[:, :, 1] = 0
    elif kind == "negative_small":
        a[:, :, 0] = np.uint64(0) - rng.integers(1, 1000, (count, N)).astype(np.uint64)
        a[:, :, 1] = ~np.uint64(0)
    elif kind == "powers":  # one bit set, and all bits above one set
        bit = rng.integers(0, 128, (count, N))
        lo = np.where(bit < 64, np.left_shift(np.uint64(1), (bit % 64).astype(np.uint64)), np.uint64(0))
        hi = np.where(bit >= 64, np.left_shift(np.uint64(1), (bit % 64).astype(np.uint64)), np.uint64(0))
        flip = rng.integers(0, 2, (count, N)).astype(bool)
        a[:, :, 0], a[:, :, 1] = np.where(flip, ~lo, lo), np.where(flip, ~hi, hi)
    elif kind == "halves":  # remainders of exactly half a unit of the high word
        a[:, :, 0] = rng.integers(0, 2, (count, N)).astype(np.uint64) * top
        a[:, :, 1] &= np.uint64(2 ** 62 - 1)
    elif kind == "extremes":
        a[:, :, 0] = rng.integers(0, 2, (count, N)).astype(np.uint64) * ~np.uint64(0)
        a[:, :, 1] = top - rng.integers(0, 2, (count, N)).astype(np.uint64)
    return a


@pytest.mark.parametrize("kind", ["random", "zeros", "sparse", "small", "negative_small", "powers", "halves", "extremes"])
@pytest.mark.parametrize("N,count", [(64, 3), (256, 100), (1024, 1), (1024, 90), (4096, 2), (4096, 80), (8192, 78)])
def test_u128_product_edges(cuda, oracle, kind, N, count):
    import concrete_fft as cf
    torch = cuda
    a = _coefficients(kind, count, N)
    b = np.random.default_rng(N).integers(-128, 128, (1, N))
    plan = cf.product.U128ProductPlan(N)
    bhat = torch.empty((1, 4, N // 2), dtype=torch.float64, device="cuda")
    plan.prepare_operand(torch.from_numpy(b).cuda(), bhat)
    out = torch.empty((count, N, 2), dtype=torch.int64, device="cuda")
    plan.product(torch.from_numpy(a.view(np.int64)).cuda(), bhat, out, shared_operand=True)
    got = out.cpu().numpy().view(np.uint64)
    rows = sorted({0, count // 2, count - 1})
    operand = oracle.u128_prepare(N, b)
    for r in rows:
        assert np.array_equal(got[r].reshape(-1), oracle.u128_product(N, a[r:r + 1], operand).reshape(-1)), r


def test_u128_product_in_parts(cuda):
    """More products than one workspace holds: every part gives the bits of a product alone."""
    import concrete_fft as cf
    torch = cuda
    N, count = 1 << 22, 17
    plan = cf.product.U128ProductPlan(N)
    g = torch.Generator(device="cuda").manual_seed(5)
    one = torch.randint(-(1 << 63), (1 << 63) - 1, (1, N, 2), generator=g, device="cuda", dtype=torch.int64)
    b = torch.randint(-128, 128, (1, N), generator=g, device="cuda", dtype=torch.int64)
    bhat = torch.empty((1, 4, N // 2), dtype=torch.float64, device="cuda")
    plan.prepare_operand(b, bhat)
    want = torch.empty_like(one)
    plan.product(one, bhat, want, shared_operand=True)
    a = one.expand(count, N, 2).contiguous()
    out = torch.empty_like(a)
    plan.product(a, bhat, out, shared_operand=True)
    for r in range(count):
        assert torch.equal(out[r], want[0]), r
