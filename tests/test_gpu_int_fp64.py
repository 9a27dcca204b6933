"""The integer-pipe double addition used inside the FFT kernels must equal the
native FP64 add bit for bit (it is the same IEEE operation on another pipe)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_dadd_int_equals_native_add(cuda, cfft_lib):
    import concrete_fft as cf
    bad = ctypes.c_uint64()
    pair = (ctypes.c_uint64 * 2)()
    for seed in (1, 2, 3):
        cf.check(cfft_lib.cfft_diag_dadd_check(1 << 28, seed, ctypes.byref(bad), pair))
        assert bad.value == 0, "first mismatch x=%016x y=%016x" % (pair[0], pair[1])


def test_dadd_int_rate_is_reported(cuda, cfft_lib):
    import concrete_fft as cf
    r = ctypes.c_double()
    cf.check(cfft_lib.cfft_diag_dadd_int_rate(ctypes.byref(r)))
    assert r.value > 1e10


def test_fp64_rates(cfft_lib):
    """The FP64 roof microbenchmarks: four positive rates, the peak is their best."""
    import concrete_fft as cf
    r = (ctypes.c_double * 4)()
    cf.check(cfft_lib.cfft_diag_fp64_rates(r))
    rates = list(r)
    assert all(x > 1e10 for x in rates), rates
    p = ctypes.c_double()
    cf.check(cfft_lib.cfft_diag_fp64_peak(ctypes.byref(p)))
    assert p.value > 0.9 * max(rates)


def _edge_data(kind, batch, n):
    """Inputs that leave the integer additions' range: each pair then takes the FP64 pipe."""
    import numpy as np
    rng = np.random.default_rng(n + batch)
    x = rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))
    if kind == "zeros":
        x[:] = 0
    elif kind == "impulses":
        x[:] = 0
        x[np.arange(batch), np.arange(batch) % n] = 1.5 - 0.25j
    elif kind == "constant":  # every difference cancels exactly
        x[:] = 0.75 + 0.5j
    elif kind == "real":
        x.imag = 0
    elif kind == "small_integers":  # exact halves: ties in every rounding
        x = (rng.integers(-3, 4, (batch, n)) + 1j * rng.integers(-3, 4, (batch, n))).astype(np.complex128)
    elif kind == "spread":  # exponents up to 1200 apart, neighbours too
        x = x * np.exp2(rng.integers(-600, 600, (batch, n)))
    elif kind == "near_limits":  # gaps of 8 to 13 bits around the 10 that are exact
        x = x * np.exp2(rng.integers(8, 14, (batch, n)) * rng.integers(0, 2, (batch, n)))
    elif kind == "subnormal":
        x = x * 2.0 ** -1060
    return x


@pytest.mark.parametrize("kind", ["zeros", "impulses", "constant", "real", "small_integers", "spread", "near_limits",
                                  "subnormal"])
@pytest.mark.parametrize("algo", range(8))
def test_transforms_outside_the_integer_range(cuda, oracle, algo, kind):
    """Split (half and whole butterflies) and one-CTA kernels on inputs that the integer additions leave
    to the FP64 pipe, bit for bit."""
    import concrete_fft as cf
    import numpy as np
    torch = cuda
    for n, batch in ((256, 1), (1024, 3), (1024, 200), (512, 700)):
        x = _edge_data(kind, batch, n)
        plan = cf.ordered.Plan(n, cf.ordered.Method.UserProvided(algo))
        d = torch.from_numpy(x.copy()).cuda()
        plan.fwd(d)
        f = oracle.ordered_fwd(algo, x)
        assert np.array_equal(d.cpu().numpy().view(np.uint64), f.view(np.uint64)), (n, batch, "fwd")
        plan.inv(d)
        assert np.array_equal(d.cpu().numpy().view(np.uint64), oracle.ordered_inv(algo, f).view(np.uint64)), (n, batch)


@pytest.mark.parametrize("algo", [4, 5, 6, 7])
@pytest.mark.parametrize("N", [64, 128, 512, 1024, 2048])
def test_one_cta_kernels_with_few_and_many_warps(cuda, oracle, algo, N):
    """Radix 8 and 16: launches of about a warp per SM sub-partition keep their additions on the FP64
    pipe, larger ones move them; counts on both sides of the line, bit for bit."""
    import concrete_fft as cf
    import numpy as np
    torch = cuda
    n = N // 2
    rng = np.random.default_rng(N + algo)
    plan = cf.product.U64ProductPlan(N, algo, n)
    fft = cf.ordered.Plan(n, cf.ordered.Method.UserProvided(algo))
    warps = -(-min(128, max(1, n >> (algo // 2 + 1))) // 32)
    line = 5 * torch.cuda.get_device_properties(0).multi_processor_count // warps  # first count that is not few
    for count in (1, 3, line - 1, line, 2 * line + 5):
        a = rng.integers(0, 1 << 64, (count, N), dtype=np.uint64)
        b = rng.integers(-512, 512, (count, N), dtype=np.int64)
        bhat = torch.empty((count, n), dtype=torch.complex128, device="cuda")
        plan.prepare_operand(torch.from_numpy(b).cuda(), bhat)
        want_bhat = oracle.u64_prepare(N, algo, n, b)
        assert np.array_equal(bhat.cpu().numpy().view(np.uint64), want_bhat.view(np.uint64)), count
        da = torch.from_numpy(a.view(np.int64)).cuda()
        out = torch.empty_like(da)
        plan.product(da, bhat, out)
        want = oracle.u64_product(N, algo, n, a, want_bhat, nthreads=0)
        assert np.array_equal(out.cpu().numpy().view(np.uint64), want), count
        plan.product_sum(da.reshape(count, 1, N), bhat.reshape(count, 1, n), out)
        want = oracle.u64_product_sum(N, algo, n, a.reshape(count, 1, N), want_bhat.reshape(count, 1, n), nthreads=0)
        assert np.array_equal(out.cpu().numpy().view(np.uint64), want), (count, "sum")
        x = rng.uniform(-1, 1, (count, n)) + 1j * rng.uniform(-1, 1, (count, n))
        d = torch.from_numpy(x.copy()).cuda()
        fft.fwd(d)
        assert np.array_equal(d.cpu().numpy().view(np.uint64), oracle.ordered_fwd(algo, x).view(np.uint64)), count


@pytest.mark.parametrize("algo", range(8))
def test_set_int_adds_chooses_the_instance(cuda, algo):
    """0 and 8 run the FP64-pipe and the integer instance of every kernel on the same data: the same bits,
    at small and large launches alike."""
    import concrete_fft as cf
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(algo)

    def same(x, y):
        return torch.equal(x.view(torch.int64), y.view(torch.int64))

    for n, base, batch in ((64, 64, 1), (1024, 1024, 1), (1024, 1024, 700), (2048, 512, 3), (4096, 1024, 400),
                           (1 << 16, 1024, 1), (1 << 16, 512, 9)):
        plan = cf.unordered.Plan(n, cf.unordered.Method.UserProvided(algo, base))
        assert plan.int_adds() == 6
        x = torch.randn((batch, n, 2), dtype=torch.float64, device="cuda", generator=g)
        res = []
        for adds in (None, 0, 8):
            if adds is not None:
                plan.set_int_adds(adds)
                assert plan.int_adds() == adds
            f = x.clone()
            plan.fwd(torch.view_as_complex(f))
            i = f.clone()
            plan.inv(torch.view_as_complex(i))
            res.append((f, i))
        for f, i in res[1:]:
            assert same(f, res[0][0]) and same(i, res[0][1]), (n, batch)
    for N, base, count, terms in ((256, 128, 700, 1), (2048, 1024, 2, 4), (2048, 1024, 900, 1), (8192, 1024, 1, 1),
                                  (8192, 512, 100, 2), (16384, 1024, 60, 1)):
        plan = cf.product.U64ProductPlan(N, algo, base)
        assert plan.int_adds() == 6
        a = torch.randint(-(1 << 63), (1 << 63) - 1, (count, terms, N), generator=g, device="cuda")
        b = torch.randint(-128, 128, (count * terms, N), generator=g, device="cuda")
        res = []
        for adds in (None, 0, 8):
            if adds is not None:
                plan.set_int_adds(adds)
            bhat = torch.empty((count, terms, N // 2, 2), dtype=torch.float64, device="cuda")
            plan.prepare_operand(b, bhat)
            out = torch.empty((count, N), dtype=torch.int64, device="cuda")
            plan.product_sum(a, torch.view_as_complex(bhat), out)
            if terms == 1:
                p = torch.empty_like(out)
                plan.product(a.reshape(count, N), bhat, p)
                assert torch.equal(p, out)
            res.append((bhat, out))
        for bhat, out in res[1:]:
            assert same(bhat, res[0][0]) and torch.equal(out, res[0][1]), (N, count)


def test_set_int_adds_changes_the_time(cuda):
    """8192 products of N = 2048 are bound by the FP64 pipe when every addition stays on it (1.5 times)."""
    import concrete_fft as cf
    torch = cuda
    N, count = 2048, 8192
    plan = cf.product.U64ProductPlan(N, 2, 1024)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (count, N), device="cuda")
    bhat = torch.randn((count, N // 2), dtype=torch.complex128, device="cuda")
    out = torch.empty_like(a)
    ms = {}
    for adds in (0, 8, 0, 8):
        plan.set_int_adds(adds)
        plan.product(a, bhat, out)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(5):
            plan.product(a, bhat, out)
        e1.record()
        e1.synchronize()
        ms[adds] = min(ms.get(adds, 1e9), e0.elapsed_time(e1))
    assert ms[0] > 1.2 * ms[8]


def _same_or_nan(got, want):
    """The same bits, or NaN in both (whose sign and payload IEEE 754 leaves open)."""
    import numpy as np
    g, w = got.view(np.uint64).ravel(), want.view(np.uint64).ravel()
    nan = np.isnan(got.view(np.float64).ravel()) & np.isnan(want.view(np.float64).ravel())
    return bool(np.all((g == w) | nan))


@pytest.mark.parametrize("kind", ["infinities", "nans", "near_overflow", "overflowing"])
@pytest.mark.parametrize("algo", range(8))
def test_transforms_of_infinities_and_overflow(cuda, oracle, algo, kind):
    """Infinities, NaNs and values at the top of the range through transforms of both instances."""
    import concrete_fft as cf
    import numpy as np
    torch = cuda
    rng = np.random.default_rng(algo)
    for n, batch in ((256, 1), (1024, 200), (512, 700)):
        x = rng.uniform(-1, 1, (batch, n)) + 1j * rng.uniform(-1, 1, (batch, n))
        p = np.arange(batch) % n
        if kind == "infinities":
            x.real[np.arange(batch), p] = np.where(p % 2, np.inf, -np.inf)
        elif kind == "nans":
            x.imag[np.arange(batch), p] = np.nan
        elif kind == "near_overflow":  # sums just below the largest double
            x = x * 2.0 ** (1023 - n.bit_length())
        else:
            x = x * 2.0 ** 1022
        plan = cf.ordered.Plan(n, cf.ordered.Method.UserProvided(algo))
        d = torch.from_numpy(x.copy()).cuda()
        plan.fwd(d)
        with np.errstate(all="ignore"):
            f = oracle.ordered_fwd(algo, x)
        assert _same_or_nan(d.cpu().numpy(), f), (n, batch)
