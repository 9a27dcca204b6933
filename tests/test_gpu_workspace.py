"""Product calls whose workspace cannot be had, or whose stream is captured: the kernels without a workspace run."""
import ctypes
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


class no_workspace:
    """The calling thread's product calls find no memory for a workspace (cfft_diag_set_workspace_limit)."""

    def __enter__(self):
        import concrete_fft as cf
        cf.check(cf.load().cfft_diag_set_workspace_limit(1))

    def __exit__(self, *exc):
        import concrete_fft as cf
        cf.check(cf.load().cfft_diag_set_workspace_limit(0))


def run_two_instances(torch, call, wipe):
    """Captures call(), makes two instances of the graph and launches each, with wipe() before; a graph with
    allocation nodes can have one only.  Yields after each launch."""
    cu = ctypes.CDLL("libcuda.so.1")

    def ok(status, what):
        assert status == 0, (what, status)

    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    s, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    with torch.cuda.stream(stream):
        call()  # kernel attributes are set once, outside the capture
        stream.synchronize()
        ok(cu.cuStreamBeginCapture_v2(s, 1), "begin")
        try:
            call()
        finally:
            end = cu.cuStreamEndCapture(s, ctypes.byref(graph))
        ok(end, "end")
        execs = []
        try:
            for _ in range(2):
                e = ctypes.c_void_p()
                ok(cu.cuGraphInstantiateWithFlags(ctypes.byref(e), graph, ctypes.c_ulonglong(0)), "instance")
                execs.append(e)
            for e in execs:
                wipe()
                ok(cu.cuGraphLaunch(e, s), "launch")
                stream.synchronize()
                yield
        finally:
            for e in execs:
                cu.cuGraphExecDestroy(e)
            cu.cuGraphDestroy(graph)


def u128_case(torch, N, count):
    import concrete_fft as cf
    g = torch.Generator(device="cuda").manual_seed(N + count)
    plan = cf.product.U128ProductPlan(N)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (count, N, 2), generator=g, device="cuda")
    bhat = torch.empty((1, 4, N // 2), dtype=torch.float64, device="cuda")
    plan.prepare_operand(torch.randint(-128, 128, (1, N), generator=g, device="cuda"), bhat)
    return plan, lambda out: plan.product(a, bhat, out, shared_operand=True), torch.empty_like(a)


@pytest.mark.parametrize("N,count", [(4096, 80), (8192, 78), (8192, 3), (2048, 20)])
def test_u128_product_without_workspace(cuda, N, count):
    plan, product, want = u128_case(cuda, N, count)
    product(want)
    out = want.clone().fill_(-1)
    with no_workspace():
        product(out)
    assert cuda.equal(out, want)


def test_u128_product_that_needs_a_workspace(cuda):
    """Refused as out of memory, and nothing of that is left for the launch check of the next call."""
    import concrete_fft as cf
    plan, product, want = u128_case(cuda, 16384, 3)
    fused, fused_product, fused_out = u128_case(cuda, 1024, 200)
    product(want)
    out = want.clone().fill_(-1)
    with no_workspace(), pytest.raises(cf.CfftError, match="workspace"):
        product(out)
    fused_product(fused_out)
    product(out)
    assert cuda.equal(out, want)


@pytest.mark.parametrize("N,count", [(4096, 80), (8192, 78)])
def test_u128_product_captured_without_allocations(cuda, N, count):
    plan, product, want = u128_case(cuda, N, count)
    product(want)
    out = want.clone()
    for _ in run_two_instances(cuda, lambda: product(out), lambda: out.fill_(-1)):
        assert cuda.equal(out, want)


def test_workspace_parts_stay_in_the_pool(cuda):
    """A batch beyond one part, waited for and called again, takes no more memory from the device."""
    N, count = 16384, 4200  # 1050 MiB of f64 in all
    plan, product, out = u128_case(cuda, N, count)
    product(out)
    cuda.cuda.synchronize()
    before = cuda.cuda.mem_get_info()[0]
    product(out)
    after = cuda.cuda.mem_get_info()[0]
    cuda.cuda.synchronize()
    assert before - after <= 32 << 20


def sum_case(torch, N, algo, base, count, terms):
    import concrete_fft as cf
    g = torch.Generator(device="cuda").manual_seed(N + count + terms)
    plan = cf.product.U64ProductPlan(N, algo, base)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (count, terms, N), generator=g, device="cuda")
    bhat = torch.empty((count, terms, N // 2), dtype=torch.complex128, device="cuda")
    plan.prepare_operand(torch.randint(-128, 128, (count * terms, N), generator=g, device="cuda"), bhat)
    want = torch.empty((count, N), dtype=torch.int64, device="cuda")
    plan.set_cluster_size(1 if N <= 8192 else 2)  # the kernels that need no workspace
    plan.product_sum(a, bhat, want)
    plan.set_cluster_size(0)
    return plan, lambda out: plan.product_sum(a, bhat, out), want


SUMS = [(2048, 2, 1024, 2, 4), (1024, 4, 512, 3, 5), (2048, 0, 1024, 75, 2), (4096, 2, 1024, 2, 4), (8192, 4, 1024, 1, 3),
        (16384, 2, 1024, 2, 3), (8192, 6, 512, 5, 2), (2048, 3, 1024, 4, 3), (2048, 7, 1024, 2, 2), (8192, 5, 1024, 40, 3),
        (4096, 1, 512, 3, 2), (8192, 7, 512, 1, 2), (64, 1, 32, 5, 3), (2048, 7, 1024, 2, 1), (4096, 1, 512, 3, 1),
        (8192, 7, 512, 1, 1), (16384, 3, 1024, 2, 1)]


@pytest.mark.parametrize("N,algo,base,count,terms", SUMS)
def test_u64_product_sum_without_workspace(cuda, N, algo, base, count, terms):
    plan, product_sum, want = sum_case(cuda, N, algo, base, count, terms)
    out = want.clone().fill_(-1)
    product_sum(out)
    assert cuda.equal(out, want)
    out.fill_(-1)
    with no_workspace():
        product_sum(out)
    assert cuda.equal(out, want)


@pytest.mark.parametrize("N,algo,base,count,terms", SUMS)
def test_u64_product_sum_captured_without_allocations(cuda, N, algo, base, count, terms):
    plan, product_sum, want = sum_case(cuda, N, algo, base, count, terms)
    out = want.clone()
    for _ in run_two_instances(cuda, lambda: product_sum(out), lambda: out.fill_(-1)):
        assert cuda.equal(out, want)


@pytest.mark.parametrize("N,algo,base,count", [(4096, 2, 1024, 612), (8192, 5, 512, 610), (16384, 4, 1024, 305)])
def test_u64_products_without_workspace_and_captured(cuda, N, algo, base, count):
    import concrete_fft as cf
    g = cuda.Generator(device="cuda").manual_seed(N)
    plan = cf.product.U64ProductPlan(N, algo, base)
    a = cuda.randint(-(1 << 63), (1 << 63) - 1, (count, N), generator=g, device="cuda")
    bhat = cuda.empty((count, N // 2), dtype=cuda.complex128, device="cuda")
    plan.prepare_operand(cuda.randint(-128, 128, (count, N), generator=g, device="cuda"), bhat)
    want = cuda.empty_like(a)
    plan.product(a, bhat, want)
    out = want.clone().fill_(-1)
    with no_workspace():
        plan.product(a, bhat, out)
    assert cuda.equal(out, want)
    for _ in run_two_instances(cuda, lambda: plan.product(a, bhat, out), lambda: out.fill_(-1)):
        assert cuda.equal(out, want)


def test_u64_product_sum_of_one_term_takes_a_bounded_workspace(cuda):
    """75 products of N = 2^21 go through parts of 1 GiB, not through 75 transforms (1.2 GiB) at once."""
    import concrete_fft as cf
    cf.check(cf.load().cfft_diag_set_workspace_limit(1 << 30))
    try:
        plan, product_sum, out = u64_large_sum(cuda)
        product_sum()
    finally:
        cf.check(cf.load().cfft_diag_set_workspace_limit(0))


def u64_large_sum(torch):
    import concrete_fft as cf
    N, count = 1 << 21, 75
    plan = cf.product.U64ProductPlan(N, 2, 1024)
    a = torch.ones((count, 1, N), dtype=torch.int64, device="cuda")
    bhat = torch.ones((count, 1, N // 2), dtype=torch.complex128, device="cuda")
    out = torch.empty((count, N), dtype=torch.int64, device="cuda")
    return plan, lambda: plan.product_sum(a, bhat, out), out


@pytest.mark.parametrize("case", ["sum", "sum_unfused", "products", "u128"])
def test_graph_workspace_on_request(cuda, case):
    """Captured calls of a plan that allows it take the workspace routes: the same bits, in one instance."""
    torch = cuda
    if case.startswith("sum"):
        plan, call, want = sum_case(torch, *((2048, 2, 1024, 2, 4) if case == "sum" else (2048, 3, 1024, 4, 3)))
    elif case == "u128":
        plan, call, want = u128_case(torch, 4096, 80)
        call(want)
    else:
        import concrete_fft as cf
        plan = cf.product.U64ProductPlan(4096, 2, 1024)
        a = torch.randint(-(1 << 63), (1 << 63) - 1, (612, 4096), device="cuda")
        bhat = torch.randn((612, 2048), dtype=torch.complex128, device="cuda")
        want = torch.empty_like(a)
        plan.product(a, bhat, want)

        def call(out):
            plan.product(a, bhat, out)
    plan.set_graph_workspace(True)
    out = want.clone()
    with pytest.raises(AssertionError, match="instance"):  # the second one, as CUDA documents it
        for _ in run_two_instances(torch, lambda: call(out), lambda: out.fill_(-1)):
            pass
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(out)
    for _ in range(2):
        out.fill_(-1)
        graph.replay()
        assert torch.equal(out, want)
    plan.set_graph_workspace(False)
    for _ in run_two_instances(torch, lambda: call(out), lambda: out.fill_(-1)):
        assert torch.equal(out, want)


def test_workspace_calls_on_two_streams_at_once(cuda):
    """Sums in two launches, unfused sums and large products interleaved on two streams: every call has a
    workspace of its own."""
    torch = cuda
    cases = [sum_case(torch, *c) for c in ((2048, 2, 1024, 2, 4), (2048, 3, 1024, 40, 3), (16384, 2, 1024, 2, 3))]
    plan, product, want = u128_case(torch, 4096, 80)
    product(want)
    cases.append((plan, product, want))
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[want.clone().fill_(-1) for _, _, want in cases] for _ in streams]
    torch.cuda.synchronize()
    for _ in range(20):
        for k, (_, call, _) in enumerate(cases):
            for s, out in zip(streams, outs):
                with torch.cuda.stream(s):
                    call(out[k])
    torch.cuda.synchronize()
    for out in outs:
        for (_, _, want), o in zip(cases, out):
            assert torch.equal(o, want)


def test_u64_products_go_through_parts_of_the_pool(cuda):
    """130 products of N = 2^20 need 1.02 GiB at once: they run in two parts of at most 1 GiB, with the same bits."""
    import concrete_fft as cf
    torch = cuda
    N, count = 1 << 20, 130
    g = torch.Generator(device="cuda").manual_seed(3)
    plan = cf.product.U64ProductPlan(N, 2, 1024)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (count, N), generator=g, device="cuda")
    bhat = torch.empty((1, N // 2), dtype=torch.complex128, device="cuda")
    plan.prepare_operand(torch.randint(-128, 128, (1, N), generator=g, device="cuda"), bhat)
    out = torch.empty_like(a)
    cf.check(cf.load().cfft_diag_set_workspace_limit(1 << 30))
    try:
        plan.product(a, bhat, out, True)
    finally:
        cf.check(cf.load().cfft_diag_set_workspace_limit(0))
    for r in (0, 64, 65, 129):
        one = torch.empty((1, N), dtype=torch.int64, device="cuda")
        plan.product(a[r:r + 1].contiguous(), bhat, one, True)
        assert torch.equal(out[r], one[0]), r


LAST_PLAN = """
import sys
sys.path.insert(0, %r)
import torch
import concrete_fft as cf
plan = cf.product.U128ProductPlan(16384)
a = torch.ones((2000, 16384, 2), dtype=torch.int64, device="cuda")
bhat = torch.ones((1, 4, 8192), dtype=torch.float64, device="cuda")
out = torch.empty_like(a)
s = torch.cuda.Stream()
with torch.cuda.stream(s):
    plan.product(a, bhat, out, shared_operand=True)  # a first call loads the kernels
torch.cuda.synchronize()
del plan
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
plan = cf.product.U128ProductPlan(16384)
with torch.cuda.stream(s):
    for _ in range(3):
        plan.product(a, bhat, out, shared_operand=True)
del plan  # with the products and the free of their workspace still to run
torch.cuda.synchronize()
torch.cuda.synchronize()
assert free - torch.cuda.mem_get_info()[0] <= 32 << 20, (free, torch.cuda.mem_get_info()[0])
"""


def test_last_plan_gives_the_pool_back(cuda):
    """The workspace pool goes with the last product plan, also where a stream has not run its frees yet."""
    pkg = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "concrete-fft_gb300")
    r = subprocess.run([sys.executable, "-c", LAST_PLAN % pkg], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
