"""Performance cases of the library, through its public Python entry points.

A case is a dict of plain values; `kind` says which path it takes:

  slice      one transform on a host array, the reference's slice API (copy in, transform, copy out)
  ordered    ordered::Plan, batched, device data
  unordered  unordered::Plan, batched, device data
  serde      standard-order conversion of permuted Fourier data
  u64        negacyclic u64 products with resident Fourier operands
  sum        products summed in the Fourier domain, one inverse per output (the external product)
  prepare    Fourier operands from signed digits
  u128       negacyclic u128 products (double-double)
  f128       fft128::Plan, batched, split double-double arrays
  mixed      transforms of mixed sizes in one persistent launch

Transforms work in place, so a pass copies its input over the work buffer first, as a caller does
that keeps its polynomial.  Every plan names its algorithm (Method::UserProvided), so that a pass
runs the same operations on every run.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "concrete-fft_gb300"))
import concrete_fft as cf  # noqa: E402

# The base algorithms and sizes that Method::Measure chooses among in practice on this part: radix 4
# at base 1024, radix 8 at base 512, and their DIT twins, plus radix 16 (the product plan's default).
ALGOS = ("Dif4", "Dif8", "Dit4", "Dif16", "Dit8")


def listed():
    return [
        # one small polynomial through the drop-in slice API
        {"name": "slice_ordered_1024", "kind": "slice", "n": 1024, "algo": "Dif4"},
        # the ordered plan's largest size in a batch: forward and inverse, as in the benchmark
        {"name": "ordered_1024_x256", "kind": "ordered", "n": 1024, "batch": 256, "algo": "Dif4", "dir": "fwd_inv"},
        # a ragged batch of the size under an N = 4096 polynomial, forward, radix 8 over base 512
        {"name": "unordered_2048_x613_fwd", "kind": "unordered", "n": 2048, "base_n": 512, "batch": 613,
         "algo": "Dif8", "dir": "fwd"},
        # large transforms whose outer levels run in global memory, inverse
        {"name": "unordered_65536_x37_inv", "kind": "unordered", "n": 65536, "base_n": 1024, "batch": 37,
         "algo": "Dif4", "dir": "inv"},
        # one product alone: the latency of a request served by itself
        {"name": "u64_2048_x1", "kind": "u64", "N": 2048, "base_n": 1024, "count": 1, "algo": "Dif4",
         "shared": False},
        # the headline: a full launch of products, one operand each
        {"name": "u64_2048_x8192", "kind": "u64", "N": 2048, "base_n": 1024, "count": 8192, "algo": "Dif4",
         "shared": False},
        # large polynomials on thread-block clusters, a batch that fills no whole wave, one operand for all
        {"name": "u64_16384_x203", "kind": "u64", "N": 16384, "base_n": 1024, "count": 203, "algo": "Dif4",
         "shared": True},
        # one blind-rotation step: 2 outputs of 4 digit polynomials each
        {"name": "sum_2048_2x4", "kind": "sum", "N": 2048, "base_n": 1024, "count": 2, "terms": 4, "algo": "Dif4"},
        # double-double products, a full launch
        {"name": "u128_1024_x2048", "kind": "u128", "N": 1024, "count": 2048, "shared": False},
        # double-double transforms: a ragged batch, and one of the largest benchmark size alone
        {"name": "f128_512_x1999", "kind": "f128", "n": 512, "batch": 1999, "dir": "fwd_inv"},
        {"name": "f128_16384_x1_fwd", "kind": "f128", "n": 16384, "batch": 1, "dir": "fwd"},
        # a stream of transforms of every size in one launch, forward and inverse
        {"name": "mixed_1500", "kind": "mixed", "count": 1500, "log2_min": 8, "log2_max": 16, "dir": "fwd_inv"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _base(rng, n):
    """A base size the plan accepts: at least 32, at most 1024 and n."""
    return n if n <= 512 else min(n, rng.choice((512, 1024)))


def draw(rng):
    kind = rng.choice(("slice", "ordered", "unordered", "unordered", "serde", "u64", "u64", "u64", "sum", "prepare",
                       "u128", "f128", "f128", "mixed"))
    direction = rng.choice(("fwd", "inv", "fwd_inv"))
    algo = rng.choice(ALGOS)
    if kind == "slice":
        return {"kind": kind, "n": 1 << rng.randint(6, 10), "algo": algo}
    if kind == "ordered":
        n = 1 << rng.randint(6, 10)
        return {"kind": kind, "n": n, "batch": _log_int(rng, 1, (1 << 22) // n), "algo": algo, "dir": direction}
    if kind == "unordered":
        n = 1 << rng.randint(7, 17)
        return {"kind": kind, "n": n, "base_n": _base(rng, n), "batch": _log_int(rng, 1, (1 << 22) // n),
                "algo": algo, "dir": direction}
    if kind == "serde":
        n = 1 << rng.randint(7, 14)
        return {"kind": kind, "n": n, "base_n": _base(rng, n), "batch": _log_int(rng, 1, (1 << 24) // n),
                "to_standard": rng.random() < 0.5}
    if kind in ("u64", "sum", "prepare"):
        N = 1 << rng.randint(8, 16)
        case = {"kind": kind, "N": N, "base_n": _base(rng, N // 2), "algo": algo}
        if kind == "sum":
            case["terms"] = rng.randint(2, 8)
            case["count"] = _log_int(rng, 1, max(2, (1 << 23) // (N * case["terms"])))
        else:
            case["count"] = _log_int(rng, 1, (1 << 24 if N <= 4096 else 1 << 23) // N)
        if kind == "u64":
            case["shared"] = rng.random() < 0.5
        return case
    if kind == "u128":
        N = 1 << rng.randint(8, 14)
        return {"kind": kind, "N": N, "count": _log_int(rng, 1, (1 << 20) // N), "shared": rng.random() < 0.5}
    if kind == "f128":
        n = 1 << rng.randint(6, 14)
        return {"kind": kind, "n": n, "batch": _log_int(rng, 1, (1 << 20) // n), "dir": direction}
    return {"kind": "mixed", "count": _log_int(rng, 30, 1500), "log2_min": 8, "log2_max": rng.randint(11, 16),
            "dir": "fwd_inv"}


# ---------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _complex(shape, g):
    """Values in [0, 1) like the reference's tests, centred."""
    v = torch.rand(shape + (2,), generator=g, device="cuda", dtype=torch.float64) - 0.5
    return torch.view_as_complex(v)


def _torus(shape, g):
    """Uniform 64-bit words, as int64."""
    return torch.randint(-(1 << 63), (1 << 63) - 1, shape, generator=g, device="cuda", dtype=torch.int64)


def _digits(shape, g):
    """Signed 8-bit decomposition digits."""
    return torch.randint(-128, 128, shape, generator=g, device="cuda", dtype=torch.int64)


def _mixed_items(case, seed):
    rng = np.random.default_rng(int(seed) + 1)
    # the sizes and kinds belong to the case, not to the data: every seed has the same work
    shape = np.random.default_rng(case["count"] * 32 + case["log2_max"])
    log2n = shape.integers(case["log2_min"], case["log2_max"] + 1, case["count"])
    kind = np.where(log2n > 10, cf.batch.UNORDERED, shape.integers(0, 2, case["count"]))
    order = rng.permutation(case["count"])
    log2n, kind = log2n[order], kind[order]
    sizes = (1 << log2n).astype(np.int64)
    items = np.zeros(case["count"], dtype=cf.batch.ITEM_DTYPE)
    items["offset"] = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    items["log2n"], items["kind"], items["direction"] = log2n, kind, _direction(case)
    return items, int(sizes.sum())


def _direction(case):
    return {"fwd": cf.batch.FWD, "inv": cf.batch.INV, "fwd_inv": cf.batch.FWD_THEN_INV}[case["dir"]]


def _input(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "slice":
        rng = np.random.default_rng(int(seed))
        return rng.random(case["n"]) - 0.5 + 1j * (rng.random(case["n"]) - 0.5)
    if kind in ("ordered", "unordered", "serde"):
        return _complex((case["batch"], case["n"]), g)
    if kind == "f128":
        x = torch.rand((4, case["batch"], case["n"]), generator=g, device="cuda", dtype=torch.float64) - 0.5
        x[1::2] *= 2.0 ** -55  # low words: under half a unit of the high words' last place
        return x
    if kind == "prepare":
        return _digits((case["count"], case["N"]), g)
    return None


# ---------------------------------------------------------------------------------------- prepare
def _unordered_plan(case):
    return cf.unordered.Plan(case["n"], cf.unordered.Method.UserProvided(cf.FftAlgo[case.get("algo", "Dif4")],
                                                                        case["base_n"]))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("slice", "ordered"):
        s["plan"] = cf.ordered.Plan(case["n"], cf.ordered.Method.UserProvided(cf.FftAlgo[case["algo"]]))
        s["x"] = _input(case, seed)
        s["work"] = np.empty_like(s["x"]) if kind == "slice" else torch.empty_like(s["x"])
    elif kind == "unordered":
        s["plan"] = _unordered_plan(case)
        s["x"] = _input(case, seed)
        s["work"] = torch.empty_like(s["x"])
    elif kind == "serde":
        s["plan"] = _unordered_plan(case)
        s["x"] = _input(case, seed)
        s["out"] = torch.empty_like(s["x"])
    elif kind == "f128":
        s["plan"] = cf.fft128.Plan(case["n"])
        s["x"] = _input(case, seed)
        s["work"] = torch.empty_like(s["x"])
    elif kind == "mixed":
        items, points = _mixed_items(case, seed)
        s["plan"] = cf.batch.Batch(items)
        s["x"] = _complex((points,), _generator(seed))
        s["work"] = torch.empty_like(s["x"])
    elif kind == "u128":
        g = _generator(seed)
        N, count = case["N"], case["count"]
        s["plan"] = cf.product.U128ProductPlan(N)
        s["a"] = _torus((count, N, 2), g)
        operands = 1 if case["shared"] else count
        s["bhat"] = torch.empty((operands, 4, N // 2), device="cuda", dtype=torch.float64)
        s["plan"].prepare_operand(_digits((operands, N), g), s["bhat"])
        s["out"] = torch.empty_like(s["a"])
    else:
        g = _generator(seed)
        N, count, terms = case["N"], case["count"], case.get("terms", 1)
        s["plan"] = cf.product.U64ProductPlan(N, cf.FftAlgo[case["algo"]], case["base_n"])
        if kind == "prepare":
            s["digits"] = _input(case, seed)
            s["bhat"] = torch.empty((count, N // 2), device="cuda", dtype=torch.complex128)
            return s
        operands = 1 if case.get("shared") else count * terms
        s["bhat"] = torch.empty((operands, N // 2), device="cuda", dtype=torch.complex128)
        if kind == "sum":  # digit polynomials times a torus-valued key
            s["plan"].prepare_operand(_torus((operands, N), g), s["bhat"])
            s["a"] = _digits((count, terms, N), g)
        else:  # torus polynomials times a digit operand
            s["plan"].prepare_operand(_digits((operands, N), g), s["bhat"])
            s["a"] = _torus((count, N), g)
        s["out"] = torch.empty((count, N), device="cuda", dtype=torch.int64)
    return s


# ---------------------------------------------------------------------------------------- run
def run(s):
    case, plan = s["case"], s["plan"]
    kind = case["kind"]
    if kind == "slice":
        np.copyto(s["work"], s["x"])
        plan.fwd(s["work"])
        return s["work"]
    if kind in ("ordered", "unordered", "f128"):
        s["work"].copy_(s["x"])
        bufs = tuple(s["work"]) if kind == "f128" else (s["work"],)
        if case["dir"] != "inv":
            plan.fwd(*bufs)
        if case["dir"] != "fwd":
            plan.inv(*bufs)
        return list(bufs) if kind == "f128" else s["work"]
    if kind == "mixed":
        s["work"].copy_(s["x"])
        return plan.run(s["work"])
    if kind == "serde":
        return plan.to_standard(s["x"], s["out"]) if case["to_standard"] else plan.from_standard(s["x"], s["out"])
    if kind == "prepare":
        return plan.prepare_operand(s["digits"], s["bhat"])
    if kind == "sum":
        return plan.product_sum(s["a"], s["bhat"], s["out"])
    return plan.product(s["a"], s["bhat"], s["out"], shared_operand=case["shared"])


# ---------------------------------------------------------------------------------------- work
def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: 5 n log2 n per n-point transform and
    8 per complex product; a double-double addition counts 11 and a product 9 (the textbook sequences)."""
    kind = case["kind"]
    passes = 2 if case.get("dir") == "fwd_inv" else 1
    if kind == "slice":
        return {"bytes": 32.0 * case["n"], "flops": _fft_flops(case["n"])}
    if kind in ("ordered", "unordered"):
        return {"bytes": 32.0 * case["n"] * case["batch"], "flops": passes * case["batch"] * _fft_flops(case["n"])}
    if kind == "serde":
        return {"bytes": 32.0 * case["n"] * case["batch"], "flops": 0.0}
    if kind == "f128":
        n = case["n"]
        return {"bytes": 64.0 * n * case["batch"], "flops": passes * case["batch"] * 0.5 * n * math.log2(n) * 102.0}
    if kind == "mixed":
        items, points = _mixed_items(case, 0)
        return {"bytes": 32.0 * points, "flops": passes * float(sum(_fft_flops(1 << int(k)) for k in items["log2n"]))}
    N, n, count, terms = case["N"], case["N"] // 2, case["count"], case.get("terms", 1)
    if kind == "prepare":
        return {"bytes": 16.0 * N * count, "flops": count * (_fft_flops(n) + 6.0 * n)}
    if kind == "sum":
        return {"bytes": 8.0 * N * count * (2 * terms + 1),
                "flops": count * ((terms + 1) * (_fft_flops(n) + 6.0 * n) + terms * 8.0 * n)}
    operands = 1 if case["shared"] else count
    if kind == "u64":
        return {"bytes": 8.0 * N * (2 * count + operands), "flops": count * (2 * _fft_flops(n) + 18.0 * n)}
    return {"bytes": 16.0 * N * (2 * count + operands), "flops": count * n * (math.log2(n) * 102.0 + 58.0)}


# ---------------------------------------------------------------------------------------- exact
def _bit_reverse(bits):
    i = np.arange(1 << bits)
    r = np.zeros_like(i)
    for k in range(bits):
        r |= ((i >> k) & 1) << (bits - 1 - k)
    return r


def _permuted_place(n, base_n):
    """place[i]: where frequency i stands in the unordered plan's order."""
    nb, bb = n.bit_length() - 1, base_n.bit_length() - 1
    rev = _bit_reverse(nb)
    low = base_n - 1
    return (rev & ~low) | _bit_reverse(bb)[rev & low]


def _dft(x, inverse):
    """Unnormalised DFT over the last dimension."""
    return torch.fft.ifft(x, norm="forward") if inverse else torch.fft.fft(x)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("u64", "sum", "u128"):
        return None  # whole numbers
    if kind == "slice":
        return np.fft.fft(_input(case, seed))
    if kind == "mixed":
        items, points = _mixed_items(case, seed)
        x = _complex((points,), _generator(seed))  # forward then inverse: n times the input
        return x * torch.from_numpy(np.repeat(np.exp2(items["log2n"]), 1 << items["log2n"].astype(np.int64))).cuda()
    if kind == "f128":
        x = _input(case, seed)
        n = case["n"]
        if case["dir"] == "fwd_inv":
            return [x[0] * n, None, x[2] * n, None]
        order = torch.from_numpy(_bit_reverse(n.bit_length() - 1)).cuda()
        angle = torch.arange(n, device="cuda", dtype=torch.float64) * (math.pi / (2 * n))
        twist = torch.polar(torch.ones_like(angle), angle)
        z = torch.complex(x[0], x[2])
        y = _dft(z * twist, True)[:, order] if case["dir"] == "fwd" else _dft(z[:, order], False) * twist.conj()
        return [y.real.contiguous(), None, y.imag.contiguous(), None]
    if kind == "prepare":
        d = _input(case, seed).double()
        n = case["N"] // 2
        angle = torch.arange(n, device="cuda", dtype=torch.float64) * (math.pi / case["N"])
        z = torch.complex(d[:, :n], d[:, n:]) * torch.polar(torch.ones_like(angle), angle)
        out = torch.empty_like(z)
        out[:, torch.from_numpy(_permuted_place(n, case["base_n"])).cuda()] = _dft(z, False)
        return out
    x = _input(case, seed)
    if kind == "ordered":
        return x * case["n"] if case["dir"] == "fwd_inv" else _dft(x, case["dir"] == "inv")
    place = torch.from_numpy(_permuted_place(case["n"], case["base_n"])).cuda()
    if kind == "serde":
        if case["to_standard"]:
            return x[:, place]
        out = torch.empty_like(x)
        out[:, place] = x
        return out
    if case["dir"] == "fwd_inv":
        return x * case["n"]
    if case["dir"] == "inv":
        return _dft(x[:, place], True)
    out = torch.empty_like(x)
    out[:, place] = _dft(x, False)
    return out
