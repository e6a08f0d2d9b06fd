"""The work this library is asked for, as cases that can be timed and compared.

A case is a dict of plain values.  `kind` says which public entry point it goes through:

  sgemm    tcec.sgemm                  one product on device operands
  strided  tcec.sgemm_strided_batched  a batch with a uniform stride
  pointers tcec_sgemm_batched_cublas   a batch by device pointer tables, cuBLAS's argument list (C ABI)
  packed   tcec.pack_a + sgemm_packed  B split once beforehand, every call brings a new A
  complex  tcec.cgemm                  one complex64 product
  host     tcec.sgemm_host             operands and result in pinned host memory
"""
import ctypes
import math

import torch

from wmma_extension_b200 import tcec

DEVICE = "cuda:0"


def _sgemm(m, n, k, policy="fp16_ec", values="uniform", layouts="rrr", alpha=1.0, beta=0.0):
    return {"kind": "sgemm", "m": m, "n": n, "k": k, "policy": policy, "values": values, "layouts": layouts,
            "alpha": alpha, "beta": beta}


def listed():
    return [
        # The reference's unit-test shape (one warp's 32 x 32 x 32 tile): what a caller with many
        # small, dependent products sees is the latency of one call.
        dict(_sgemm(32, 32, 32), name="tile_32"),
        # An ordinary call from numerical code: nothing is a multiple of anything, B and C are
        # column-major as from Fortran or BLAS code, and C is updated in place.
        dict(_sgemm(1000, 777, 1111, layouts="rcc", alpha=1.5, beta=0.5), name="ragged_1000"),
        # Square product, FP32 row-major, U(-1, 1), half policy: the ordinary large call.
        dict(_sgemm(4096, 4096, 4096), name="square_4096"),
        # The size the throughput target is stated at; the longest single call.
        dict(_sgemm(16384, 16384, 16384), name="square_16384"),
        # Values spread over 2^-15..2^15 overflow fp16 heads: the tf32 policy is the one to use.
        dict(_sgemm(8192, 8192, 8192, policy="tf32_ec", values="wide"), name="wide_tf32_8192"),
        # Without error correction: the caller takes half precision of the inputs for speed.
        dict(_sgemm(8192, 8192, 8192, policy="fp16_no_ec"), name="no_ec_8192"),
        # Batched configuration of the benchmark: 8192 independent 256^3 products, N(0, 1).
        {"name": "batch_256", "kind": "strided", "m": 256, "n": 256, "k": 256, "batch": 8192, "policy": "fp16_ec"},
        # Many small matrices (blocks, heads, elements): memory-bound, one tile or less each.
        {"name": "batch_64", "kind": "strided", "m": 64, "n": 64, "k": 64, "batch": 16384, "policy": "fp16_ec"},
        # The reference's benchmark call: cublasSgemmBatched(OP_T, OP_N), batch 256, m = n = 512.
        {"name": "pointers_512", "kind": "pointers", "m": 512, "n": 512, "k": 512, "batch": 256, "policy": "fp16_ec"},
        # A layer applied to a few rows at a time: B is split once and kept, A is new in every call.
        {"name": "packed_rows_64", "kind": "packed", "m": 64, "n": 4096, "k": 4096, "policy": "fp16_ec"},
        # Complex product, interleaved storage.
        {"name": "complex_2048", "kind": "complex", "m": 2048, "n": 2048, "k": 2048, "policy": "fp16_ec"},
        # Operands that live in (pinned) host memory: copy in, multiply, copy out.
        {"name": "host_8192", "kind": "host", "m": 8192, "n": 8192, "k": 8192, "policy": "fp16_ec"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _within(rng, lo, hi, most, dims=3):
    """`dims` extents spread over the logarithm of lo..hi whose product is at most `most`."""
    while True:
        d = [_log(rng, lo, hi) for _ in range(dims)]
        if math.prod(d) <= most:
            return d


def draw(rng):
    family = rng.choice(["tile", "ragged", "large", "wide", "no_ec", "batch_mid", "batch_small", "pointers", "packed",
                         "complex", "host"])
    ec = rng.choice(["fp16_ec", "fp16_ec", "tf32_ec"])
    if family == "tile":
        return _sgemm(_log(rng, 4, 128), _log(rng, 4, 128), _log(rng, 4, 128), policy=ec)
    if family == "ragged":
        m, n, k = (_log(rng, 128, 3000) for _ in range(3))
        # |beta| < 1: a call repeated on one C keeps it bounded
        alpha, beta = rng.choice([(1.0, 0.0), (1.0, -0.25), (1.5, 0.5), (-0.5, 0.0)])
        return _sgemm(m, n, k, policy=ec, layouts="".join(rng.choice("rc") for _ in range(3)), alpha=alpha, beta=beta)
    if family == "large":
        m, n, k = _within(rng, 1024, 16384, 12288 ** 3)
        return _sgemm(m, n, k)
    if family == "wide":
        m, n, k = _within(rng, 512, 10000, 8192 ** 3)
        return _sgemm(m, n, k, policy="tf32_ec", values="wide")
    if family == "no_ec":
        m, n, k = _within(rng, 512, 12000, 8192 ** 3)
        return _sgemm(m, n, k, policy=rng.choice(["fp16_no_ec", "fp16_no_ec", "tf32_no_ec"]))
    if family == "batch_mid":
        m, n, k = (rng.randrange(130, 513) for _ in range(3))
        most = (8192 * 3 * 65536) // (m * k + k * n + m * n)
        return {"kind": "strided", "m": m, "n": n, "k": k, "batch": _log(rng, 64, min(8192, most)), "policy": ec}
    if family == "batch_small":
        m, n, k = (rng.randrange(8, 129) for _ in range(3))
        return {"kind": "strided", "m": m, "n": n, "k": k, "batch": _log(rng, 500, 16384), "policy": ec}
    if family == "pointers":
        m, k = _log(rng, 256, 1024), _log(rng, 128, 2048)
        return {"kind": "pointers", "m": m, "n": m, "k": k, "batch": rng.randrange(16, 257), "policy": ec}
    if family == "packed":
        return {"kind": "packed", "m": _log(rng, 1, 1024), "n": _log(rng, 512, 8192), "k": _log(rng, 512, 8192),
                "policy": ec}
    if family == "complex":
        m, n, k = _within(rng, 100, 4096, 3000 ** 3)
        return {"kind": "complex", "m": m, "n": n, "k": k, "policy": ec}
    m, n, k = _within(rng, 1000, 8192, 6144 ** 3)
    return {"kind": "host", "m": m, "n": n, "k": k, "policy": ec}


def _values(gen, kind, *shape):
    if kind == "normal":
        return torch.randn(shape, generator=gen, device=DEVICE)
    u = torch.rand(shape, generator=gen, device=DEVICE)
    if kind == "uniform":
        return u.mul_(2).sub_(1)
    # sign * U[1, 2) * 2^U{-15..15}
    e = torch.randint(-15, 16, shape, generator=gen, device=DEVICE)
    sign = torch.randint(0, 2, shape, generator=gen, device=DEVICE).mul_(2).sub_(1)
    return torch.ldexp(u.add_(1), e).mul_(sign)


def _matrix(gen, kind, rows, cols, layout):
    """rows x cols view of row-major ("r") or column-major ("c") storage."""
    return _values(gen, kind, rows, cols) if layout == "r" else _values(gen, kind, cols, rows).t()


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind, m, n, k = case["kind"], case["m"], case["n"], case["k"]
    s = dict(case)
    if kind == "sgemm":
        la, lb, lc = case["layouts"]
        s["a"] = _matrix(gen, case["values"], m, k, la)
        s["b"] = _matrix(gen, case["values"], k, n, lb)
        # a fresh row-major result is left to the call to allocate
        s["c"] = None if case["beta"] == 0.0 and lc == "r" else _matrix(gen, "uniform", m, n, lc)
    elif kind == "strided":
        s["a"] = _values(gen, "normal", case["batch"], m, k)
        s["b"] = _values(gen, "normal", case["batch"], k, n)
        s["c"] = torch.empty((case["batch"], m, n), device=DEVICE)
    elif kind == "pointers":
        # OP_T, OP_N: A is k x m and B is k x n in column-major storage, C is m x n column-major
        s["a"] = _values(gen, "normal", case["batch"], m, k)
        s["b"] = _values(gen, "normal", case["batch"], n, k)
        s["c"] = torch.empty((case["batch"], n, m), device=DEVICE)
        s["tables"] = [torch.tensor([x.data_ptr() for x in s[key]], dtype=torch.int64, device=DEVICE)
                       for key in ("a", "b", "c")]
    elif kind == "packed":
        s["a"] = _values(gen, "normal", m, k)
        s["b_packed"] = tcec.pack_b(_values(gen, "normal", k, n), case["policy"])
    elif kind == "complex":
        s["a"] = torch.complex(_values(gen, "uniform", m, k), _values(gen, "uniform", m, k))
        s["b"] = torch.complex(_values(gen, "uniform", k, n), _values(gen, "uniform", k, n))
    else:
        s["a"] = torch.empty((m, k), pin_memory=True).copy_(_values(gen, "uniform", m, k))
        s["b"] = torch.empty((k, n), pin_memory=True).copy_(_values(gen, "uniform", k, n))
        s["c"] = torch.empty((m, n), pin_memory=True)
    return s


def run(state):
    s = state
    kind, policy = s["kind"], s["policy"]
    if kind == "sgemm":
        return tcec.sgemm(s["a"], s["b"], s["c"], alpha=s["alpha"], beta=s["beta"], policy=policy)
    if kind == "strided":
        return tcec.sgemm_strided_batched(s["a"], s["b"], s["c"], policy=policy)
    if kind == "pointers":
        one, zero = ctypes.c_float(1.0), ctypes.c_float(0.0)
        pa, pb, pc = s["tables"]
        status = tcec.load().tcec_sgemm_batched_cublas(
            1, 0, s["m"], s["n"], s["k"], ctypes.byref(one), pa.data_ptr(), s["k"], pb.data_ptr(), s["k"],
            ctypes.byref(zero), pc.data_ptr(), s["m"], s["batch"], tcec.POLICIES[policy],
            torch.cuda.current_stream().cuda_stream)
        if status != tcec.OK:
            raise tcec.TcecError(status, "tcec_sgemm_batched_cublas")
        return s["c"]
    if kind == "packed":
        a_packed = tcec.pack_a(s["a"], policy)
        return tcec.sgemm_packed(a_packed, s["b_packed"], s["m"], s["n"], s["k"], policy=policy)
    if kind == "complex":
        return tcec.cgemm(s["a"], s["b"], policy=policy)
    return tcec.sgemm_host(s["a"], s["b"], s["c"], policy=policy)


def work(case):
    m, n, k = case["m"], case["n"], case["k"]
    batch = case.get("batch", 1)
    width = 8 if case["kind"] == "complex" else 4
    products = 1 if case["policy"].endswith("no_ec") else 3
    if case["kind"] == "complex":
        products *= 4
    c_reads = 1 if case.get("beta", 0.0) != 0.0 else 0
    b_width = width
    if case["kind"] == "packed":  # B arrives split: two halves (fp16) or two words (tf32) per element
        b_width = 8 if case["policy"].startswith("tf32") else 4
    return {"bytes": batch * (width * (m * k + m * n * (1 + c_reads)) + b_width * k * n),
            "flops": 2.0 * products * batch * m * n * k}


def tolerance(case):
    # About four times what was measured against FP64 products of the same operands and against the
    # same products summed in other chunks: with error correction 2.4e-7 (largest 1.4e-6) up to a
    # K of 4096 and 6.3e-7 (2.9e-6) above; without it the inputs' rounding is the same in every
    # implementation and the sums differ by 9.6e-6 (3.7e-5).
    if case["policy"].endswith("no_ec"):
        return {"rel": 4e-5, "max": 1.5e-4}
    terms = case["k"] * (2 if case["kind"] == "complex" else 1)
    return {"rel": 1e-6, "max": 6e-6} if terms <= 4096 else {"rel": 2.5e-6, "max": 1.2e-5}


def exact(case, seed):
    """What run(prepare(case, seed)) returns, from FP64 products of the same operands."""
    s = prepare(dict(case, kind="sgemm", values="normal", layouts="rrr", beta=0.0) if case["kind"] == "packed" else case,
                seed)
    kind = case["kind"]
    if kind == "complex":
        return s["a"].to(torch.complex128) @ s["b"].to(torch.complex128)
    if kind == "host":
        return (s["a"].to(DEVICE).double() @ s["b"].to(DEVICE).double()).cpu()
    if kind == "pointers":  # column-major storage: c holds the transpose of a^T b
        return torch.bmm(s["b"].double(), s["a"].double().transpose(1, 2))
    if kind == "strided":
        return torch.bmm(s["a"].double(), s["b"].double())
    c = s["a"].double() @ s["b"].double()
    if kind == "sgemm":
        c *= case["alpha"]
        if case["beta"] != 0.0:
            c += case["beta"] * s["c"].double()
    return c
