"""The calls whose time is tracked: transforms as a user of this framework makes them, through the
public entry points of fmm-fft_b200/fmmfft.py.

A case names one entry point ("kind"), a shape (N = 2^log2n points in P blocks, `terms` Chebyshev
terms, b points per leaf box) and the plan's precision:

  execute    one transform of a device vector                  Plan.__call__
  inverse    the unnormalised inverse transform                Plan.__call__(inverse=True)
  graph      one transform through the plan's CUDA graph       Plan.execute_graph_ptr
  many       `count` transforms of one shape, contiguous       Plan.execute_many_ptr
  refined    complex64 in, FP64 residual-corrected out         Plan.execute_refined_ptr
  mft        the reference's call on host memory, complex128   mfti / mft
  uneven     transforms of mixed shapes as one graph           Batch.launch
  plain_fft  the conventional FFT beside the FMM-FFT           PlainFFT.execute_ptr

Inputs are iid N(0, 1) complex values, as in the benchmark.  Shapes follow the benchmark's own
workloads (the single large transform, the precision sweep, the served requests, the uneven batch)
and the reference's recorded runs (b = 32 with 15 terms, b = 2048 with 16).
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmm-fft_b200"))
import fmmfft  # noqa: E402


def listed():
    return [
        # the smallest request of the served mix in its 1e-4 class: launches and latency only
        dict(name="smallest_request", kind="graph", log2n=10, P=2, terms=8, b=32, precision="f32_tc"),
        # an ordinary small request in the 1e-6 class
        dict(name="small_request", kind="graph", log2n=14, P=32, terms=20, b=32, precision="f32_tc"),
        # the reference's arithmetic at its recorded order: FP64, an odd number of terms
        dict(name="reference_order_f64", kind="execute", log2n=20, P=32, terms=15, b=32, precision="f64"),
        # the reference's own call and its wide-box configuration, host memory in and out
        dict(name="reference_call_host", kind="mft", log2n=16, P=4, terms=16, b=2048, precision="f64"),
        # FP64-accurate results of complex64 data: two FP32 transforms and an FP64 inverse
        dict(name="refined", kind="refined", log2n=20, P=64, terms=16, b=32, precision="f32"),
        # the inverse direction on the CUDA-core FP32 plan
        dict(name="inverse_f32", kind="inverse", log2n=20, P=64, terms=20, b=32, precision="f32"),
        # the headline: one large transform on the tensor-core plan
        dict(name="single_large", kind="execute", log2n=24, P=64, terms=24, b=32, precision="f32_tc"),
        # the precision sweep's size, the largest transform of the benchmark
        dict(name="largest", kind="execute", log2n=26, P=256, terms=16, b=32, precision="f32_tc"),
        # the 1e-4 accuracy class in BF16x3
        dict(name="class_1e4_bf16x3", kind="execute", log2n=22, P=64, terms=8, b=32, precision="bf16x3"),
        # continuous batching: equal requests in one launch sequence
        dict(name="batch", kind="many", log2n=16, P=64, terms=20, b=32, precision="f32_tc", count=16),
        # many unequal transforms as one graph
        dict(name="uneven_batch", kind="uneven", jobs=48, jobs_seed=4, log2n_lo=12, log2n_hi=18, terms=16, b=32,
             precision="f32_tc"),
        # the conventional FFT that the reference times beside its own
        dict(name="plain_fft", kind="plain_fft", log2n=22, precision="f32"),
    ]


def draw(rng):
    """A case of the same kinds: log2 N over the whole range (sizes are powers of two by the
    transform's definition), any number of terms, odd ones among them, any batch count."""
    kind = rng.choice(["execute", "execute", "execute", "graph", "many", "inverse", "refined", "mft", "uneven",
                       "plain_fft"])
    if kind == "plain_fft":
        return dict(kind=kind, log2n=rng.randint(8, 24), precision=rng.choice(["f32", "f64"]))
    if kind == "uneven":
        return dict(kind=kind, jobs=rng.randint(9, 48), jobs_seed=rng.randint(0, 1 << 20), log2n_lo=12, log2n_hi=18,
                    terms=rng.randint(8, 24), b=32, precision=rng.choice(["f32", "f32_tc"]))
    if kind == "mft":
        log2n, b = rng.randint(12, 18), rng.choice([32, 32, 256, 2048])
        P = 1 << rng.randint(1, 5)
        while (1 << log2n) // P < 4 * b:
            log2n += 1
        return dict(kind=kind, log2n=log2n, P=P, terms=rng.randint(12, 18), b=b, precision="f64")
    precision = {"refined": rng.choice(["f32", "f32_tc"]), "many": rng.choice(["f32_tc", "f32_tc", "f32"]),
                 "graph": rng.choice(["f32_tc", "f32_tc", "f32"])}.get(
                     kind, rng.choice(["f32_tc", "f32_tc", "f32", "f64", "bf16x3"]))
    lo, hi = {"graph": (10, 18), "many": (10, 18), "refined": (14, 21)}.get(kind, (10, 24))
    if precision == "f64":
        hi = min(hi, 22)
    log2n = rng.randint(lo, hi)
    b = rng.choice([16, 32, 32, 32, 64])
    P = 1 << rng.randint(1, 8)
    while P > 2 and (1 << log2n) // P < max(256, 4 * b):
        P //= 2
    while (1 << log2n) // P < 4 * b:
        b //= 2
    while (1 << log2n) // P > 1 << 20:
        P *= 2
    terms = rng.randint(8, 12) if precision == "bf16x3" else rng.randint(16, 24) if kind == "refined" else \
        rng.choice([8, 12, 15, 16, 20, 24, rng.randint(8, 32)])
    case = dict(kind=kind, log2n=log2n, P=P, terms=terms, b=b, precision=precision)
    if kind == "many":
        case["count"] = rng.randint(2, 24)
    return case


def _jobs(case):
    """Shapes of an uneven batch: N log-uniform, P from {8, 16, 32, 64} with N / P >= 256; grouped
    by shape as (N, P, transforms)."""
    rng = random.Random(case["jobs_seed"])
    groups = {}
    while sum(groups.values()) < case["jobs"]:
        N, P = 1 << rng.randint(case["log2n_lo"], case["log2n_hi"]), rng.choice([8, 16, 32, 64])
        if N // P >= 256:
            groups[(N, P)] = groups.get((N, P), 0) + 1
    return [(N, P, c) for (N, P), c in sorted(groups.items())]


def _dtype(case):
    return torch.complex128 if case["precision"] == "f64" else torch.complex64


def _total(case):
    if case["kind"] == "uneven":
        return sum(N * c for N, P, c in _jobs(case))
    return (1 << case["log2n"]) * case.get("count", 1)


def _input(case, seed):
    """iid N(0, 1) real and imaginary parts."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float64 if case["precision"] == "f64" else torch.float32
    return torch.view_as_complex(torch.randn(_total(case), 2, generator=gen, device="cuda", dtype=real))


def prepare(case, seed):
    kind, x = case["kind"], _input(case, seed)
    state = dict(kind=kind, x=x)
    if kind == "plain_fft":
        state.update(plan=fmmfft.PlainFFT(1 << case["log2n"], case["precision"]), y=torch.empty_like(x))
        return state
    if kind == "uneven":
        jobs = _jobs(case)
        y = torch.empty_like(x)
        at, ins, outs, plans = 0, [], [], []
        for N, P, c in jobs:
            plans.append(fmmfft.Plan(N, P, case["terms"], case["b"], case["precision"], max_transforms=c))
            ins.append(x[at:].data_ptr())
            outs.append(y[at:].data_ptr())
            at += N * c
        state.update(y=y, batch=fmmfft.Batch(plans, ins, outs, nbranch=16, counts=[c for _, _, c in jobs]))
        return state
    N, P, T, b = 1 << case["log2n"], case["P"], case["terms"], case["b"]
    if kind == "mft":
        lq = N // P
        w, v = np.zeros(fmmfft.getwlen2(lq, T, P, b)), np.zeros(fmmfft.getvlen(lq, T, P, b))
        fmmfft.mfti(lq, P, T, b, w, v)
        h = x.cpu().numpy()
        state.update(x=h, q=np.empty_like(h), w=w, v=v, lq=lq, P=P, terms=T, b=b)
        return state
    plan = fmmfft.Plan(N, P, T, b, case["precision"], max_transforms=case.get("count", 1))
    state.update(plan=plan, y=torch.empty_like(x), count=case.get("count", 1))
    if kind == "refined":
        plan.enable_refinement()
        state["y"] = torch.empty(N, dtype=torch.complex128, device="cuda")
    return state


def run(state):
    kind, x = state["kind"], state["x"]
    if kind == "mft":
        np.copyto(state["q"], x)  # the transform is in place: the caller fills its buffer
        fmmfft.mft(state["lq"], state["q"], 1, state["P"], 0, state["terms"], state["b"], state["w"], state["v"])
        return state["q"]
    y = state["y"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "execute":
        state["plan"](x, out=y)
    elif kind == "inverse":
        state["plan"](x, out=y, inverse=True)
    elif kind == "graph":
        state["plan"].execute_graph_ptr(x.data_ptr(), y.data_ptr(), stream)
    elif kind == "many":
        state["plan"].execute_many_ptr(state["count"], x.data_ptr(), y.data_ptr(), stream)
    elif kind == "refined":
        state["plan"].execute_refined_ptr(x.data_ptr(), y.data_ptr(), stream)
    elif kind == "uneven":
        state["batch"].launch(stream)
    else:
        state["plan"].execute_ptr(x.data_ptr(), y.data_ptr(), stream)
    return y


def work(case):
    """Each input read and each output written once; the arithmetic of the FMM's contractions (2
    planes of P - 1 sections: S2M, M2M, M2L + L2L, L2T and the near field over three boxes) and of
    the FFTs."""
    size = 16 if case["precision"] == "f64" else 8
    total = _total(case)

    def fmm(N, P, T, b):
        boxes = 2 * (P - 1) * (N // P // b)
        return 2.0 * boxes * (2 * T * b + 10 * T * T + 3 * b * b) + 5.0 * N * math.log2(N)

    kind = case["kind"]
    if kind == "plain_fft":
        return dict(bytes=2 * size * total, flops=5.0 * total * case["log2n"])
    if kind == "uneven":
        return dict(bytes=2 * size * total, flops=sum(c * fmm(N, P, case["terms"], case["b"]) for N, P, c in _jobs(case)))
    one = fmm(1 << case["log2n"], case["P"], case["terms"], case["b"])
    if kind == "refined":
        return dict(bytes=24 * total, flops=3 * one)
    return dict(bytes=2 * size * total, flops=one * case.get("count", 1))


def exact(case, seed):
    """The discrete Fourier transform of the same inputs in FP64."""
    x = _input(case, seed).to(torch.complex128)
    kind = case["kind"]
    if kind == "inverse":
        return torch.fft.ifft(x, norm="forward")
    if kind == "many":
        return torch.fft.fft(x.view(case["count"], -1)).reshape(-1)
    if kind == "uneven":
        at, parts = 0, []
        for N, P, c in _jobs(case):
            parts.append(torch.fft.fft(x[at:at + N * c].view(c, N)).reshape(-1))
            at += N * c
        return torch.cat(parts)
    y = torch.fft.fft(x)
    return y.cpu().numpy() if kind == "mft" else y
