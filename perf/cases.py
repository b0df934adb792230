"""The work that performance is measured on: convolutions, transforms and
filter spectra through the library's public entry points.

A case is a dict of plain values; `kind` says which entry points it takes:

  conv       Plan.convolve with a filter spectrum that the program keeps
             (one filter for the whole batch)
  filtered   Plan.filter_spectrum and Plan.convolve: every problem of the
             batch has a filter of its own, and the filters are new on every
             call
  transform  Plan.transform forward and back: natural order (FFT, IFFT) or
             the digit-reversed order of the butterflies (A^T, conj(A))
  uneven     MultiPlan.convolve: many problems of different shapes in a call
  dropin     permutation_avoiding_convolution{,_2d,_3d} of fft.h on host
             arrays, as a program written for the reference calls it

Sizes are those of the benchmark configurations (workloads.py), of the tests,
and generic ones between them.  Every axis is a power of its digit base (the
library takes no other); batches are any whole number.
"""
import ctypes
import importlib

import numpy as np
import torch

pac = importlib.import_module("c-permutation-avoiding-convolution_b200")
workloads = importlib.import_module("c-permutation-avoiding-convolution_b200.workloads")

FORMS = {"f64": pac.PAC_FORM_F64, "f32": pac.PAC_FORM_F32, "tc": pac.PAC_FORM_TC}


def listed():
    return [
        # one signal of 4096 points: the smallest call, bound by its launch
        {"name": "conv1d_4096_f64", "kind": "conv", "dims": "4096", "batch": 1, "bases": "2",
         "form": "f64"},
        # an odd number of short signals, every one with a new filter: an
        # adaptive filter bank
        {"name": "filtered1d_77x8192_f32", "kind": "filtered", "dims": "8192", "batch": 77,
         "bases": "2", "form": "f32"},
        # the largest: 1024 signals of 2^16 points through one FIR filter
        {"name": "conv1d_1024x65536_f32", "kind": "conv", "dims": "65536", "batch": 1024,
         "bases": "2", "form": "f32"},
        # one long recording in double precision
        {"name": "conv1d_4m_f64", "kind": "conv", "dims": "4194304", "batch": 1, "bases": "2",
         "form": "f64"},
        # one ordinary image in single precision at the reference's radix 4
        {"name": "conv2d_1024_f32_r4", "kind": "conv", "dims": "1024x1024", "batch": 1,
         "bases": "4", "form": "f32"},
        # the benchmark's image, 2048 x 2048 in double precision ...
        {"name": "conv2d_2048_f64", "kind": "conv", "dims": "2048x2048", "batch": 1,
         "bases": "2", "form": "f64"},
        # ... and in the tensor-core form
        {"name": "conv2d_2048_tc", "kind": "conv", "dims": "2048x2048", "batch": 1,
         "bases": "2", "form": "tc"},
        # a cubic volume in single precision
        {"name": "conv3d_256_f32", "kind": "conv", "dims": "256x256x256", "batch": 1,
         "bases": "2", "form": "f32"},
        # an anisotropic volume in double precision, a digit base per axis
        {"name": "conv3d_512x256x128_f64", "kind": "conv", "dims": "512x256x128", "batch": 1,
         "bases": "8,4,2", "form": "f64"},
        # a few images to the frequency domain and back, natural order
        {"name": "transform2d_5x1024x512_f64", "kind": "transform", "dims": "1024x512",
         "batch": 5, "bases": "2", "form": "f64", "order": "natural"},
        # an uneven batch: 512 signals of 2^8 .. 2^20 points and 8 images
        {"name": "uneven_512+8_f32", "kind": "uneven", "n1d": 512, "n2d": 8, "shapes": 5,
         "form": "f32"},
        # a program of the reference's: host arrays in, host arrays out
        {"name": "dropin2d_1024_r4", "kind": "dropin", "dims": "1024x1024", "batch": 1,
         "bases": "4", "form": "f64"},
    ]


def draw(rng):
    """One more case of the ranges above: any of the kinds, 1D to 3D, 2^10 to
    2^26 elements a call (2^25 in double precision; host calls to 2^22)."""
    kind = rng.choice(["conv", "conv", "conv", "conv", "filtered", "transform", "transform",
                       "uneven", "dropin"])
    form = rng.choice(["f64", "f64", "f32", "f32", "tc"] if kind == "conv" else ["f64", "f32"])
    if kind == "uneven":
        return {"kind": kind, "n1d": int(2 ** rng.uniform(3, 9)), "n2d": rng.randint(0, 8),
                "shapes": rng.randrange(1 << 20), "form": form}
    if kind == "dropin":
        form = "f64"
    rank = rng.choice([1, 1, 2, 2, 3])
    most = 22 if kind == "dropin" else 24 if kind == "filtered" else 25 if form == "f64" else 26
    total = rng.uniform(12, most)
    # the shape takes what it can of 2^total elements, the batch the rest
    lo, hi = {1: (10, 22), 2: (5, 12), 3: (3, 9)}[rank]
    if kind == "dropin":
        bases = [rng.choice([2, 4])] * rank
    elif rank > 1 and rng.random() < 0.2:
        bases = [rng.choice([2, 4, 8]) for _ in range(rank)]
    else:
        bases = [rng.choice([2, 2, 2, 4, 8])] * rank
    logs, left = [], total
    for a in range(rank):
        b = {2: 1, 4: 2, 8: 3}[bases[a]]
        rest = lo * (rank - 1 - a)
        want = rng.uniform(lo, max(lo, min(hi, left - rest)))
        lg = max(b, int(want) // b * b)
        logs.append(lg)
        left -= lg
    batch = 1
    if kind != "dropin" and left > 0:
        batch = max(1, min(4096, int(2 ** (left * rng.choice([1.0, rng.random()])))))
        if batch > 2 and rng.random() < 0.5:
            batch |= 1
    case = {"kind": kind, "dims": "x".join(str(1 << v) for v in logs), "batch": batch,
            "bases": ",".join(map(str, bases)) if len(set(bases)) > 1 else str(bases[0]),
            "form": form}
    if kind == "transform":
        case["order"] = rng.choice(["natural", "digit"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _bases(case):
    b = [int(v) for v in case["bases"].split(",")]
    return b[0] if len(b) == 1 else b


def _real(case):
    return torch.float64 if case["form"] == "f64" else torch.float32


def _normal(shape, seed, dtype, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(scale)
            for _ in range(2)]


def _filter(lead, dims, seed):
    """Filters supported on the first 1/16 of every axis, of unit power."""
    part = tuple(max(1, d // 16) for d in dims)
    out = [torch.zeros(lead + dims, device="cuda", dtype=torch.float64) for _ in range(2)]
    where = (Ellipsis,) + tuple(slice(0, p) for p in part)
    for o, v in zip(out, _normal(lead + part, seed, torch.float64, float(np.prod(part)) ** -0.5)):
        o[where] = v
    return out


def _inputs(case, seed):
    """(x re, x im, h re, h im) on the GPU; h in double precision."""
    if case["kind"] == "uneven":
        shapes = workloads.c5_shapes(case["n1d"], case["n2d"], case["shapes"])
        n = [int(np.prod(s)) for s in shapes]
        x = _normal((sum(n),), 2 * seed, _real(case))
        h = [torch.zeros(sum(n), device="cuda", dtype=torch.float64) for _ in range(2)]
        at = 0
        for p, s in enumerate(shapes):
            for o, v in zip(h, _filter((), s, (2 * seed + 1) * 8192 + p)):
                o[at:at + n[p]] = v.reshape(-1)
            at += n[p]
        return x + h
    dims = _dims(case)
    x = _normal((case["batch"],) + dims, 2 * seed, _real(case))
    if case["kind"] == "transform":
        return x
    lead = (case["batch"],) if case["kind"] == "filtered" else ()
    return x + _filter(lead, dims, 2 * seed + 1)


def _ptr(tensors):
    return [t.data_ptr() for t in tensors]


_stream = None


def prepare(case, seed):
    global _stream
    L = pac.load()
    kind, form = case["kind"], FORMS[case["form"]]
    state = {"kind": kind, "L": L, "in": _inputs(case, seed)}
    if kind == "dropin":
        dims, base = _dims(case), _bases(case)
        state["in"] = [t.reshape(dims).cpu().numpy() for t in state["in"]]
        state["out"] = [np.empty_like(a) for a in state["in"]]
        state["f"] = getattr(L, "permutation_avoiding_convolution" +
                             ("" if len(dims) == 1 else "_%dd" % len(dims)))
        re, im, hr, hi = (a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in state["out"])
        state["args"] = [re, im, *dims, base] + [None] * (2 * len(dims)) + [hr, hi]
        return state
    x = state["in"][:2]
    real = x[0].dtype
    if kind == "uneven":
        # one stream for every multi-plan of the program (its launches are
        # recorded once and replayed on a stream of the caller's)
        if _stream is None:
            _stream = torch.cuda.Stream()
        state["stream"] = _stream.cuda_stream
        shapes = workloads.c5_shapes(case["n1d"], case["n2d"], case["shapes"])
        state["plan"] = plan = pac.MultiPlan(L, shapes, 2, form)
        state["hhat"] = [torch.empty(x[0].shape, device="cuda", dtype=real) for _ in range(2)]
        plan.filter_spectra(*_ptr(state["in"][2:]), *_ptr(state["hhat"]))
    else:
        state["plan"] = plan = pac.Plan(L, _dims(case), case["batch"], _bases(case), form)
        if kind in ("conv", "filtered"):
            state["hhat"] = [torch.empty(h.shape, device="cuda", dtype=real)
                             for h in state["in"][2:]]
        if kind == "conv":
            plan.filter_spectrum(*_ptr(state["in"][2:]), *_ptr(state["hhat"]))
        if kind == "transform":
            state["ops"] = ((pac.OP_FFT, pac.OP_IFFT) if case["order"] == "natural"
                            else (pac.OP_AT, pac.OP_CONJ_A))
            state["mid"] = [torch.empty_like(t) for t in x]
    if kind in ("conv", "uneven"):
        state["in"] = x  # the program keeps the spectrum, not the filter
    state["out"] = [torch.empty_like(t) for t in x]
    state["batch"] = case.get("batch", 1)
    torch.cuda.synchronize()
    return state


def run(state):
    kind, out = state["kind"], state["out"]
    if kind == "dropin":
        # the call overwrites the signal and the filter
        for dst, src in zip(out, state["in"]):
            np.copyto(dst, src)
        state["f"](*state["args"])
        return out
    plan, x = state["plan"], state["in"]
    if kind == "conv":
        plan.convolve(*_ptr(x), *_ptr(state["hhat"]), *_ptr(out))
        return out
    if kind == "filtered":
        plan.filter_spectrum(*_ptr(x[2:]), *_ptr(state["hhat"]), nfilters=state["batch"])
        plan.convolve(*_ptr(x[:2]), *_ptr(state["hhat"]), *_ptr(out), per_problem=1)
        return out
    if kind == "uneven":
        plan.convolve(*_ptr(x), *_ptr(state["hhat"]), *_ptr(out), state["stream"])
        return out
    mid = state["mid"]
    plan.transform(state["ops"][0], *_ptr(x), *_ptr(mid))
    plan.transform(state["ops"][1], *_ptr(mid), *_ptr(out))
    return mid + out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    size = 8 if case["form"] == "f64" else 4
    if case["kind"] == "uneven":
        n = [int(np.prod(s)) for s in
             workloads.c5_shapes(case["n1d"], case["n2d"], case["shapes"])]
        total = float(sum(n))
        return {"bytes": 6 * size * total,
                "flops": float(sum(10 * v * np.log2(v) + 6 * v for v in n))}
    one = float(np.prod(_dims(case)))
    total = one * case["batch"]
    flops = 10 * total * np.log2(one)  # two transforms of 5 N log2 N
    if case["kind"] == "transform":  # x in, the spectrum and the signal out
        return {"bytes": 6 * size * total, "flops": flops}
    if case["kind"] == "dropin":  # x and h in and out
        return {"bytes": 8 * size * total, "flops": 1.5 * flops + 6 * total}
    if case["kind"] == "filtered":  # x and double-precision h in, y out
        return {"bytes": (4 * size + 16) * total, "flops": 1.5 * flops + 6 * total}
    return {"bytes": 4 * size * total + 2 * size * one, "flops": flops + 6 * total}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _complex(re, im):
    return torch.complex(re.double(), im.double())


def _parts(z):
    return [z.real.contiguous(), z.imag.contiguous()]


def _reversal(n, base):
    """Digit reversal of 0 .. n-1 in `base`."""
    i, r, v = np.arange(n), np.zeros(n, np.int64), n
    while v > 1:
        r = r * base + i % base
        i //= base
        v //= base
    return torch.from_numpy(r)


def _digit_order(z, dims, bases):
    """The last len(dims) axes of z in digit-reversed order."""
    for a, n in enumerate(dims):
        b = bases[a] if isinstance(bases, list) else bases
        z = z.index_select(z.dim() - len(dims) + a, _reversal(n, b).to(z.device))
    return z


def exact(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "uneven":
        shapes = workloads.c5_shapes(case["n1d"], case["n2d"], case["shapes"])
        at, ys = 0, []
        for s in shapes:
            n = int(np.prod(s))
            xr, xi, hr, hi = (t[at:at + n].reshape(s) for t in x)
            ys.append(torch.fft.ifftn(torch.fft.fftn(_complex(xr, xi)) *
                                      torch.fft.fftn(_complex(hr, hi))).reshape(-1))
            at += n
        return _parts(torch.cat(ys))
    dims, bases = _dims(case), _bases(case)
    axes = tuple(range(-len(dims), 0))
    xs = torch.fft.fftn(_complex(*x[:2]), dim=axes)
    if case["kind"] == "transform":
        if case["order"] == "natural":
            return _parts(xs) + [t.double() for t in x]
        # conj(A) A^T x = N x
        n = float(np.prod(dims))
        return _parts(_digit_order(xs, dims, bases)) + [t.double() * n for t in x]
    hs = torch.fft.fftn(_complex(*x[2:]), dim=axes)
    y = torch.fft.ifftn(xs * hs, dim=axes)
    if case["kind"] == "dropin":
        return ([t.reshape(dims) for t in _parts(y)] +
                _parts(_digit_order(hs, dims, bases)))
    return _parts(y)
