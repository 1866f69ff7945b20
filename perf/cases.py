"""Workloads that stand for what a program does with this library, with their
inputs, one pass through the public entry points, and the exact results.

Every case is one of seven kinds of call:

  product    one FP32 product on device matrices (``Handle.cgemm3m`` or
             ``Handle.cgemm``), the drop-in call
  tensor     one product in a tensor-core form, any shape (no rounding pass)
  pass       one contiguous square unit product of order 2048..4096, which runs
             the rounding-correction pass
  strided    a strided batch of equal problems
  batch      a planned batch of unequal problems, executed as one launch
  train      the differentiable form, forward and backward
  host       one product on host matrices (page-locked buffers)

Matrices are column-major complex64, as everywhere in the library; a matrix of
c columns with leading dimension ld is a tensor of shape (c, ld).
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ascend-open-source-contributions_b200"))

import cg3m  # noqa: E402
from cg3m.autograd import cgemm3m_autograd  # noqa: E402
from cg3m.workloads import batch_shapes, stored_shape  # noqa: E402

PAIRS = [a + b for a in "NTC" for b in "NTC"]


def listed():
    return [
        # The smallest useful product: latency of one call.
        dict(name="product_32", kind="product", call="cgemm3m", ops="NN", m=32, n=32, k=32, pad=0, unit=True),
        # The plain drop-in call of ordinary size, with general scalars.
        dict(name="product_512", kind="product", call="cgemm3m", ops="NN", m=512, n=512, k=512, pad=0, unit=False),
        # Odd sizes, both operands transposed or conjugated, padded leading dimensions.
        dict(name="product_ragged", kind="product", call="cgemm3m", ops="CT", m=1000, n=777, k=3001, pad=13,
             unit=False),
        # A small output over a very long inner dimension.
        dict(name="product_long_k", kind="product", call="cgemm3m", ops="NN", m=128, n=128, k=65536, pad=0,
             unit=True),
        # The drop-in exactly as called on a large contiguous square: the rounding pass is on.
        dict(name="pass_fp32_2048", kind="pass", form="fp32", ops="NC", n=2048, data="uniform"),
        # The precision form at full size, on data that cancels in the imaginary part.
        dict(name="pass_bf16x6_4096", kind="pass", form="bf16x6", ops="NN", n=4096, data="precision"),
        # A tensor-core form with the pass on data that rarely cancels.
        dict(name="pass_tf32x3_3072", kind="pass", form="tf32x3", ops="CN", n=3072, data="uniform"),
        # A rectangular product on the tensor cores, sizes off every tile.
        dict(name="tensor_rect", kind="tensor", form="bf16x6", ops="NT", m=1500, n=3100, k=2000, pad=0, unit=False),
        # Many equal problems in one call.
        dict(name="strided_64", kind="strided", ops="TN", m=256, n=192, k=320, batch=64, unit=False),
        # Many unequal problems, planned once and executed repeatedly.
        dict(name="batch_512", kind="batch", count=512, lo=16, hi=1024, shape_seed=20261029),
        # A training step's products: forward, and both gradients backward.
        dict(name="train_16", kind="train", form="bf16x6", ops="NN", batch=16, m=1024, n=1024, k=1024),
        # Matrices that live in host memory, at full size.
        dict(name="host_4096", kind="host", form="bf16x6", ops="NN", m=4096, n=4096, k=4096, data="precision"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "tensor", "pass", "strided", "batch", "train", "host"])
    ops = rng.choice(PAIRS)
    if kind == "product":
        m, n = _log(rng, 16, 2048), _log(rng, 16, 2048)
        k = _log(rng, 16, 65536 if m * n <= 256 * 256 else 4096)
        return dict(kind=kind, call=rng.choice(["cgemm3m", "cgemm3m", "cgemm"]), ops=ops, m=m, n=n, k=k,
                    pad=rng.choice([0, 0, 13]), unit=rng.random() < 0.5)
    if kind == "tensor":
        return dict(kind=kind, form=rng.choice(["tf32x3", "bf16x6", "bf16x9"]), ops=ops, m=_log(rng, 200, 4096),
                    n=_log(rng, 200, 4096), k=_log(rng, 200, 4096), pad=rng.choice([0, 0, 13]),
                    unit=rng.random() < 0.5)
    if kind == "pass":
        # The FP32 pass costs several times the tensor-core forms' time per output.
        form = rng.choice(["fp32", "tf32x3", "bf16x6", "bf16x9"])
        return dict(kind=kind, form=form, ops=ops, n=rng.randint(2048, 2600 if form == "fp32" else 4096),
                    data="uniform" if form == "fp32" else rng.choice(["uniform", "precision"]))
    if kind == "strided":
        return dict(kind=kind, ops=ops, m=_log(rng, 24, 512), n=_log(rng, 24, 512), k=_log(rng, 24, 512),
                    batch=_log(rng, 4, 128), unit=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 48, 512), lo=16, hi=rng.choice([256, 512, 1024]),
                    shape_seed=rng.randrange(1 << 20))
    if kind == "train":
        return dict(kind=kind, form=rng.choice(["fp32", "bf16x6", "bf16x6", "tf32x3"]), ops=ops,
                    batch=rng.choice([0, 2, 4, 8, 16]), m=_log(rng, 128, 1024), n=_log(rng, 128, 1024),
                    k=_log(rng, 128, 1024))
    return dict(kind=kind, form=rng.choice(["fp32", "bf16x6", "bf16x6"]), ops=ops, m=_log(rng, 256, 3000),
                n=_log(rng, 256, 3000), k=_log(rng, 256, 3000), data="uniform")


# ---- inputs -------------------------------------------------------------------------

def _shapes(case):
    """Stored (rows, columns) of A and B."""
    ops = case["ops"]
    m, n, k = case.get("m", case["n"]), case["n"], case.get("k", case["n"])
    return stored_shape(ops[0], m, k), stored_shape(ops[1], k, n), (m, n, k)


def _uniform(gen, *shape, scale=1.0):
    x = torch.rand(*shape, 2, generator=gen, device="cuda").mul_(2 * scale).sub_(scale)
    return torch.view_as_complex(x)


def _matrix(gen, rows, cols, ld, data):
    """Column-major rows x cols matrix with leading dimension ld, as (cols, ld)."""
    if data == "precision":
        # Re ~ N(0, 1); Im ~ N(0, 1) 2^e, one e in [-8, 8] per column
        x = torch.randn(cols, ld, 2, generator=gen, device="cuda")
        e = torch.rand(cols, 1, generator=gen, device="cuda").mul_(16).sub_(8)
        x[:, :, 1] *= torch.exp2(e)
        return torch.view_as_complex(x)
    return _uniform(gen, cols, ld, scale=5.0 if data == "uniform" else 1.0)


def _scalars(case):
    return (1.0, 0.0) if case.get("unit", True) else (complex(0.7, 0.3), complex(-0.5, 0.4))


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _inputs(case, seed):
    """The tensors of the case, made from the seed alone."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "train":
        (ar, ac), (br, bc), (m, n, k) = _shapes(case)
        lead = (case["batch"],) if case["batch"] else ()
        # row-major torch matrices here: the differentiable form's own layout
        return dict(A=_uniform(gen, *lead, ar, ac), B=_uniform(gen, *lead, br, bc), dC=_uniform(gen, *lead, m, n))
    if kind == "batch":
        shapes = batch_shapes(case["count"], case["lo"], case["hi"], case["shape_seed"])
        place, a, b, c = [], 0, 0, 0
        for ta, tb, m, n, k, _, _ in shapes:
            place.append((a, b, c))
            a, b, c = (x + (y + 63) // 64 * 64 for x, y in ((a, m * k), (b, k * n), (c, m * n)))
        return dict(shapes=shapes, place=place, A=_uniform(gen, a), B=_uniform(gen, b), C=_uniform(gen, c))
    (ar, ac), (br, bc), (m, n, k) = _shapes(case)
    pad = case.get("pad", 0)
    if kind == "strided":
        b = case["batch"]
        return dict(A=_uniform(gen, b, ac, ar), B=_uniform(gen, b, bc, br), C=_uniform(gen, b, n, m))
    data = case.get("data", "unit")
    A = _matrix(gen, ar, ac, ar + pad, data)
    B = _matrix(gen, br, bc, br + pad, data)
    C = _uniform(gen, n, m + pad)
    return dict(A=A, B=B, C=C)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    s["handle"] = cg3m.default_handle()
    if case["kind"] == "batch":
        problems = []
        for (ta, tb, m, n, k, alpha, beta), (a, b, c) in zip(s["shapes"], s["place"]):
            (ar, _), (br, _) = stored_shape(ta, m, k), stored_shape(tb, k, n)
            problems.append((ta, tb, m, n, k, alpha, s["A"][a:], ar, s["B"][b:], br, beta, s["C"][c:], m))
        s["plan"] = s["handle"].batch_plan(problems)
    elif case["kind"] == "host":
        for name in "ABC":
            s[name] = s[name].cpu().pin_memory()
    elif case["kind"] == "train":
        s["A"].requires_grad_(True)
        s["B"].requires_grad_(True)
    return s


# ---- one pass -------------------------------------------------------------------------

def run(s):
    case, h = s["case"], s["handle"]
    kind = case["kind"]
    A, B = s["A"], s["B"]
    if kind == "train":
        out = cgemm3m_autograd(A, B, case["ops"][0], case["ops"][1], case["form"])
        gA, gB = torch.autograd.grad(out, (A, B), s["dC"])
        return out.detach(), gA, gB
    C = s["C"]
    if kind == "batch":
        s["plan"].execute()
        return C
    ta, tb = case["ops"]
    m, n, k = case.get("m", case["n"]), case["n"], case.get("k", case["n"])
    alpha, beta = _scalars(case)
    if kind == "strided":
        st = h.cgemm3m_strided_batched(ta, tb, m, n, k, alpha, A, A.shape[2], A.stride(0), B, B.shape[2],
                                       B.stride(0), beta, C, m, C.stride(0), case["batch"])
        if st != cg3m.SUCCESS:
            raise cg3m.Cg3mError(st, "cgemm3m_strided_batched")
    elif kind == "host":
        h.cgemm3m_host(ta, tb, m, n, k, alpha, A, A.shape[1], B, B.shape[1], beta, C, C.shape[1], form=case["form"])
    elif case.get("call") == "cgemm":
        st = h.cgemm(ta, tb, m, n, k, alpha, A, A.shape[1], B, B.shape[1], beta, C, C.shape[1])
        if st != cg3m.SUCCESS:
            raise cg3m.Cg3mError(st, "cgemm")
    else:
        h.cgemm3m(ta, tb, m, n, k, alpha, A, A.shape[1], B, B.shape[1], beta, C, C.shape[1],
                  form=case.get("form", "fp32"))
    return C


# ---- the work and the exact results ---------------------------------------------------

def _sizes(case):
    """[(m, n, k, reads C)] of every product of a pass."""
    kind = case["kind"]
    if kind == "batch":
        return [(m, n, k, beta != 0) for _, _, m, n, k, _, beta in
                batch_shapes(case["count"], case["lo"], case["hi"], case["shape_seed"])]
    m, n, k = case.get("m", case["n"]), case["n"], case.get("k", case["n"])
    if kind == "train":
        return [(m, n, k, False), (m, k, n, False), (k, n, m, False)] * max(1, case["batch"])
    return [(m, n, k, not case.get("unit", True))] * case.get("batch", 1)


def work(case):
    """Matrices read and written once; three real products of 2 m n k."""
    nbytes = flops = 0
    for m, n, k, reads_c in _sizes(case):
        nbytes += 8 * (m * k + k * n + m * n * (2 if reads_c else 1))
        flops += 6 * m * n * k
    if case["kind"] == "train":
        # forward and backward read A, B and dC between them: each once
        m, n, k = case["m"], case["n"], case["k"]
        nbytes = 8 * max(1, case["batch"]) * 2 * (m * k + k * n + m * n)
    return {"bytes": nbytes, "flops": flops}


def _op(x, op):
    """op() of a stored matrix (..., rows, columns)."""
    if op in "TC":
        x = x.mT
    return x.conj() if op in "CR" else x


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    wide = torch.complex128
    if kind == "train":
        A = s["A"].to(wide).requires_grad_(True)
        B = s["B"].to(wide).requires_grad_(True)
        out = _op(A, case["ops"][0]) @ _op(B, case["ops"][1])
        gA, gB = torch.autograd.grad(out, (A, B), s["dC"].to(wide))
        return out.detach(), gA, gB
    C = s["C"].to(wide)
    if kind == "batch":
        for (ta, tb, m, n, k, alpha, beta), (a, b, c) in zip(s["shapes"], s["place"]):
            (ar, ac), (br, bc) = stored_shape(ta, m, k), stored_shape(tb, k, n)
            X = _op(s["A"][a:a + m * k].view(ac, ar).mT.to(wide), ta)
            Y = _op(s["B"][b:b + k * n].view(bc, br).mT.to(wide), tb)
            Z = C[c:c + m * n].view(n, m)
            Z.copy_(alpha * (X @ Y).mT + beta * Z)
        return C
    (ar, _), (br, _), (m, _, _) = _shapes(case)
    alpha, beta = _scalars(case)
    X = _op(s["A"][..., :ar].mT.to(wide), case["ops"][0])
    Y = _op(s["B"][..., :br].mT.to(wide), case["ops"][1])
    C[..., :m] = alpha * (X @ Y).mT + (beta * C[..., :m] if beta != 0 else 0)
    return C
