"""Timed cases of the platform's work, through the calls a program makes.

Every case registers its matrix once (``prepare``), binds the kernel to torch's
current stream and then times one pass (``run``): an ``apply()`` on device
tensors, a SpGEMM ``run()`` with its host result, a batched solve, or one
differentiable operation forward and backward.  Flags keep their defaults
(stopwatches on, automatic kernel choice) unless the case is about the flag.

Matrices are made on the GPU from the seed: grid stencils with random
coefficients (7-point and 27-point in 3D, 5-point triangles in 2D), block
stencils, and irregular matrices with lognormal row lengths and uniform
columns.  ``exact`` is the same operation in float64 with torch's own
operators.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import smaxkernels_b200 as sb
from smaxkernels_b200 import autograd
from smaxkernels_b200.interface import TriangularBatch

DEV = "cuda"
T = {"f64": torch.float64, "f32": torch.float32}
LAP7 = [(0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
BOX27 = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
LOWER5 = [(-1, 0), (0, -1), (0, 0)]
FULL5 = [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)]


def listed():
    return [
        # a solver's inner product on a small grid: launches and latency count
        dict(name="spmv_crs_f64_grid64", op="spmv", fmt="crs", mat="lap7", size=64, type="f64"),
        # a large irregular matrix (graph, network): gathers of x through L2
        dict(name="spmv_crs_f64_irregular", op="spmv", fmt="crs", mat="lognormal", size=1 << 22, type="f64"),
        # the same kind of matrix in SELL-32-1024, single precision
        dict(name="spmv_sell_f32_irregular", op="spmv", fmt="sell", mat="lognormal", size=1 << 20, type="f32"),
        # a finite-element operator with four unknowns a node, as 4x4 blocks
        dict(name="spmv_bcrs4_f64_grid48", op="spmv", fmt="bcrs", mat="box27", size=48, type="f64", bs=4),
        # a block of 16 vectors (block Krylov, multiple loads), row-major
        dict(name="spmm_row_k16_f64_grid128", op="spmm", row_major=True, mat="box27", size=128, type="f64", k=16),
        # a block width that is no power of two, on an irregular matrix
        dict(name="spmm_row_k20_f32_irregular", op="spmm", row_major=True, mat="lognormal", size=600_000, type="f32",
             k=20),
        # a column-major block, the layout of dense linear algebra libraries
        dict(name="spmm_col_k8_f64_grid96", op="spmm", row_major=False, mat="box27", size=96, type="f64", k=8),
        # A*A of a finite-element stencil (coarse-grid operators), C on the host
        dict(name="spgemm_f64_box48", op="spgemm", mat="box27", size=48, type="f64"),
        # one triangular solve in natural order: a preconditioner application, thousands of levels
        dict(name="sptrsv_f64_natural2048", op="sptrsv", order="natural", size=2048, type="f64", k=1),
        # 32 right-hand sides at once
        dict(name="sptrsm_k32_f64_natural1024", op="sptrsm", order="natural", size=1024, type="f64", k=32,
             row_major=True),
        # many independent subdomain solves in one launch
        dict(name="batch48_f64", op="batch", size=600, low=100, count=48, type="f64"),
        # a training step through a solve: x = L(val)^-1 b and the gradients of val and b
        dict(name="grad_sptrsv_f64_512", op="grad", kind="sptrsv", mat="lower5", size=512, type="f64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same families: sizes over the logarithm of their range, odd ones
    among them."""
    op = rng.choice(["spmv", "spmv", "sell", "bcrs", "spmm", "spmm", "spmm", "spgemm", "solve", "solve", "batch",
                     "grad"])
    ty = rng.choice(["f64", "f64", "f32"])
    if op in ("spmv", "sell", "spmm"):
        mat = rng.choice(["lap7", "box27", "lognormal"])
    if op == "spmv":
        size = {"lap7": _log(rng, 24, 190), "box27": _log(rng, 16, 120), "lognormal": _log(rng, 1 << 14, 1 << 22)}[mat]
        return dict(op="spmv", fmt="crs", mat=mat, size=size, type=ty)
    if op == "sell":
        size = {"lap7": _log(rng, 24, 128), "box27": _log(rng, 16, 72), "lognormal": _log(rng, 1 << 14, 1 << 20)}[mat]
        return dict(op="spmv", fmt="sell", mat=mat, size=size, type=ty)
    if op == "bcrs":
        mat, bs = rng.choice(["lap7", "box27"]), rng.choice([2, 3, 4, 4, 8])
        hi = (64 if mat == "lap7" else 48) if bs <= 4 else 28
        return dict(op="spmv", fmt="bcrs", mat=mat, size=_log(rng, 12, hi), type=ty, bs=bs)
    if op == "spmm":
        k = rng.choice([2, 3, 4, 5, 8, 10, 16, 24, 32, 48, 64, rng.randint(2, 64)])
        row_major = rng.random() < 0.7
        # the block of vectors and the products stay within those of 128^3 x 16
        most = (1 << 21) * 16 // k
        size = {"lap7": _log(rng, 20, min(128, round(most ** (1 / 3)))),
                "box27": _log(rng, 16, min(96, round(most ** (1 / 3)))),
                "lognormal": _log(rng, 1 << 13, min(1 << 20, most // 2))}[mat]
        if not row_major and k > 16:
            k = rng.choice([2, 4, 6, 8, 12, 16])
        return dict(op="spmm", row_major=row_major, mat=mat, size=size, type=ty, k=k)
    if op == "spgemm":
        mat = rng.choice(["lap7", "box27", "lognormal"])
        size = {"lap7": _log(rng, 16, 72), "box27": _log(rng, 10, 46), "lognormal": _log(rng, 1 << 11, 36_000)}[mat]
        return dict(op="spgemm", mat=mat, size=size, type=ty)
    if op == "solve":
        # "levels": the level sets of a random order, few and wide
        k = rng.choice([1, 1, 1, 2, 4, 8, 16, 32])
        order = rng.choice(["natural", "natural", "levels"])
        if k == 1:
            return dict(op="sptrsv", order=order, size=_log(rng, 100, 2048 if order == "natural" else 1024), type=ty,
                        k=1)
        return dict(op="sptrsm", order=order, size=_log(rng, 100, 900), type=ty, k=k, row_major=rng.random() < 0.7)
    if op == "batch":
        low = _log(rng, 40, 120)
        return dict(op="batch", size=_log(rng, low + 20, 600), low=low, count=rng.randint(3, 48), type=ty)
    if rng.random() < 0.5:
        return dict(op="grad", kind="sptrsv", mat="lower5", size=_log(rng, 64, 640), type=ty)
    mat = rng.choice(["lap7", "lognormal"])
    size = _log(rng, 20, 96) if mat == "lap7" else _log(rng, 1 << 13, 1 << 19)
    return dict(op="grad", kind="spmv", mat=mat, size=size, type=ty)


# ---------------------------------------------------------------- matrices --
def _rng(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _uniform(n, g, dt, lo=-1.0, hi=1.0):
    return torch.rand(n, generator=g, dtype=dt, device=DEV) * (hi - lo) + lo


def _stencil(dims, offsets):
    """(row_ptr, col, is_diag) of a box stencil in natural order, ascending columns."""
    n = math.prod(dims)
    strides = [math.prod(dims[i + 1:]) for i in range(len(dims))]
    offsets = sorted(offsets, key=lambda o: sum(a * b for a, b in zip(o, strides)))
    idx = torch.arange(n, dtype=torch.int32, device=DEV)
    coord = [(idx // s) % d for s, d in zip(strides, dims)]
    ok = torch.empty(n, len(offsets), dtype=torch.bool, device=DEV)
    for m, o in enumerate(offsets):
        good = torch.ones(n, dtype=torch.bool, device=DEV)
        for c, d, e in zip(coord, dims, o):
            if e:
                good &= (c + e >= 0) & (c + e < d)
        ok[:, m] = good
    shift = torch.tensor([sum(a * b for a, b in zip(o, strides)) for o in offsets], dtype=torch.int32, device=DEV)
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = ok.sum(1).cumsum(0)
    col = (idx[:, None] + shift[None, :])[ok]
    diag = (shift == 0).expand(n, -1)[ok]
    return rp, col.contiguous(), diag


def _lognormal(n, g):
    """Row lengths round(LogNormal) of mean 16 in [1, 4096], uniform columns without repeats,
    sorted (repeated columns are drawn once, so a row may be a little shorter)."""
    z = torch.randn(n, generator=g, dtype=torch.float64, device=DEV)
    lens = torch.exp(z + math.log(16.0) - 0.5).round().clamp(1, min(4096, max(1, n // 4))).long()
    row = torch.repeat_interleave(torch.arange(n, device=DEV), lens)
    key = torch.unique(row * n + torch.randint(0, n, (row.numel(),), generator=g, device=DEV))
    row = key // n
    rp = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    rp[1:] = torch.bincount(row, minlength=n).cumsum(0)
    return rp, (key - row * n).int()


def _matrix(case, seed):
    """(n, row_ptr, col, val) of the case's matrix on the GPU."""
    g, dt, mat, size = _rng(seed), T[case["type"]], case["mat"], case["size"]
    if mat == "lognormal":
        # products and gradients repeat on one pattern with new values; its
        # size is then that of the outputs
        rp, col = _lognormal(size, g if case["op"] in ("spmv", "spmm") else _rng(size, 5))
        return size, rp, col, _uniform(col.numel(), g, dt)
    if mat == "lower5":
        return _lower5((size, size), g, dt)
    rp, col, diag = _stencil((size,) * 3, LAP7 if mat == "lap7" else BOX27)
    if mat == "lap7":
        val = torch.where(diag, _uniform(col.numel(), g, dt, 5.0, 7.0), _uniform(col.numel(), g, dt, -1.25, -0.75))
    else:
        val = torch.where(diag, torch.full((), 27.0, dtype=dt, device=DEV), _uniform(col.numel(), g, dt, 0.5, 1.0))
    return rp.numel() - 1, rp, col, val


def _lower5(dims, g, dt):
    """Lower triangle of a 5-point operator with varying coefficients, diagonal last."""
    rp, col, diag = _stencil(dims, LOWER5)
    val = torch.where(diag, _uniform(col.numel(), g, dt, 3.5, 4.5), _uniform(col.numel(), g, dt, -1.25, -0.75))
    return rp.numel() - 1, rp, col, val


def _rows(rp):
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device=DEV), (rp[1:] - rp[:-1]).long())


def _permuted(size, seed, dt):
    """The 5-point operator under a random symmetric order: the order itself (n, row_ptr, col, val of the
    whole matrix), before any level sets."""
    g = _rng(seed)
    rp, col, diag = _stencil((size, size), FULL5)
    val = torch.where(diag, _uniform(col.numel(), g, dt, 3.5, 4.5), _uniform(col.numel(), g, dt, -1.25, -0.75))
    n = rp.numel() - 1
    new = torch.randperm(n, generator=g, device=DEV)  # new number of each old row
    row, c = new[_rows(rp)], new[col.long()]
    at = torch.argsort(row * n + c)
    out = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    out[1:] = torch.bincount(row, minlength=n).cumsum(0)
    return n, out, c[at].int(), val[at].contiguous()


def _lower_of(n, rp, col, val):
    row = _rows(rp)
    keep = col.long() <= row
    out = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    out[1:] = torch.bincount(row[keep], minlength=n).cumsum(0)
    return out, col[keep].contiguous(), val[keep].contiguous()


def _sides(case):
    lo, hi, m = case["low"], case["size"], case["count"]
    return [lo + round((hi - lo) * i / max(1, m - 1)) for i in range(m)]


def _k(case):
    return case.get("k", 1)


def _block(n, case, seed, salt):
    """A dense operand: n values, or an n x k block (stored k x n when column-major)."""
    k, dt, g = _k(case), T[case["type"]], _rng(seed, salt)
    if case["op"] in ("spmm", "sptrsm"):
        return _uniform((n, k) if case["row_major"] else (k, n), g, dt)
    return _uniform(n, g, dt)


# ----------------------------------------------------------------- program --
def _kernel(kind, ty):
    smax = sb.Interface()
    smax.register_kernel("op", getattr(sb.KernelType, kind), sb.PlatformType.CUDA, sb.IntType.INT32,
                         sb.FloatType.FLOAT64 if ty == "f64" else sb.FloatType.FLOAT32)
    k = smax.kernel("op")
    k.set_stream(torch.cuda.current_stream().cuda_stream)
    return smax, k


def prepare(case, seed):
    op, ty, dt = case["op"], case["type"], T[case["type"]]
    st = {"op": op}
    if op == "batch":
        mats = []
        for i, s in enumerate(_sides(case)):
            _, rp, col, val = _lower5((s, s), _rng(seed, 7 + i), dt)
            mats.append((rp.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()))
        st["solver"] = TriangularBatch(mats, sb.FloatType.FLOAT64 if ty == "f64" else sb.FloatType.FLOAT32)
        n = sum(s * s for s in _sides(case))
        st["rhs"] = _uniform(n, _rng(seed, 1), dt)
        st["out"] = torch.zeros(n, dtype=dt, device=DEV)
        return st
    if op == "grad":
        n, rp, col, val = _matrix(case, seed)
        st["A"] = autograd.SparsePattern(rp.cpu().numpy(), col.cpu().numpy(), kind=case["kind"], dtype=dt)
        st["f"] = autograd.spmv if case["kind"] == "spmv" else autograd.sptrsv
        st["val"] = val.requires_grad_()
        st["x"] = _uniform(n, _rng(seed, 1), dt).requires_grad_()
        st["g"] = _uniform(n, _rng(seed, 2), dt)
        return st
    if op in ("sptrsv", "sptrsm"):
        smax, k = _kernel(op.upper(), ty)
        if case["order"] == "natural":
            n, rp, col, val = _lower5((case["size"],) * 2, _rng(seed), dt)
        else:
            # the library orders the rows by level sets and the solve sweeps them
            n, rp, col, val = (v.cpu().numpy() if torch.is_tensor(v) else v
                               for v in _permuted(case["size"], seed, dt))
            perm, inv = np.empty(n, np.int32), np.empty(n, np.int32)
            smax.utils.generate_perm(n, rp, col, perm, inv, "RS")
            prp, pcol, pval = np.empty_like(rp), np.empty_like(col), np.empty_like(val)
            smax.utils.apply_mat_perm(n, rp, col, val, prp, pcol, pval, perm, inv)
            rp, col, val = _lower_of(n, *(torch.from_numpy(a).to(DEV) for a in (prp, pcol, pval)))
            k.set_mat_perm(True)
            st["perm"] = torch.from_numpy(perm).to(DEV)
        k.set_mat_lower_triang(True)
        b = _block(n, case, seed, 1)
        if op == "sptrsm":
            k.set_vec_row_major(case["row_major"])
        x = torch.zeros_like(b)
        k.register_A(n, n, col.numel(), col, rp, val)
        dims = (n, _k(case)) if op == "sptrsm" else (n,)
        k.register_B(*dims, x)
        k.register_C(*dims, b)
        st["keep"] = (smax, rp, col, val, b)
        st["out"] = x
        st["k"] = k
        k.initialize()
        return st
    if op == "spgemm":
        n, rp, col, val = _matrix(case, seed)
        smax, k = _kernel("SPGEMM", ty)
        k.register_A(n, n, col.numel(), col, rp, val)
        k.register_B(n, n, col.numel(), col, rp, val)
        k.register_C()
        st["keep"] = (smax, rp, col, val)
        st["k"] = k
        k.initialize()
        return st
    smax, k = _kernel(op.upper(), ty)
    if case.get("fmt") == "bcrs":
        bs, g = case["bs"], _rng(seed, 3)
        rp, col, diag = _stencil((case["size"],) * 3, LAP7 if case["mat"] == "lap7" else BOX27)
        val = _uniform((col.numel(), bs, bs), g, dt)
        nb, n = rp.numel() - 1, (rp.numel() - 1) * bs
        host = (col.cpu().numpy(), rp.cpu().numpy(), val.reshape(-1).cpu().numpy())
        k.set_mat_bcrs(True)
        k.register_A(nb, nb, col.numel(), bs, bs, bs, bs, *host)
        st["keep"] = (smax, host)
        rows = n
    elif case.get("fmt") == "sell":
        n, rp, col, val = _matrix(case, seed)
        d = smax.utils.convert_crs_to_scs(n, n, col.numel(), col.cpu().numpy(), rp.cpu().numpy(), val.cpu().numpy(),
                                          32, 1024)
        k.set_mat_scs(True)
        k.register_A(d["C"], d["sigma"], d["n_rows"], d["n_rows_padded"], d["n_cols"], d["n_chunks"],
                     d["n_elements"], d["nnz"], d["chunk_ptr"], d["chunk_lengths"], d["col"], d["val"], d["perm"])
        st["keep"] = (smax, d)
        rows = d["n_rows_padded"]
    else:
        n, rp, col, val = _matrix(case, seed)
        k.register_A(n, n, col.numel(), col, rp, val)
        st["keep"] = (smax, rp, col, val)
        rows = n
    x = _block(n, case, seed, 1)
    if op == "spmm":
        k.set_vec_row_major(case["row_major"])
        y = torch.zeros_like(x)
        k.register_B(n, _k(case), x)
        k.register_C(n, _k(case), y)
    else:
        # SELL-C-sigma works on vectors of the padded row count
        x = torch.nn.functional.pad(x, (0, rows - n)) if rows > n else x
        y = torch.zeros(rows, dtype=dt, device=DEV)
        k.register_B(rows, x)
        k.register_C(rows, y)
    st["x"], st["out"], st["k"] = x, y, k
    k.initialize()
    return st


def run(st):
    op = st["op"]
    if op == "batch":
        st["solver"].solve(st["rhs"], st["out"], stream=torch.cuda.current_stream().cuda_stream)
        return st["out"]
    if op == "grad":
        y = st["f"](st["A"], st["val"], st["x"])
        dval, dx = torch.autograd.grad(y, (st["val"], st["x"]), st["g"])
        return {"y": y.detach(), "dval": dval, "dx": dx}
    if op == "spgemm":
        st["k"].run()
        n_rows, n_cols, nnz, row_ptr, col, val = st["k"].result()
        return {"row_ptr": row_ptr, "col": col, "val": val}
    st["k"].apply()
    return st["out"]


# -------------------------------------------------------------------- work --
def _stencil_nnz(size, offsets):
    return sum(math.prod(max(0, size - abs(e)) for e in o) for o in offsets)


def _nnz(case):
    s = case["size"]
    m = case.get("mat")
    if m == "lognormal":
        return s, 16 * s
    if m in ("lap7", "box27"):
        return s ** 3, _stencil_nnz(s, LAP7 if m == "lap7" else BOX27)
    return s * s, _stencil_nnz(s, LOWER5)


def work(case):
    op, v, k = case["op"], 8 if case["type"] == "f64" else 4, _k(case)
    if op == "batch":
        n, z = sum(s * s for s in _sides(case)), sum(_stencil_nnz(s, LOWER5) for s in _sides(case))
        return {"bytes": (v + 4) * z + 4 * n + 2 * v * n, "flops": 2 * z}
    n, z = _nnz(case)
    a = (v + 4) * z + 4 * (n + 1)
    if op == "spgemm":
        if case["mat"] == "lap7":
            zc = _stencil_nnz(case["size"], [(i, j, l) for i in range(-2, 3) for j in range(-2, 3)
                                             for l in range(-2, 3) if abs(i) + abs(j) + abs(l) <= 2])
            prod = 49 * n
        elif case["mat"] == "box27":
            zc, prod = _stencil_nnz(case["size"], [(i, j, l) for i in range(-2, 3) for j in range(-2, 3)
                                                   for l in range(-2, 3)]), 729 * n
        else:
            prod = 256 * n
            zc = min(prod, n * n)
        return {"bytes": 2 * a + (v + 4) * zc + 4 * (n + 1), "flops": 2 * prod}
    if op == "grad":
        # values, pattern and vectors in; result and gradients out
        return {"bytes": 2 * a + v * z + 5 * v * n, "flops": 5 * z}
    if case.get("fmt") == "bcrs":
        b = case["bs"]
        return {"bytes": (v * b * b + 4) * z + 4 * (n + 1) + 2 * v * n * b, "flops": 2 * z * b * b}
    return {"bytes": a + 2 * v * n * k, "flops": 2 * z * k}


# ------------------------------------------------------------------- exact --
def _csr(n, rp, col, val):
    return torch.sparse_csr_tensor(rp.long(), col.long(), val.double(), size=(n, n))


def _mul(A, x):
    return A @ x if x.dim() == 2 else (A @ x[:, None])[:, 0]


def _solve(n, rp, col, val, b):
    """Forward substitution as the iteration x <- D^-1 (b - N x), which is exact once it has
    passed every level (N is nilpotent)."""
    row, c, v = _rows(rp), col.long(), val.double()
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    d[row[c == row]] = v[c == row]
    off = c != row
    out = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    out[1:] = torch.bincount(row[off], minlength=n).cumsum(0)
    N = torch.sparse_csr_tensor(out, c[off], v[off], size=(n, n))
    inv = 1.0 / (d if b.dim() == 1 else d[:, None])
    x = b * inv
    for _ in range(n):
        for _ in range(32):
            last, x = x, (b - _mul(N, x)) * inv
        if torch.equal(last, x):
            return x
    return x


def _transposed(n, rp, col, val):
    row, c = _rows(rp), col.long()
    at = torch.argsort(c * n + row)
    out = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    out[1:] = torch.bincount(c, minlength=n).cumsum(0)
    return out, row[at], val[at]


def exact(case, seed):
    op, dt = case["op"], T[case["type"]]
    if op == "batch":
        rps, cols, vals, o, z = [torch.zeros(1, dtype=torch.int64, device=DEV)], [], [], 0, 0
        for i, s in enumerate(_sides(case)):
            n, rp, col, val = _lower5((s, s), _rng(seed, 7 + i), dt)
            rps.append(rp[1:].long() + z)
            cols.append(col.long() + o)
            vals.append(val)
            o, z = o + n, z + col.numel()
        return _solve(o, torch.cat(rps), torch.cat(cols), torch.cat(vals), _uniform(o, _rng(seed, 1), dt).double())
    if op == "grad":
        n, rp, col, val = _matrix(case, seed)
        x, g = _uniform(n, _rng(seed, 1), dt).double(), _uniform(n, _rng(seed, 2), dt).double()
        row, c = _rows(rp), col.long()
        if case["kind"] == "spmv":
            return {"y": _mul(_csr(n, rp, col, val), x), "dval": g[row] * x[c],
                    "dx": _mul(_csr(n, *_transposed(n, rp, col, val)), g)}
        y = _solve(n, rp, col, val, x)
        lam = _solve(n, *_transposed(n, rp, col, val), g)
        return {"y": y, "dval": -lam[row] * y[c], "dx": lam}
    if op in ("sptrsv", "sptrsm"):
        rows_first = op == "sptrsv" or case["row_major"]
        if case["order"] != "natural":
            return None  # the order of the rows is the library's
        n, rp, col, val = _lower5((case["size"],) * 2, _rng(seed), dt)
        b = _block(n, case, seed, 1).double()
        x = _solve(n, rp, col, val, b if rows_first else b.t().contiguous())
        return x if rows_first else x.t().contiguous()
    if op == "spgemm":
        n, rp, col, val = _matrix(case, seed)
        rp, c, v = rp.long(), col.long(), val.double()
        row = _rows(rp)
        cnt = rp[c + 1] - rp[c]
        j = torch.repeat_interleave(torch.arange(c.numel(), device=DEV), cnt)
        first = torch.cumsum(cnt, 0) - cnt
        e = torch.arange(j.numel(), device=DEV) - first[j] + rp[c[j]]
        key, prod = row[j] * n + c[e], v[j] * v[e]
        del e, j
        key, at = torch.sort(key, stable=True)
        new = torch.ones(key.numel(), dtype=torch.bool, device=DEV)
        new[1:] = key[1:] != key[:-1]
        group = torch.cumsum(new, 0) - 1
        out = torch.zeros(int(group[-1]) + 1, dtype=torch.float64, device=DEV).index_add_(0, group, prod[at])
        # C's columns stand in the order in which the products first reach them
        return {"row_ptr": None, "col": None, "val": out[torch.argsort(at[new])]}
    if case.get("fmt") == "bcrs":
        bs = case["bs"]
        rp, col, _ = _stencil((case["size"],) * 3, LAP7 if case["mat"] == "lap7" else BOX27)
        val = _uniform((col.numel(), bs, bs), _rng(seed, 3), dt).double()
        n = (rp.numel() - 1) * bs
        x = _uniform(n, _rng(seed, 1), dt).double().view(-1, bs)
        y = torch.zeros_like(x).index_add_(0, _rows(rp), torch.einsum("eij,ej->ei", val, x[col.long()]))
        return y.reshape(-1)
    n, rp, col, val = _matrix(case, seed)
    x = _block(n, case, seed, 1).double()
    A = _csr(n, rp, col, val)
    if op == "spmm":
        return _mul(A, x) if case["row_major"] else _mul(A, x.t().contiguous()).t().contiguous()
    y = _mul(A, x)
    # SELL-C-sigma leaves y in its own row order, which is the library's
    return None if case.get("fmt") == "sell" else y
