"""Workloads of the randomized-Cholesky PCG library, as its users run them.

Every case goes through the public Python face of the C ABI (`rchol_b200`):
a factorization of a matrix that is already on the GPU, one application of
the preconditioner, a PCG solve of one or several right-hand sides, a batch of
independent systems, or a whole call from host triplets to the solution.
Matrices are the families of the repository's configurations and tests: 2-D
5-point, 3-D 7-point and 3-D 27-point grids as SDDM systems with a ground
vertex, in ascending-nnz order with seeded ties, and Chung-Lu power-law graph
Laplacians.
"""
import math
import os
import sys
import time

import numpy as np
import torch

# imported with the repository's root as the working folder
sys.path.insert(0, os.path.join(os.getcwd(), "parallel-randomized-cholesky_b200"))
import rchol_b200 as R  # noqa: E402

DEV = torch.device("cuda", 0)


def listed():
    return [
        # a small 2-D system solved from host arrays: the interactive call, all launches and latency
        dict(name="solve_grid2d_61x47", op="solve", kind="grid2d", nx=61, ny=47, nz=1, wlo=1e-2, whi=1e2,
             excess=0.1, k=1, fp32=False, tol=1e-8, host=True),
        # the default-size 2-D system in the plain FP64 form, device resident
        dict(name="solve_grid2d_256", op="solve", kind="grid2d", nx=256, ny=256, nz=1, wlo=1e-2, whi=1e2,
             excess=0.1, k=1, fp32=False, tol=1e-8, host=False),
        # the headline operator (128^3, conductances over six decades): a factorization in a time-stepping
        # loop, new values on the device
        dict(name="factor_grid3d_128", op="factor", kind="grid3d", nx=128, ny=128, nz=128, wlo=1e-3, whi=1e3,
             excess=1e-2, fp32=True),
        # the same operator inside another solver's iteration: one preconditioner application, FP32 factor
        dict(name="apply_grid3d_128_fp32", op="apply", kind="grid3d", nx=128, ny=128, nz=128, wlo=1e-3, whi=1e3,
             excess=1e-2, k=1, fp32=True),
        # the headline solve: one right-hand side, FP32 factor and FP64 PCG
        dict(name="solve_grid3d_128_fp32", op="solve", kind="grid3d", nx=128, ny=128, nz=128, wlo=1e-2, whi=1e2,
             excess=0.1, k=1, fp32=True, tol=1e-6, host=False),
        # an ordinary ragged 3-D system from host triplets: convert, order, factor and solve in one go
        dict(name="whole_grid3d_61x53x47", op="whole", kind="grid3d", nx=61, ny=53, nz=47, wlo=1e-2, whi=1e2,
             excess=0.1, fp32=True, tol=1e-6),
        # the anisotropic 27-point operator: long gathers in the factorization
        dict(name="factor_grid27_72x70x67", op="factor", kind="grid27", nx=72, ny=70, nz=67, wlo=0.1, whi=10.0,
             excess=1e-4, fp32=True),
        # its block solve: 32 right-hand sides at once (a load-case sweep)
        dict(name="solve_grid27_64_k32", op="solve", kind="grid27", nx=64, ny=64, nz=64, wlo=0.1, whi=10.0,
             excess=1e-4, k=32, fp32=True, tol=1e-8, host=False),
        # eight preconditioner applications at once on an odd grid, FP64
        dict(name="apply_grid3d_75x71x69_k8", op="apply", kind="grid3d", nx=75, ny=71, nz=69, wlo=1e-2, whi=1e2,
             excess=0.1, k=8, fp32=False),
        # a power-law graph (hubs, a dense core eliminated last): factorization with a cooperative tail, as the
        # autotuner sets it for such graphs
        dict(name="factor_powerlaw_100k", op="factor", kind="chunglu", n=100000, degree=20, fp32=False, tail=1500),
        # effective-resistance style solve on the power-law Laplacian
        dict(name="solve_powerlaw_100k", op="solve", kind="chunglu", n=100000, degree=20, k=1, fp32=True, tol=1e-8,
             host=False),
        # many uneven independent systems, eight right-hand sides each, host arrays
        dict(name="batch_12x8", op="batch", systems=12, lo=16, hi=40, k=8, fp32=True, tol=1e-6),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["factor", "apply", "solve", "solve", "whole", "batch"])
    fp32 = rng.random() < 0.6
    if op == "batch":
        lo = rng.randint(12, 32)
        return dict(op=op, systems=rng.randint(3, 16), lo=lo, hi=lo + rng.randint(1, 16), k=rng.choice([1, 2, 8]),
                    fp32=fp32, tol=1e-6)
    kind = rng.choice(["grid2d", "grid3d", "grid3d", "grid27", "chunglu"])
    if kind == "chunglu" and op != "whole":
        c = dict(op=op, kind=kind, n=side(5000, 100000), degree=rng.randint(12, 20), fp32=fp32)
        if rng.random() < 0.5:
            c["tail"] = c["n"] // 80
    else:
        kind = "grid3d" if kind == "chunglu" else kind
        if kind == "grid2d":
            nx, ny, nz = side(24, 512), side(24, 512), 1
        elif kind == "grid3d":
            hi = 64 if op == "whole" else 112
            nx, ny, nz = side(8, hi), side(8, hi), side(8, hi)
        else:
            nx, ny, nz = side(8, 64), side(8, 64), side(8, 64)
        c = dict(op=op, kind=kind, nx=nx, ny=ny, nz=nz, wlo=0.1 if kind == "grid27" else 1e-2,
                 whi=10.0 if kind == "grid27" else 1e2, excess=1e-4 if kind == "grid27" else 0.1, fp32=fp32)
    if op == "apply":
        rows = c["n"] if kind == "chunglu" else c["nx"] * c["ny"] * c["nz"]
        # the allocation-free apply takes n * k <= 2^22
        c["k"] = rng.choice([k for k in (1, 1, 2, 4, 8, 16) if rows * k <= 1 << 21])
    elif op == "solve":
        c.update(k=rng.choice([1, 1, 1, 8]), tol=1e-8, host=rng.random() < 0.3)
    elif op == "whole":
        c["tol"] = 1e-8
    return c


# ---------------------------------------------------------------------------
# matrices
# ---------------------------------------------------------------------------

def grid_triplets(case, seed):
    """The case's grid on the GPU in its own numbering: vertices, edges (a, b, w), weighted degrees and the
    diagonal excess that makes the system an SDDM."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    idx = torch.arange(n, device=DEV).reshape(nz, ny, nx)
    if case["kind"] == "grid27":
        steps = [(dz, dy, dx) for dz in (0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) > (0, 0, 0)]
    else:
        steps = [(0, 0, 1), (0, 1, 0), (1, 0, 0)]
    a, b, w = [], [], []
    deg = torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    for step in steps:
        lo = tuple(slice(max(0, -d), s - max(0, d)) for d, s in zip(step, (nz, ny, nx)))
        hi = tuple(slice(max(0, d), s - max(0, -d)) for d, s in zip(step, (nz, ny, nx)))
        u = torch.rand(idx[lo].shape, dtype=torch.float64, device=DEV, generator=g)
        wt = torch.exp(math.log(case["wlo"]) + u * math.log(case["whi"] / case["wlo"]))
        if case["kind"] == "grid27" and step[0]:
            wt = 100.0 * wt  # anisotropy: conductances along z are 100 times larger
        deg[lo] += wt
        deg[hi] += wt
        a.append(idx[lo].reshape(-1))
        b.append(idx[hi].reshape(-1))
        w.append(wt.reshape(-1))
    a, b, w, deg = torch.cat(a), torch.cat(b), torch.cat(w), deg.reshape(-1)
    u = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    if case["kind"] == "grid27":
        exc = case["excess"] * deg
    else:
        exc = torch.where(torch.rand(n, dtype=torch.float64, device=DEV, generator=g) < 0.05, u * case["excess"] * deg,
                          torch.zeros_like(deg))
    return n, a, b, w, deg, exc


def compress(n, rows, cols, vals):
    """CSC (int32) of device triplets, rows ascending in each column."""
    order = torch.argsort(cols * n + rows)
    cnt = torch.bincount(cols, minlength=n)
    colptr = torch.cat([cnt.new_zeros(1), torch.cumsum(cnt, 0)]).to(torch.int32)
    return colptr, rows[order].to(torch.int32).contiguous(), vals[order].contiguous()


def powerlaw(case, seed):
    """A Chung-Lu graph Laplacian, host CSC: one topology per case, edge weights U[1, 10] of the seed."""
    n, r, c, v, _ = R.generate("chunglu", [case["n"], case["n"] * case["degree"] // 2, 2, case["n"] // 20], seed=3)
    up = r < c
    r, c = r[up], c[up]
    w = np.random.default_rng(seed).uniform(1.0, 10.0, len(r))
    deg = np.bincount(r, weights=w, minlength=n) + np.bincount(c, weights=w, minlength=n)
    i = np.arange(n, dtype=np.int32)
    return n, *R.csc_from_triplets(n, np.concatenate([r, c, i]), np.concatenate([c, r, i]),
                                   np.concatenate([-w, -w, deg]))


def matrix(case, seed):
    """(n, colptr, rowind, val, ground) on the GPU, ordered by ascending nnz with seeded ties; with
    `ground` the last vertex is the appended ground."""
    if case["kind"] == "chunglu":
        n, *csc = powerlaw(case, seed)
        return n, *(torch.from_numpy(t).to(DEV) for t in csc), False
    n, a, b, w, deg, exc = grid_triplets(case, seed)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    cnt = torch.bincount(a, minlength=n) + torch.bincount(b, minlength=n)
    shuffled = torch.randperm(n, device=DEV, generator=g)
    order = shuffled[torch.argsort(cnt[shuffled], stable=True)]
    pos = torch.empty_like(order)
    pos[order] = torch.arange(n, device=DEV)
    a, b = pos[a], pos[b]
    rows, cols, vals = [a, b, pos], [b, a, pos], [-w, -w, deg + exc]
    at = torch.nonzero(exc > 0).reshape(-1)
    last = torch.full_like(at, n)
    end = torch.full((1,), n, device=DEV)
    rows += [pos[at], last, end]
    cols += [last, pos[at], end]
    vals += [-exc[at], -exc[at], exc[at].sum().reshape(1)]
    return n + 1, *compress(n + 1, torch.cat(rows), torch.cat(cols), torch.cat(vals)), True


def rhs(n, k, seed):
    """Zero-mean N(0,1) right-hand sides, column-major on the GPU ((k, n) in torch terms)."""
    g = torch.Generator(device=DEV).manual_seed(seed + 2)
    b = torch.randn((k, n), dtype=torch.float64, device=DEV, generator=g)
    return b - b.mean(dim=1, keepdim=True)


def batch_systems(case, seed):
    """Uneven 2-D and 3-D grid Laplacians without a ground vertex, host CSC."""
    rng = np.random.default_rng(case["systems"])
    out = []
    for s in range(case["systems"]):
        side = int(rng.integers(case["lo"], case["hi"] + 1))
        kind, dims = ("grid2d", [6 * side, 6 * side]) if s % 2 else ("grid3d", [side, side, side])
        n, r, c, v, _ = R.generate(kind, dims, wlo=1e-2, whi=1e2, log_weights=True, seed=seed * 100 + s)
        out.append((n, *R.csc_from_triplets(n, r, c, v)))
    return out


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def options(case):
    kw = dict(seed=1, device=0, precision=R.PREC_FP32_FACTOR if case["fp32"] else R.PREC_FP64)
    if "tail" in case:
        kw.update(tail_vertices=case["tail"])
    if "tol" in case:
        kw.update(tol=case["tol"], stop_rule=R.STOP_RELRES)
    return kw


def prepare(case, seed):
    st = dict(case=case, ctx=R.Context(**options(case)), f=None)
    ctx = st["ctx"]
    if case["op"] == "batch":
        systems = batch_systems(case, seed)
        off = ctx.batch_set(systems)
        B = rhs(int(off[-1]), case["k"], seed).cpu().numpy().T  # column-major, as the library takes it
        for s in range(len(off) - 1):
            B[off[s]:off[s + 1]] -= B[off[s]:off[s + 1]].mean(axis=0)
        st.update(f=ctx.factor(), b=B, off=off, sizes=np.diff(off)[:, None])
        return st
    if case["op"] == "whole":
        n, a, b, w, deg, exc = grid_triplets(case, seed)
        i = torch.arange(n, device=DEV)
        st.update(n=n, rows=torch.cat([a, b, i]).to(torch.int32).cpu().numpy(),
                  cols=torch.cat([b, a, i]).to(torch.int32).cpu().numpy(),
                  vals=torch.cat([-w, -w, deg + exc]).cpu().numpy(), b=rhs(n, 1, seed)[0].cpu().numpy())
        return st
    n, colptr, rowind, val, ground = matrix(case, seed)
    st.update(n=n, colptr=colptr, rowind=rowind, val=val, ground=ground)
    if case["op"] == "factor":
        # the buffers the factor is handed over in, with room for any weights' fill
        cap = int(1.3 * sizes(case)[2])
        st["out"] = [torch.zeros(m, dtype=t, device=DEV)
                     for m, t in ((n + 1, torch.int64), (cap, torch.int32), (cap, torch.float64), (n, torch.float64))]
        torch.cuda.synchronize()
        return st
    set_matrix(st)
    ns = n - 1 if ground else n
    st["f"] = ctx.factor()
    b = rhs(ns, case["k"], seed)
    if case["op"] == "apply":
        st.update(b=b.T.contiguous(), x=torch.empty((ns, case["k"]), dtype=torch.float64, device=DEV))
    elif case["host"]:
        st["b"] = b.T.cpu().numpy() if case["k"] > 1 else b[0].cpu().numpy()
    else:
        st.update(b=b, x=torch.empty_like(b))
    torch.cuda.synchronize()
    return st


def set_matrix(st):
    torch.cuda.current_stream().synchronize()  # the library copies on its own stream
    st["ctx"].set_csc(st["n"], st["colptr"].data_ptr(), st["rowind"].data_ptr(), st["val"].data_ptr(),
                      trim_ground=st["ground"], on_device=True)


class DeviceArray:
    """A device array of the library, for torch.as_tensor."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=2)


def hand_over(f, out):
    """The factor (L strict CSC and D) copied from the library's buffers to the caller's."""
    fi = f.info()
    src = [(fi.lc_ptr, fi.n + 1, "<i8"), (fi.lc_idx, fi.nnz_strict, "<i4"), (fi.lc_val, fi.nnz_strict, "<f8"),
           (fi.diag, fi.n, "<f8")]
    for dst, (ptr, m, typestr) in zip(out, src):
        dst[:m].copy_(torch.as_tensor(DeviceArray(ptr, m, typestr), device=DEV))
    torch.cuda.current_stream().synchronize()  # before the library may reuse its buffers
    return out


def run(st):
    case, ctx = st["case"], st["ctx"]
    if case["op"] == "factor":
        if st["f"] is not None:
            st["f"].free()
        set_matrix(st)
        st["f"] = ctx.factor()
        return hand_over(st["f"], st["out"])
    if case["op"] == "apply":
        stream = torch.cuda.current_stream().cuda_stream
        ctx.precond_apply_noalloc(st["f"], st["b"].data_ptr(), st["x"].data_ptr(), case["k"], case["fp32"], stream)
        return st["x"]
    if case["op"] == "batch":
        X = ctx.batch_solve(st["f"], st["b"])[0].reshape(st["b"].shape)
        # a Laplacian's solution is defined up to a constant: the zero-mean one of every system
        return X - np.repeat(np.add.reduceat(X, st["off"][:-1]) / st["sizes"], st["sizes"][:, 0], axis=0)
    if case["op"] == "whole":
        if st["f"] is not None:
            st["f"].free()
        perm, ground = ctx.set_sddm(st["n"], st["rows"], st["cols"], st["vals"])
        st["f"] = ctx.factor()
        b = np.empty_like(st["b"])
        b[perm] = st["b"]
        return ctx.pcg_solve(st["f"], b)[0][perm]
    if case["host"]:
        x = ctx.pcg_solve(st["f"], st["b"])[0]
        # a Laplacian's solution is defined up to a constant: the zero-mean one
        return x if st["ground"] else x - x.mean(axis=0)
    torch.cuda.current_stream().synchronize()  # the library reads b on its own stream
    ctx.pcg_solve_device(st["f"], case["k"], st["b"].data_ptr(), st["x"].data_ptr(), st["b"].shape[1])
    return st["x"] if st["ground"] else st["x"] - st["x"].mean(dim=1, keepdim=True)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def sizes(case):
    """(unknowns, entries of A, estimated off-diagonal entries of L) of a case."""
    if case["op"] == "batch":
        side = 0.5 * (case["lo"] + case["hi"])
        n = case["systems"] * 0.5 * (side ** 3 + (6 * side) ** 2)
        return n, 6.0 * n, 8.0 * n
    if case["kind"] == "chunglu":
        n = case["n"]
        return n, n * (case["degree"] + 1), 1.15 * n * case["degree"]
    n = case["nx"] * case["ny"] * case["nz"]
    per_row, fill = {"grid2d": (5, 5.0), "grid3d": (7, 9.6), "grid27": (27, 31.5)}[case["kind"]]
    return n, n * per_row, n * fill


def work(case):
    n, a, l_nnz = sizes(case)
    k = case.get("k", 1)
    v = 4 if case["fp32"] else 8
    l_bytes = l_nnz * (4 + v) + n * v
    if case["op"] == "factor":
        # A in, L and D out; per entry of L a division, its share of the prefix sums and a sample
        return dict(bytes=12 * a + 12 * l_nnz + 8 * n, flops=8 * l_nnz)
    if case["op"] == "apply":
        # L read by each sweep, the vectors once
        return dict(bytes=2 * l_bytes + 16 * n * k, flops=4 * l_nnz * k)
    # a solve cannot do without one pass over A, the sweeps over L, the right-hand sides and the solutions
    once = dict(bytes=12 * a + 2 * l_bytes + 16 * n * k, flops=(2 * a + 4 * l_nnz) * k)
    if case["op"] == "whole":
        return dict(bytes=once["bytes"] + 28 * a + 12 * l_nnz, flops=once["flops"] + 8 * l_nnz)
    return once


# ---------------------------------------------------------------------------
# reference solutions in 64 bits
# ---------------------------------------------------------------------------

def cg(matvec, diag, b, seconds):
    """Diagonally preconditioned CG to the rounding of 64 bits; None if it takes longer than `seconds`."""
    began = time.monotonic()
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = (r * z).sum(0)
    b2 = (b * b).sum(0)
    for it in range(200000):
        q = matvec(p)
        alpha = rz / (p * q).sum(0)
        x += alpha * p
        r -= alpha * q
        if it % 50 == 49:
            r = b - matvec(x) if it % 500 == 499 else r
            if bool(((r * r).sum(0) <= 1e-26 * b2).all()):
                return x
            if time.monotonic() - began > seconds:
                return None
        z = r / diag
        new = (r * z).sum(0)
        p = z + (new / rz) * p
        rz = new
    return None


def solve_exact(n, colptr, rowind, val, b, seconds):
    """x with A x = b for the leading n x n part of a symmetric CSC on the GPU; b is (n, k)."""
    cols = torch.repeat_interleave(torch.arange(colptr.numel() - 1, device=DEV), torch.diff(colptr.long()))
    keep = (cols < n) & (rowind < n)
    rows, cols, val = rowind[keep].long(), cols[keep], val[keep]
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), val, (n, n)).coalesce().to_sparse_csr()
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    on = rows == cols
    diag[rows[on]] = val[on]
    return cg(lambda p: A @ p, diag[:, None], b, seconds)


def exact(case, seed):
    """The solution itself, by plain CG in 64 bits.  The factor and its application are random samples keyed by
    the library's own generator, so they have no value apart from it."""
    if case["op"] in ("factor", "apply"):
        return None
    if case["op"] == "batch":
        systems = batch_systems(case, seed)
        off = np.concatenate([[0], np.cumsum([s[0] for s in systems])])
        B = rhs(int(off[-1]), case["k"], seed).T.contiguous()
        out, began = [], time.monotonic()
        for s, (n, cp, ri, v) in enumerate(systems):
            b = B[off[s]:off[s + 1]]
            x = solve_exact(n, *(torch.from_numpy(t).to(DEV) for t in (cp, ri, v)), b - b.mean(0), 15.0)
            if x is None or time.monotonic() - began > 15.0:
                return None
            out.append((x - x.mean(0)).cpu().numpy())
        return np.concatenate(out)
    if case["op"] == "whole":
        n, a, b, w, deg, exc = grid_triplets(case, seed)
        i = torch.arange(n, device=DEV)
        A = compress(n, torch.cat([a, b, i]), torch.cat([b, a, i]), torch.cat([-w, -w, deg + exc]))
        x = solve_exact(n, *A, rhs(n, 1, seed).T.contiguous(), 15.0)
        return None if x is None else x[:, 0].cpu().numpy()
    n, colptr, rowind, val, ground = matrix(case, seed)
    ns = n - 1 if ground else n
    x = solve_exact(ns, colptr, rowind, val, rhs(ns, case["k"], seed).T.contiguous(), 15.0)
    if x is None:
        return None
    if not ground:
        x = x - x.mean(0)
    if case["host"]:
        return x.cpu().numpy() if case["k"] > 1 else x[:, 0].cpu().numpy()
    return x.T.contiguous()
