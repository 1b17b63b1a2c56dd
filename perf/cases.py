"""What the performance of this package is measured on.

A case is one numeric pass on a sparse system whose ordering and symbolic
factorisation are done (once per pattern, as a program keeps them): value
assembly, factorisation, solves, refinement and the adjoint through the
package's public calls.  The matrices are the gallery's (the sizes of the
tests and the benchmark, and odd ones between), with rows and columns scaled
by random factors of the seed so that every state holds other values; the
rows of the unsymmetric forms are scaled on their own, so that the in-block
pivoting meets interchanges.

A case's fields:
  matrix   laplace | convection | diffusion | batch (gallery.laplacian,
           convection_diffusion, diffusion_2d, batched_diffusion)
  nx ny nz the grid; 1 for the dimensions it does not have (batch: nx systems
           with sides of ny .. nz)
  order    nd (nested dissection) | mmd (minimum degree, the default)
  form     fp64 | fp32 | bf16s, with +spd for the symmetric form
  call     refactor  new values on the host into a kept factorisation
                     (sparspaklu_), then ldiv, as the reference is called
           step      new values and right-hand sides on the device:
                     assembly, factorisation and solution refined to 1e-12
           direct    the same without refinement: factor, then solve
           refine    right-hand sides for a kept factor, refined to 1e-12
           refine_t  the same for the transposed system
           solve     one plain solve with a kept factor
           adjoint   factor, solve, transposed solve, dloss/dA
  nrhs     right-hand sides
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparspak.jl_gb300"))

import sparspak as S  # noqa: E402

TOL = 1e-12
KEPT = ("refine", "refine_t", "solve")   # calls on a factor made beforehand


def case(name, matrix, n, order, form, call, nrhs):
    c = {"matrix": matrix, "nx": n[0], "ny": n[1], "nz": n[2], "order": order, "form": form, "call": call, "nrhs": nrhs}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest calls: a 1-D problem of the reference's tests, refactored
        # and solved through host arrays; host work, launches and copies count
        case("tridiag1101_refactor", "laplace", (1101, 1, 1), "mmd", "fp64", "refactor", 1),
        # the 2-D configuration (100 x 100, minimum degree) as the reference is called
        case("grid2d_100_refactor", "laplace", (100, 100, 1), "mmd", "fp64", "refactor", 1),
        # gradient of a loss of the solution: factor, solve, transposed solve, dA
        case("diffusion2d_256_adjoint", "diffusion", (256, 256, 1), "nd", "fp64", "adjoint", 1),
        # a small 3-D system, odd sides, the whole mixed-precision step
        case("convection_23x25x27_step", "convection", (23, 25, 27), "nd", "fp32", "step", 1),
        # the convection-diffusion configuration in the default precision and mixed
        case("convection_48_fp64", "convection", (48, 48, 48), "nd", "fp64", "direct", 1),
        case("convection_48_step", "convection", (48, 48, 48), "nd", "fp32", "step", 1),
        # the benchmark's workload: 64^3, four right-hand sides
        case("laplace_64_step", "laplace", (64, 64, 64), "nd", "fp32", "step", 4),
        # the symmetric form, a box that is no cube
        case("laplace_41x50x63_spd_step", "laplace", (41, 50, 63), "nd", "fp32+spd", "step", 4),
        # BF16 rank updates
        case("laplace_40_bf16s_step", "laplace", (40, 40, 40), "nd", "bf16s", "step", 4),
        # many independent systems at once
        case("batch_512_step", "batch", (512, 20, 120), "nd", "fp32", "step", 1),
        # many right-hand sides, or one a time step, with the factor kept
        case("laplace_64_refine16", "laplace", (64, 64, 64), "nd", "fp32", "refine", 16),
        case("convection_48_solve", "convection", (48, 48, 48), "nd", "fp64", "solve", 1),
    ]


def draw(rng):
    """One more case of the same families, sizes spread over their logarithm."""
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["1d", "2d", "2d", "3d", "3d", "3d", "3d", "batch"])
    if kind == "1d":
        return case(None, "laplace", (side(100, 20000), 1, 1), "mmd", "fp64", rng.choice(["refactor", "direct"]),
                    rng.choice([1, 1, 3]))
    if kind == "batch":
        return case(None, "batch", (side(16, 512), 20, side(30, 120)), "nd", rng.choice(["fp32", "fp32", "fp64"]),
                    rng.choice(["step", "refine"]), 1)
    nrhs = rng.choice([1, 1, 2, 4, 7, 16])
    if kind == "2d":
        n = (side(16, 400), side(16, 400), 1)
        m = rng.choice(["laplace", "diffusion"])
        if m == "diffusion":
            n = (n[0], n[0], 1)
        call = rng.choice(["refactor", "direct", "adjoint", "step", "refine"])
        form = rng.choice(["fp64", "fp32", "fp32+spd"]) if call in ("step", "refine") else "fp64"
        return case(None, m, n, rng.choice(["nd", "mmd"]), form, call, 1 if call == "refactor" else nrhs)
    m = rng.choice(["laplace", "convection"])
    call = rng.choice(["step", "step", "step", "refine", "refine_t", "solve", "direct", "adjoint"])
    form = "fp64" if call in ("direct", "adjoint", "solve") else rng.choice(["fp32", "fp32", "bf16s"])
    if m == "laplace" and call != "adjoint" and rng.random() < 0.25:
        form += "+spd"
    hi = 44 if form.startswith("fp64") else 60
    return case(None, m, (side(10, hi), side(10, hi), side(10, hi)), "nd", form, call, nrhs)


# ---------------------------------------------------------------------------
# Matrices.  Every one is A = R D^-1 M D C: M symmetric positive definite, D
# diagonal (the identity but for convection-diffusion), R and C the seed's
# row and column factors (equal for the symmetric form).
# ---------------------------------------------------------------------------
def _base(c):
    """(the unscaled matrix, the diagonal of D, the sides of the batch's systems)."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    if c["matrix"] == "batch":
        A, sizes = S.gallery.batched_diffusion(nx, ny, nz, seed=0)
        return A, None, sizes
    if c["matrix"] == "diffusion":
        t = np.random.Generator(np.random.PCG64(0))
        return S.gallery.diffusion_2d(nx, t.lognormal(0.0, 1.0, (nx, nx + 1)), 0.1 * t.lognormal(0.0, 1.0, (nx + 1, nx))), None, None
    shape = tuple(k for k in (nx, ny, nz) if k > 1)
    if c["matrix"] == "laplace":
        return S.gallery.laplacian(shape, diag=4.0 if len(shape) == 1 else None, shift=1e-3), None, None
    # first-order upwind convection-diffusion (Peclet 10) on a box: the
    # gallery's coefficients on a grid of its own for each side
    v, h = np.array([1.0, 0.5, 0.25]), 1.0 / (max(shape) + 1)
    up = 1.0 + 10.0 * h * v                      # coupling to the upstream neighbour; 1 downstream
    A = S.gallery.laplacian(shape, diag=6.0 + 10.0 * h * v.sum())
    A.sort_indices()
    coo = A.tocoo()
    i, j = coo.row.astype(np.int64), coo.col.astype(np.int64)
    stride = np.array([ny * nz, nz, 1])
    for ax in range(3):
        coo.data[i - j == stride[ax]] = -up[ax]
    g = np.indices(shape).reshape(3, -1)
    out = coo.tocsc()
    out.sort_indices()
    return out, np.exp(-0.5 * (np.log(up) @ g)), None


def _factors(c, n, seed):
    """R and C of the seed."""
    t = np.random.Generator(np.random.PCG64(seed))
    r = t.lognormal(0.0, 0.3, n)
    return (r, r.copy()) if "+spd" in c["form"] else (r, t.lognormal(0.0, 0.3, n))


def _scaled(A, r, c):
    B = A.copy()
    B.data = A.data * r[A.indices] * np.repeat(c, np.diff(A.indptr))
    return B


def _rhs(c, n, seed):
    """The right-hand sides (and the adjoint's loss gradients), nrhs x n."""
    t = np.random.Generator(np.random.PCG64(seed + 7919))
    return t.uniform(-1.0, 1.0, (c["nrhs"], n)), t.uniform(-1.0, 1.0, (c["nrhs"], n))


def _order(c, sizes):
    if c["order"] == "mmd":
        return None
    return S.nd_grid_batched(sizes) if c["matrix"] == "batch" else S.nd_grid(c["nx"], c["ny"], c["nz"])


def prepare(c, seed):
    A, _, sizes = _base(c)
    n = A.shape[0]
    A = _scaled(A, *_factors(c, n, seed))
    b, g = _rhs(c, n, seed)
    s = {"case": c}
    if c["call"] == "refactor":
        s["lu"] = S.sparspaklu(A, precision=c["form"], orderfunction=_order(c, sizes))
        s["A"] = A
        s["b"] = np.asfortranarray(b.T) if c["nrhs"] > 1 else b[0]
        return s
    lu = S.SparseSolver(A, precision=c["form"])
    S.findorder_(lu, _order(c, sizes))
    S.symbolicfactor_(lu)
    S.inmatrix_(lu)
    if c["call"] in KEPT:
        S.factor_(lu)
    s["lu"] = lu
    s["engine"] = lu.slvr.engine
    s["stream"] = torch.cuda.Stream()
    s["engine"].set_stream(s["stream"].cuda_stream)
    s["values"] = torch.tensor(A.data, device="cuda")
    s["b"] = torch.tensor(b, device="cuda")
    s["x"] = torch.zeros_like(s["b"])
    if c["call"] == "adjoint":
        s["g"] = torch.tensor(g, device="cuda")
        s["lam"] = torch.zeros_like(s["g"])
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    form, call = c["form"], c["call"]
    if call == "refactor":
        return S.ldiv(S.sparspaklu_(s["lu"], s["A"]), s["b"])
    eng, b, x = s["engine"], s["b"], s["x"]
    with torch.cuda.stream(s["stream"]):
        if call not in KEPT:
            eng.load_values(s["values"], form)
        if call == "step":
            eng.factor_refine(b, x, form, tol=TOL)
        elif call == "refine" or call == "refine_t":
            eng.refine(b, x, form, tol=TOL, transpose=call == "refine_t")
        else:
            if call != "solve":
                eng.factor(form)
            x.copy_(b)
            eng.solve(x, form)
        if call == "adjoint":
            lam = s["lam"]
            lam.copy_(s["g"])
            eng.solve(lam, form, transpose=True)
            return {"x": x, "lam": lam, "dA": eng.grad_pattern(lam, x)}
    return x


def work(c):
    """Values, right-hand sides and results once; the factorisation's flops
    (a kept factor instead: its entries read once in each direction)."""
    A, _, sizes = _base(c)
    n, nrhs = A.shape[0], c["nrhs"]
    lu = S.SparseSolver(A)
    S.findorder_(lu, _order(c, sizes))
    S.symbolicfactor_(lu)
    f = lu.slvr
    w = np.diff(f.xsuper)
    k = np.arange(n) - np.repeat(f.xsuper[:-1] - 1, w)
    cnt = (np.repeat(np.diff(f.xlindx), w) - k).astype(np.float64)   # column counts of L
    spd = "+spd" in c["form"]
    entries = float(np.sum(2.0 * cnt - 1.0))
    size = 8 if c["form"].startswith("fp64") else 4
    solve = 2.0 * entries * nrhs
    if c["call"] in KEPT:
        return {"bytes": entries * size + 16.0 * n * nrhs, "flops": solve}
    fact = float(np.sum((cnt - 1) + (1.0 if spd else 2.0) * (cnt - 1) ** 2))
    vec = 16.0 * n * nrhs * (2 if c["call"] == "adjoint" else 1)
    nbytes = 8.0 * A.nnz * (2 if c["call"] == "adjoint" else 1) + vec
    return {"bytes": nbytes, "flops": fact + solve * (2 if c["call"] == "adjoint" else 1)}


# ---------------------------------------------------------------------------
# The same results by conjugate gradients in FP64 (diagonally preconditioned,
# restarted from the true residual), on the symmetric factor M.
# ---------------------------------------------------------------------------
def _cg(M, Minv, B):
    Z = torch.zeros_like(B)
    for _ in range(4):
        R = B - M @ Z
        D = torch.zeros_like(R)
        W = Minv * R
        P, rz = W.clone(), (R * W).sum(0)
        stop = 1e-8 * torch.linalg.vector_norm(R, dim=0)
        for it in range(20000):
            Q = M @ P
            a = rz / (P * Q).sum(0).clamp_min(1e-300)
            D += a * P
            R -= a * Q
            if it % 20 == 19 and bool((torch.linalg.vector_norm(R, dim=0) <= stop).all()):
                break
            W = Minv * R
            new = (R * W).sum(0)
            P = W + (new / rz.clamp_min(1e-300)) * P
            rz = new
        Z += D
    return Z


def exact(c, seed):
    A, d, _ = _base(c)
    n = A.shape[0]
    r, q = _factors(c, n, seed)
    b, g = _rhs(c, n, seed)
    d = np.ones(n) if d is None else d
    M = _scaled(A, d, 1.0 / d)
    M = (M + M.T).tocsr() * 0.5
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    Mt = torch.sparse_csr_tensor(torch.tensor(M.indptr.astype(np.int64)), torch.tensor(M.indices.astype(np.int64)),
                                 torch.tensor(M.data), size=(n, n)).to(dev)
    Minv = torch.tensor(1.0 / M.diagonal()).to(dev)[:, None]

    def solve(rhs, pre, post):   # rows of rhs: post * M^-1 (pre * rhs)
        return _cg(Mt, Minv, torch.tensor((rhs * pre).T.copy()).to(dev)).T.cpu().numpy() * post

    if c["call"] == "refine_t":   # A^T = C D M D^-1 R
        return solve(b, 1.0 / (q * d), d / r)
    x = solve(b, d / r, 1.0 / (d * q))
    if c["call"] == "refactor":
        return np.asfortranarray(x.T) if c["nrhs"] > 1 else x[0]
    if c["call"] != "adjoint":
        return x
    lam = solve(g, 1.0 / (q * d), d / r)
    j = np.repeat(np.arange(n), np.diff(A.indptr))
    return {"x": x, "lam": lam, "dA": -np.einsum("re,re->e", lam[:, A.indices], x[:, j])}
