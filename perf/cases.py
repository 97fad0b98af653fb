"""The work this framework is measured on, through its public Python entry points.

A case names one entry point and the sizes it is called with. The operators are the ones the
package's problems use (5/7-point Laplacians with a random potential as CSR or matrix-free, the
complex 7-point tight-binding stencil with Peierls phases, the 27-point stencil). Their random
potentials are drawn per axis, V(x, y, z) = f(x) + g(y) + h(z), so that the eigenpairs are tensor
products of small dense eigenproblems: the Ritz blocks that the kernel-level calls meet inside a solve
can then be laid out exactly, and every result has a value in 64 bits to be compared with.

What the kinds stand for:
  eigh     the small dense eigenproblem on its own (nearly diagonal matrices, as late Ritz steps have)
  cholqr   orthonormalising a start block
  filter   the Chebyshev filter on a block, FP64 (the default precision)
  corr     the filter in correction form on Ritz pairs, the step mixed-precision solves spend most time in
  batch    the same for several small solves at once, as the request server runs them
  rr       a Rayleigh-Ritz step on an orthonormal block
  solve    a whole solve
"""
import ctypes
import math
import random

import numpy as np
import torch

from rayleighchebyshevgpgpu_b200 import runtime as R

F64, C128 = torch.float64, torch.complex128


def listed():
    return [
        # the smallest call: the dense step of a 2-D solve for 16 pairs (block 16 + 8)
        {"name": "eigh_24", "kind": "eigh", "s": 24, "complex": False, "off": 1e-2},
        # the dense step of the widest complex solve (block 128 + 64)
        {"name": "eigh_c192", "kind": "eigh", "s": 192, "complex": True, "off": 1e-3},
        # a start block of a solve for 64 pairs, an odd number of rows
        {"name": "cholqr_96", "kind": "cholqr", "n": 1000003, "s": 96, "complex": False},
        # the filter of a default (FP64) solve on the benchmark's operator
        {"name": "filter_csr_128", "kind": "filter", "form": "csr", "points": 7, "nx": 128, "ny": 128, "nz": 128,
         "complex": False, "s": 96, "degree": 13, "precision": "fp64"},
        # the filter of the benchmark's mixed solve (CSR, 64 + 32 columns)
        {"name": "corr_csr_128", "kind": "corr", "form": "csr", "points": 7, "nx": 128, "ny": 128, "nz": 128,
         "complex": False, "s": 96, "degree": 13},
        # the 27-point stencil with 32 + 16 columns
        {"name": "corr_27pt_192", "kind": "corr", "form": "stencil", "points": 27, "nx": 192, "ny": 192, "nz": 192,
         "complex": False, "s": 48, "degree": 9},
        # the complex tight-binding stencil with 128 + 64 columns
        {"name": "corr_c_884736", "kind": "corr", "form": "stencil", "points": 7, "nx": 24, "ny": 24, "nz": 1536,
         "complex": True, "s": 192, "degree": 17},
        # eight requests of a server, each a small 2-D or 3-D Laplacian of its own
        {"name": "batch_8", "kind": "batch", "jobs": 8, "nmin": 10000, "nmax": 200000, "mix": 5},
        # Ritz steps of the benchmark's solve and of the widest complex one
        {"name": "rr_csr_128", "kind": "rr", "form": "csr", "points": 7, "nx": 128, "ny": 128, "nz": 128,
         "complex": False, "s": 96, "count": 64},
        {"name": "rr_c_442368", "kind": "rr", "form": "stencil", "points": 7, "nx": 24, "ny": 24, "nz": 768,
         "complex": True, "s": 192, "count": 128},
        # whole solves: the smallest configuration (host arrays in and out), and an odd-sized mixed one on the device
        {"name": "solve_64x64", "kind": "solve", "form": "csr", "points": 5, "nx": 64, "ny": 64, "nz": 1,
         "complex": False, "k": 16, "tol": 1e-10, "precision": "fp64", "host": True},
        {"name": "solve_61x53x67", "kind": "solve", "form": "csr", "points": 7, "nx": 61, "ny": 53, "nz": 67,
         "complex": False, "k": 24, "tol": 1e-10, "precision": "mixed", "host": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_grid(rng, complex_, points, nmin, nmax):
    """Grid sides (odd and ragged ones among them) with about log-uniform n."""
    n = _log_int(rng, nmin, nmax)
    if points == 5:
        nx = max(8, int(math.sqrt(n) * rng.uniform(0.6, 1.6)))
        return nx, max(8, n // nx), 1
    if complex_:  # the x-y plane is solved densely when the inputs are laid out: at most 24 x 24
        nx, ny = rng.randint(6, 24), rng.randint(6, 24)
        return nx, ny, max(6, n // (nx * ny))
    side = n ** (1.0 / 3.0)
    nx, ny = max(6, int(side * rng.uniform(0.7, 1.4))), max(6, int(side * rng.uniform(0.7, 1.4)))
    return nx, ny, max(6, n // (nx * ny))


def draw(rng):
    """One more case of the same ranges: any kind, sizes log-uniform, no dearer than the dearest listed one."""
    most = max(max(work(c)["bytes"], work(c)["flops"] / 50) for c in listed())
    while True:
        kind = rng.choice(["eigh", "cholqr", "filter", "filter", "corr", "corr", "batch", "rr", "rr", "solve"])
        complex_ = rng.random() < 0.3
        if kind == "eigh":
            return {"kind": kind, "s": _log_int(rng, 8, 192), "complex": complex_, "off": 10.0 ** rng.randint(-6, 0)}
        if kind == "cholqr":
            c = {"kind": kind, "n": _log_int(rng, 3000, 2000000), "s": _log_int(rng, 8, 192), "complex": complex_}
        elif kind == "batch":
            c = {"kind": kind, "jobs": rng.randint(2, 16), "nmin": 5000, "nmax": _log_int(rng, 20000, 200000),
                 "mix": rng.randrange(1000)}
        elif kind == "solve":
            points = rng.choice([5, 7])
            nx, ny, nz = _draw_grid(rng, complex_, points, 1500, 4000 if points == 5 else 40000)
            if complex_ and points == 5:
                nx, ny = rng.randint(18, 24), rng.randint(18, 24)
            k = rng.choice([4, 8, 12, 16, 24])
            c = {"kind": kind, "form": rng.choice(["csr", "stencil"]), "points": points, "nx": nx, "ny": ny, "nz": nz,
                 "complex": complex_, "k": k, "tol": 1e-10,
                 "precision": rng.choice(["fp64", "mixed"]), "host": rng.random() < 0.5}
            if nx * ny * nz < 12 * k:
                continue
        else:
            points = 7 if complex_ else rng.choice([5, 7, 7] if kind == "rr" else [5, 7, 7, 27])
            nx, ny, nz = _draw_grid(rng, complex_, points, 10000, 3000000)
            form = "stencil" if points == 27 else rng.choice(["csr", "csr", "stencil"])
            c = {"kind": kind, "form": form, "points": points, "nx": nx, "ny": ny, "nz": nz, "complex": complex_,
                 "s": _log_int(rng, 8, 192)}
            if kind == "rr":
                c["count"] = max(1, 2 * c["s"] // 3)
            else:
                c["degree"] = rng.randint(4, 20)
                if kind == "filter":
                    c["precision"] = "fp64"
        w = work(c)
        if max(w["bytes"], w["flops"] / 50) <= most:
            return c


# ---- operators and their exact eigenpairs -------------------------------------------------------
FLUX = 1.0 / 17.0


def _dims(c):
    return c["nx"], c["ny"], c["nz"]


class Grid:
    """A stencil operator's data on the GPU: axis potentials, diagonal, off-diagonal weight."""

    def __init__(self, c, gen):
        nx, ny, nz = _dims(c)
        self.c, self.n, self.points, self.complex_ = c, nx * ny * nz, c["points"], c["complex"]
        draw = lambda m: torch.rand(m, generator=gen, device="cuda", dtype=F64)  # noqa: E731
        if self.points == 27:
            # weak disorder on a constant diagonal: the eigenvectors are known to the size of the disorder
            self.off = -1.0 / 26.0
            self.diag = 1.0 + 3e-9 * draw(self.n).view(nz, ny, nx)
            self.axes = None
        else:
            amp, base = (1.0, 0.0) if self.complex_ else (4.0, 6.0 if self.points == 7 else 4.0)
            self.off = -1.0
            self.axes = [amp / 3.0 * draw(m) for m in (nx, ny, nz)]
            if self.points == 5:
                self.axes[2].zero_()
            f, g, h = self.axes
            self.base = base
            self.diag = base + f[None, None, :] + g[None, :, None] + h[:, None, None]
        self.phase = None
        if self.complex_:
            t = 2.0 * math.pi * FLUX * torch.arange(nx, device="cuda", dtype=F64)
            self.phase = torch.complex(torch.cos(t), torch.sin(t))

    def lambda_bounds(self):
        """Gershgorin interval."""
        m = {5: 4, 7: 6, 27: 26}[self.points] * abs(self.off)
        return float(self.diag.min()) - m, float(self.diag.max()) + m

    def apply(self, X):
        """A X in plain torch for X of shape (columns, n)."""
        nx, ny, nz = _dims(self.c)
        x = X.view(-1, nz, ny, nx)
        if self.points == 27:
            b = x.clone()
            for d in (3, 2, 1):
                m, t = b.shape[d], b.clone()
                t.narrow(d, 1, m - 1).add_(b.narrow(d, 0, m - 1))
                t.narrow(d, 0, m - 1).add_(b.narrow(d, 1, m - 1))
                b = t
            return ((self.diag - self.off) * x + self.off * b).reshape(X.shape)
        y = self.diag * x
        for d in (3, 1) if self.complex_ else (3, 2, 1):
            m = x.shape[d]
            y.narrow(d, 1, m - 1).add_(x.narrow(d, 0, m - 1), alpha=self.off)
            y.narrow(d, 0, m - 1).add_(x.narrow(d, 1, m - 1), alpha=self.off)
        if self.complex_:
            y[:, :, 1:] += self.off * self.phase * x[:, :, :-1]
            y[:, :, :-1] += self.off * self.phase.conj() * x[:, :, 1:]
        return y.reshape(X.shape)

    def eigenpairs(self, s):
        """The lowest s eigenpairs (ascending) as values and an (s, n) block. 27 points: of the constant diagonal."""
        nx, ny, nz = _dims(self.c)
        chain = lambda v, w: torch.linalg.eigh(  # noqa: E731
            torch.diag(v) + w * (torch.diag(torch.ones(len(v) - 1, device="cuda", dtype=F64), 1)
                                 + torch.diag(torch.ones(len(v) - 1, device="cuda", dtype=F64), -1)))
        if self.points == 27:
            e, u = zip(*(chain(torch.ones(m, device="cuda", dtype=F64), 1.0) for m in (nx, ny, nz)))
            prod = e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
            lam = (1.0 - self.off) + self.off * prod
        elif self.complex_:
            m = nx * ny
            H = torch.zeros(ny, nx, ny, nx, device="cuda", dtype=C128)
            ix, iy = torch.arange(nx, device="cuda"), torch.arange(ny, device="cuda")
            f, g, h = self.axes
            H[iy[:, None], ix[None], iy[:, None], ix[None]] = (self.base + f[None] + g[:, None]).to(C128)
            H[iy[:, None], ix[None, 1:], iy[:, None], ix[None, :-1]] = self.off
            H[iy[:, None], ix[None, :-1], iy[:, None], ix[None, 1:]] = self.off
            H[iy[1:, None], ix[None], iy[:-1, None], ix[None]] = self.off * self.phase
            H[iy[:-1, None], ix[None], iy[1:, None], ix[None]] = self.off * self.phase.conj()
            exy, uxy = torch.linalg.eigh(H.view(m, m))
            ez, uz = chain(h, self.off) if nz > 1 else (h, torch.ones(1, 1, device="cuda", dtype=F64))
            lam, at = torch.sort((ez[:, None] + exy[None]).reshape(-1))
            lam, at = lam[:s], at[:s]
            return lam, torch.einsum("zs,ms->szm", uz[:, at // m].to(C128), uxy[:, at % m]).reshape(s, -1).contiguous()
        else:
            e, u = zip(*(chain(a, self.off) if len(a) > 1 else (a, torch.ones(1, 1, device="cuda", dtype=F64))
                         for a in self.axes))
            lam = self.base + e[2][:, None, None] + e[1][None, :, None] + e[0][None, None, :]
        lam, at = torch.sort(lam.reshape(-1), stable=True)
        lam, at = lam[:s], at[:s]
        x, y, z = at % nx, (at // nx) % ny, at // (nx * ny)
        return lam, torch.einsum("zs,ys,xs->szyx", u[2][:, z], u[1][:, y], u[0][:, x]).reshape(s, -1).contiguous()

    def csr(self):
        """CSR arrays (pinned int32 row pointers and columns, values), columns ascending."""
        nx, ny, nz = _dims(self.c)
        i = torch.arange(self.n, device="cuda")
        ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
        full = lambda v: torch.full((self.n,), v, device="cuda", dtype=F64)  # noqa: E731
        bonds = [(-nx * ny, iz > 0, full(self.off)), (-nx, iy > 0, full(self.off)), (-1, ix > 0, full(self.off)),
                 (0, ix >= 0, self.diag.reshape(-1)), (1, ix < nx - 1, full(self.off)), (nx, iy < ny - 1, full(self.off)),
                 (nx * ny, iz < nz - 1, full(self.off))]
        if self.complex_:
            bonds = [(o, m, v.to(C128) * ({-nx: self.phase, nx: self.phase.conj()}[o][ix] if abs(o) == nx else 1.0))
                     for o, m, v in bonds]
        ok = torch.stack([m for _, m, _ in bonds], 1)
        ptr = torch.zeros(self.n + 1, device="cuda", dtype=torch.int64)
        ptr[1:] = torch.cumsum(ok.sum(1), 0)
        col = torch.stack([i + o for o, _, _ in bonds], 1)[ok].to(torch.int32)
        val = torch.stack([v for _, _, v in bonds], 1)[ok]
        return ptr.to(torch.int32).cpu(), col.cpu(), val.cpu()

    def operator(self, ctx):
        if self.c["form"] == "csr":
            p, i, v = self.csr()
            return R.CsrOperator.from_host_pointers(ctx, self.n, i.numel(), p.data_ptr(), i.data_ptr(), v.data_ptr(),
                                                    self.complex_)
        return R.StencilOperator(ctx, self.points, _dims(self.c), self.diag.reshape(-1).cpu().numpy(), self.off,
                                 FLUX if self.complex_ else 0.0, self.complex_)


def _gammas(grid, lam0):
    """The filter's interval: damped from the lowest eigenvalue up to just above the spectrum."""
    shift = -lam0
    rho = 1.02 * (grid.lambda_bounds()[1] + shift)
    return -2.0 / (rho - 2.0 * shift), 2.0 - 4.0 * shift / rho


def _filtered(grid, X, degree, g1, g2):
    """The filter written out in plain torch: x_k = (a A + b) x_{k-1} - x_{k-2}, x_m / (m + 1); in place, few columns
    at a time."""
    a, b = g1 * g2, g2
    step = max(1, int(2e8 // X.shape[1]))
    for j in range(0, X.shape[0], step):
        old = X[j:j + step].clone()
        new = a * grid.apply(old) + b * old
        for _ in range(1, degree):
            old, new = new, (a * grid.apply(new)).add_(new, alpha=b).sub_(old)
        X[j:j + step] = new / (degree + 1)
    return X


def _orthonormal(V):
    """Columns (rows of V) orthonormalised by two Cholesky passes: the factor of a QR with a positive diagonal."""
    for _ in range(2):
        L = torch.linalg.cholesky(V.conj() @ V.mT)  # G^T = conj(V) V^T in (columns, n) layout
        V = torch.linalg.solve_triangular(L.conj(), V, upper=False)
    return V.contiguous()


# ---- state --------------------------------------------------------------------------------------
_kept = {}


def _context():
    """The program's one context, its work on the program's own stream."""
    if not _kept:
        _kept["stream"] = torch.cuda.Stream()
        _kept["ctx"] = R.Context(0)
        _kept["ctx"].set_stream(_kept["stream"].cuda_stream)
    return _kept["ctx"], _kept["stream"]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _randn(shape, gen, complex_):
    if complex_:
        return torch.complex(torch.randn(shape, generator=gen, device="cuda", dtype=F64),
                             torch.randn(shape, generator=gen, device="cuda", dtype=F64))
    return torch.randn(shape, generator=gen, device="cuda", dtype=F64)


def _jobs(c):
    """The jobs of a batch: sizes as the request server's stream has them."""
    if c["kind"] != "batch":
        return [c]
    rng, out = random.Random(c["mix"]), []
    for _ in range(c["jobs"]):
        points = rng.choice([5, 7])
        nx, ny, nz = _draw_grid(rng, False, points, c["nmin"], c["nmax"])
        out.append({"kind": "corr", "form": rng.choice(["csr", "stencil"]), "points": points, "nx": nx, "ny": ny,
                    "nz": nz, "complex": False, "s": rng.choice([16, 24, 48, 96]), "degree": rng.randint(6, 20)})
    return out


def _inputs(c, seed, j=0):
    """A case's inputs from the seed alone: (grid, block, values)."""
    gen = _gen(seed + 7919 * j)
    kind = c["kind"]
    if kind == "eigh":
        X = _randn((c["s"], c["s"]), gen, c["complex"])
        d = torch.sort(torch.randn(c["s"], generator=gen, device="cuda", dtype=F64)).values
        return None, (torch.diag(d).to(X.dtype) + c["off"] * (X + X.mH)), None
    if kind == "cholqr":
        return None, _randn((c["s"], c["n"]), gen, c["complex"]), None
    grid = Grid(c, gen)
    if kind == "solve":
        k, buf = c["k"], max(8, -(-c["k"] // 2 // 8) * 8)
        return grid, _randn((k + buf, grid.n), gen, c["complex"]), None
    if kind == "filter":
        lam, _ = grid.eigenpairs(1)
        return grid, _randn((c["s"], grid.n), gen, c["complex"]), lam
    # Ritz vectors with a residual: of a late iteration for the correction filter, of an earlier one for a Ritz step
    lam, V = grid.eigenpairs(c["s"])
    eps = 3e-9 if kind == "corr" else 1e-4
    V = V.add_(_randn(V.shape, gen, c["complex"]), alpha=eps / math.sqrt(grid.n))
    if kind == "rr":
        V = _orthonormal(V)
    return grid, V, lam


def prepare(c, seed):
    ctx, stream = _context()
    with torch.cuda.stream(stream):
        st = {"case": c, "ctx": ctx, "stream": stream, "jobs": []}
        for j, job in enumerate(_jobs(c)):
            grid, X, lam = _inputs(job, seed, j)
            p = {"case": job, "X": X}
            if grid is not None:
                p["op"] = grid.operator(ctx)
            if lam is not None:
                p["lam"] = lam.cpu().numpy()
                p["g1"], p["g2"] = _gammas(grid, float(lam[0]))
            if job["kind"] in ("corr", "rr", "cholqr", "filter"):
                p["V"] = torch.empty_like(X)  # the block the calls work on in place
            if job["kind"] == "rr":
                p["W"] = torch.empty_like(X)
            if job["kind"] == "eigh":
                p["X"] = X.cpu().numpy()
            if job["kind"] == "solve":
                k = job["k"]
                if job["host"]:
                    p["X"] = X.cpu().numpy()
                else:
                    p["E"] = torch.empty((k, grid.n), device="cuda", dtype=X.dtype)
                p["k"], p["s"] = k, X.shape[0]
            st["jobs"].append(p)
        stream.synchronize()
    return st


def run(st):
    c, ctx = st["case"], st["ctx"]
    with torch.cuda.stream(st["stream"]):
        if c["kind"] == "batch":
            for p in st["jobs"]:
                p["V"].copy_(p["X"])
            R.filter_correction_batch(ctx, [(p["op"], p["V"], p["case"]["s"], p["lam"], p["case"]["degree"], p["g1"],
                                             p["g2"]) for p in st["jobs"]])
            return [p["V"] for p in st["jobs"]]
        p = st["jobs"][0]
        if c["kind"] == "eigh":
            w, Q = R.small_eigh(ctx, p["X"])
            # an eigenvector's phase is arbitrary: make each one's largest entry positive
            q = Q[np.argmax(np.abs(Q), axis=0), np.arange(Q.shape[1])]
            return w, Q * (np.abs(q) / q)
        if c["kind"] == "solve":
            par = R.make_params(c["k"], c["tol"], precision=c["precision"], buffer=p["s"] - p["k"])
            if c["host"]:
                r = R.solve(ctx, p["op"], par, v0=p["X"])
                E = r.evecs
                q = np.take_along_axis(E, np.argmax(np.abs(E), axis=1)[:, None], 1)
                return r.evals, E * (np.abs(q) / q)
            par.v0_cols = p["s"]
            r = R.solve(ctx, p["op"], par, v0=p["X"].data_ptr(), host=False, evecs_out=p["E"])
            E = p["E"]
            q = torch.gather(E, 1, E.abs().argmax(1, keepdim=True))
            return r.evals, E * (q.abs() / q)
        p["V"].copy_(p["X"])
        if c["kind"] == "cholqr":
            R.cholqr(ctx, p["V"], c["n"], c["s"], c["complex"])
            return p["V"]
        if c["kind"] == "filter":
            R.filter_block(ctx, p["op"], p["V"], c["s"], c["degree"], p["g1"], p["g2"], c["precision"])
            return p["V"]
        if c["kind"] == "corr":
            R.filter_correction(ctx, p["op"], p["V"], c["s"], p["lam"], c["degree"], p["g1"], p["g2"])
            return p["V"]
        w, res, Q = R.rayleigh_ritz(ctx, p["op"], p["V"], p["W"], c["s"], c["count"])
        return w, res, Q, p["V"], p["W"]


def exact(c, seed):
    if c["kind"] == "batch":
        out = []
        for j, job in enumerate(_jobs(c)):
            grid, V, lam = _inputs(job, seed, j)
            out.append(_filtered(grid, V, job["degree"], *_gammas(grid, float(lam[0]))))
        return out
    grid, X, lam = _inputs(c, seed)
    if c["kind"] == "eigh":
        w, Q = torch.linalg.eigh(X)
        q = torch.gather(Q, 0, Q.abs().argmax(0, keepdim=True))
        return w, Q * (q.abs() / q)
    if c["kind"] == "cholqr":
        return _orthonormal(X)
    if c["kind"] in ("filter", "corr"):
        return _filtered(grid, X, c["degree"], *_gammas(grid, float(lam[0])))
    if c["kind"] == "solve":
        w, E = grid.eigenpairs(c["k"])
        q = torch.gather(E, 1, E.abs().argmax(1, keepdim=True))
        return w, E * (q.abs() / q)
    W = grid.apply(X)
    H = X.conj() @ W.mT
    w, Q = torch.linalg.eigh((H + H.mH) / 2)
    q = torch.diagonal(Q)[None]  # the block is nearly one of eigenvectors: Q is nearly the identity
    Q = Q * (q.abs() / q)
    V, W = Q.mT @ X, Q.mT @ W
    m = c["count"]
    res = torch.linalg.vector_norm(W[:m] - w[:m, None] * V[:m], dim=1)
    return w, res, Q, V, W


def work(c):
    """Inputs read once and outputs written once; the multiplications and additions of the operation itself."""
    if c["kind"] == "batch":
        w = [work(j) for j in _jobs(c)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    e, f = (16, 4) if c["complex"] else (8, 1)  # bytes of a scalar; real multiply-adds of one of its own
    if c["kind"] == "eigh":
        s = c["s"]
        return {"bytes": 2 * s * s * e + 8 * s, "flops": 9 * f * 2 * s ** 3 / 2}
    if c["kind"] == "cholqr":
        return {"bytes": 2 * c["n"] * c["s"] * e, "flops": 2 * f * c["n"] * c["s"] ** 2}
    n = c["nx"] * c["ny"] * c["nz"]
    op = n * (c["points"] * (e + 4) + 4) if c["form"] == "csr" else 8 * n
    apply = 2 * f * c["points"] * n
    if c["kind"] == "solve":
        s = c["k"] + max(8, -(-c["k"] // 2 // 8) * 8)
        its, deg = 40, 10  # a typical solve of this size
        return {"bytes": op + n * (s + c["k"]) * e, "flops": its * (deg * apply * s + 2 * f * 3 * n * s * s)}
    s = c["s"]
    if c["kind"] == "rr":
        return {"bytes": op + 3 * n * s * e, "flops": apply * s + 2 * f * 2.5 * n * s * s}
    return {"bytes": op + 2 * n * s * e, "flops": c["degree"] * (apply + 4 * n) * s}
