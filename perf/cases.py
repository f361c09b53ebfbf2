"""What the solver's speed is measured on: the solves that programs call, from
one small grid to the largest ones, through the Python mirror of the C ABI.

listed() are the standing cases, draw() makes more of the same ranges;
prepare() is what a program has in hand before a solve, run() is one solve (or
one batch), exact() the same discrete solution by dense transforms in torch.

Sizes are those of the benchmark (64^3, 256^3, 512^3, the 96-grid batch's edge
lengths) and generic ones: decimal edges, odd edges, a large flat grid.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

# edge lengths of the batch (the benchmark's list); nz is uniform in [32, 256]
BATCH_EDGES = (32, 48, 64, 96, 128, 160, 192)
FAMILIES = ("PP", "NN", "ND", "DD")
Z_ENDS = ("DD", "NN", "DN", "ND", "PP")
MAX_POINTS = 1024 * 1024 * 256


def _solve(name, nx, ny, nz, bc, rhs="real", precision="fp64", sweeps=0, faces=False):
    return {"name": name, "kind": "solve", "nx": nx, "ny": ny, "nz": nz, "bc": bc, "rhs": rhs,
            "precision": precision, "sweeps": sweeps, "faces": faces}


def listed():
    return [
        # a small periodic channel solved at every time step of a flow solver:
        # launches and latency count
        _solve("cube64_pp", 64, 64, 64, "PPPPDD"),
        # the smallest odd-sized grids (a coarse level, a test problem)
        _solve("odd_50x42x37", 50, 42, 37, "NNDDNN"),
        # people choose decimal edges
        _solve("decimal_200", 200, 200, 200, "NNNNDD"),
        _solve("decimal_500x400x300", 500, 400, 300, "DDNNND"),
        # mixed families, Neumann z, at a middling power of two
        _solve("cube256_nn_dd", 256, 256, 256, "NNDDNN"),
        # the benchmark's grid: the periodic family and the quarter-wave one
        _solve("cube512_pp", 512, 512, 512, "PPPPDD"),
        _solve("cube512_nd", 512, 512, 512, "NDNDDD"),
        # the largest: a wide flat domain with the caller's boundary values
        _solve("plate_1024x1024x256", 1024, 1024, 256, "DDNNDN", faces=True),
        # a complex right-hand side, periodic in all directions
        _solve("complex_192x160x144", 192, 160, 144, "PPPPPP", rhs="complex"),
        # FP32 transforms with one FP64 refinement sweep (reaches 1e-10)
        _solve("refined_256", 256, 256, 256, "NNDDNN", precision="refined", sweeps=1),
        # many uneven grids in one launch: the patches of a block-structured mesh
        {"name": "batch_48", "kind": "batch", "grids": 48, "shapes_seed": 7},
        # the drop-in call sequence of a host program: page-locked right-hand
        # side in, complex solution out
        {"name": "host_192x160x128", "kind": "host", "nx": 192, "ny": 160, "nz": 128, "bc": "NNNNDD"},
    ]


def _edge(rng: random.Random, lo: int, hi: int, any_length: bool) -> int:
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if any_length:
        return n
    # the nearest product of 2, 3 and 5
    best = None
    for a in range(11):
        for b in range(5):
            for c in range(4):
                m = 2 ** a * 3 ** b * 5 ** c
                if lo <= m <= hi and (best is None or abs(m - n) < abs(best - n)):
                    best = m
    return best


def _xy(rng: random.Random) -> str:
    # a periodic x with a non-periodic y is not a boundary set of a real problem
    # here (the reference drops the imaginary part of its x spectrum)
    x = rng.choice(FAMILIES)
    return x + ("PP" if x == "PP" else rng.choice(FAMILIES))


def draw(rng: random.Random):
    kind = rng.choices(("solve", "complex", "refined", "batch", "host"), (10, 2, 3, 2, 2))[0]
    if kind == "batch":
        return {"kind": "batch", "grids": rng.randint(8, 64), "shapes_seed": rng.randrange(1 << 30)}
    any_length = rng.random() < 0.3
    # lengths with a large prime factor are taken on small and middling grids
    limit = 1 << 22 if any_length else (1 << 24 if kind == "host" else MAX_POINTS // (10 if kind == "complex" else 5))
    top = 256 if any_length or kind == "host" else 1024
    while True:
        nx, ny = _edge(rng, 32, top, any_length), _edge(rng, 32, top, any_length)
        nz = int(round(math.exp(rng.uniform(math.log(24), math.log(min(top, 640))))))
        if nx * ny * nz <= limit:
            break
    case = {"kind": "host" if kind == "host" else "solve", "nx": nx, "ny": ny, "nz": nz,
            "bc": _xy(rng) + rng.choice(Z_ENDS)}
    if kind == "host":
        return case
    case.update(rhs="real", precision="fp64", sweeps=0, faces=False)
    if kind == "complex":
        case.update(rhs="complex", bc="PPPP" + rng.choice(Z_ENDS))
    elif kind == "refined":
        case.update(precision="refined", sweeps=1)
    else:
        case.update(faces=rng.random() < 0.3)
    return case


# ---- the grids of a case ------------------------------------------------------------
def _grids(case):
    """(nx, ny, nz, bc) of every grid of a case."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"], case["bc"])]
    rng = random.Random(case["shapes_seed"])
    out = []
    for _ in range(case["grids"]):
        nx, ny, nz = rng.choice(BATCH_EDGES), rng.choice(BATCH_EDGES), rng.randint(32, 256)
        out.append((nx, ny, nz, _xy(rng) + rng.choice(("DD", "NN"))))
    return out


def _singular(bc):
    return "D" not in bc


def _rhs(nx, ny, nz, bc, cplx, gen):
    """A forcing with large scales and noise: a few waves with N(0, 1)
    amplitudes over i.i.d. noise; zero mean where the problem is singular."""
    dev = gen.device
    dt = torch.complex128 if cplx else torch.float64
    f = torch.randn((nz, ny, nx), dtype=dt, device=dev, generator=gen)
    amp = torch.randn(4, dtype=torch.float64, device=dev, generator=gen)
    ph = torch.rand((4, 3), dtype=torch.float64, device=dev, generator=gen) * 2 * math.pi
    for w in range(4):
        z, y, x = (torch.cos(2 * math.pi * (w + 1) * torch.arange(m, dtype=torch.float64, device=dev) / m + ph[w, d])
                   for d, m in enumerate((nz, ny, nx)))
        f += (3.0 * amp[w]) * z[:, None, None] * y[None, :, None] * x[None, None, :]
    if _singular(bc):
        f -= f.mean()
    return f


def _faces(nx, ny, nz, bc, seed):
    """Boundary data of the Dirichlet faces: {face: array on the host}."""
    out = {}
    for face in range(6):
        if bc[face] != "D":
            continue
        na, nb = [(nz, ny), (nz, nx), (ny, nx)][face // 2]
        r = np.random.default_rng(seed * 7 + face)
        a = np.cos(2 * np.pi * r.integers(1, 4) * (np.arange(na) + 0.5) / na + r.uniform(0, 6))
        b = np.cos(2 * np.pi * r.integers(1, 4) * (np.arange(nb) + 0.5) / nb + r.uniform(0, 6))
        out[face] = r.standard_normal() * a[:, None] * b[None, :]
    return out


def _default_lift(nx, ny, nz, bc):
    """What the library subtracts on Dirichlet faces by default (the batch has
    no option for it): the reference's manufactured solution, sin or cos of
    pi x, 2 pi y, 3 pi z per direction, which on the unit box is zero but for
    the rounding of pi; nothing where x or y is periodic."""
    out = {}
    if "P" in bc[:4]:
        return out
    n = (nx, ny, nz)
    wave = [math.cos if bc[2 * d:2 * d + 2] == "NN" and d < 2 else math.sin for d in range(3)]
    at = lambda d, x: wave[d]((d + 1) * math.pi * x)
    centres = [np.array([at(d, (i + 0.5) / n[d]) for i in range(n[d])]) for d in range(3)]
    for face in range(6):
        d = face // 2
        if bc[face] == "D":
            u, v = [centres[e] for e in (2, 1, 0) if e != d]
            out[face] = 2.0 * at(d, float(face % 2)) * u[:, None] * v[None, :]
    return out


def _inputs(case, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    cplx = case.get("rhs") == "complex"
    return [_rhs(nx, ny, nz, bc, cplx, gen) for nx, ny, nz, bc in _grids(case)]


# ---- the measured calls -------------------------------------------------------------
def prepare(case, seed):
    import pittpack_b200 as pp
    from pittpack_b200.poisson import pinned_empty

    fs = _inputs(case, seed, "cuda")
    if case["kind"] == "batch":
        from pittpack_b200.batch import Batch

        Ps = [torch.empty(f.shape, dtype=torch.complex128, device="cuda") for f in fs]
        # launch shapes left at their defaults, so that two runs time the same work
        items = [{"nx": nx, "ny": ny, "nz": nz, "bc": bc, "d_rhs": f.data_ptr(), "d_P": P.data_ptr()}
                 for (nx, ny, nz, bc), f, P in zip(_grids(case), fs, Ps)]
        torch.cuda.synchronize()
        B = Batch(items, precision=0, autotune=False)
        return {"kind": "batch", "batch": B, "rhs": fs, "P": Ps}
    (nx, ny, nz, bc), f = _grids(case)[0], fs[0]
    M = pp.make_Poisson(nx, ny, nz)
    if case["kind"] == "host":
        M.setOptions(dirichlet_lift=0)
        M.assignBoundary(bc)
        M.setBox([0, 1, 0, 1, 0, 1])
        rhs = pinned_empty((nz, ny, nx), np.float64)
        rhs[...] = f.cpu().numpy()
        out = pinned_empty((nz, ny, nx), np.complex128)
        return {"kind": "host", "M": M, "rhs": rhs, "P": out}
    refined = case["precision"] == "refined"
    M.setOptions(dirichlet_lift=0, precision=int(refined), max_sweeps=case["sweeps"],
                 compat_zero_mode=0 if refined else 1)
    M.assignBoundary(bc)
    M.setBox([0, 1, 0, 1, 0, 1])
    if case["faces"]:
        for face, g in _faces(nx, ny, nz, bc, seed).items():
            M.setFaceValues(face, g)
    P = torch.empty((nz, ny, nx), dtype=torch.complex128, device="cuda")
    M.bindDeviceBuffers(f.data_ptr(), f.is_complex(), P.data_ptr())
    torch.cuda.synchronize()
    return {"kind": "solve", "M": M, "rhs": f, "P": P}


def run(state):
    if state["kind"] == "batch":
        state["batch"].run(torch.cuda.current_stream().cuda_stream)
        return state["P"]
    M = state["M"]
    if state["kind"] == "host":
        M.assignRhs(state["rhs"])
        M.pittPack()
        return M.getSolution(state["P"])
    M.setStream(torch.cuda.current_stream().cuda_stream)
    M.pittPack()
    return state["P"]


def work(case):
    """Right-hand side read once and the complex P written once; the real FFT
    work of both directions and the tridiagonal sweeps."""
    cplx = case.get("rhs") == "complex"
    nbytes = flops = 0.0
    for nx, ny, nz, _bc in _grids(case):
        n = nx * ny * nz
        nbytes += n * (32 if cplx else 24)
        per = 2 * (2.5 * math.log2(nx) + 2.5 * math.log2(ny)) + 8
        flops += n * per * (2 if cplx else 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # FP64: 4e-13 against exact() at 512^3, the rounding of 2 cos t - 2 in the
    # lowest modes' eigenvalues, which grows with the square of the edge; one
    # refinement sweep from FP32 transforms leaves 4e-12
    if case.get("precision") == "refined":
        return {"rel": 1.6e-11}
    m = max(max(g[:3]) for g in _grids(case))
    return {"rel": 1.6e-12 * max(1.0, (m / 512) ** 2)}


# ---- the same solution by dense transforms --------------------------------------------
def _basis(n, ends, dev):
    """Orthonormal eigenvectors (rows) of the 1-D second difference with the
    given ends, and its eigenvalues.  Angles are whole multiples of pi / (4 n),
    reduced in integers."""
    k = torch.arange(n, dtype=torch.int64, device=dev)[:, None]
    j = torch.arange(n, dtype=torch.int64, device=dev)[None, :]
    ang = lambda m, den: (m % (2 * den)).to(torch.float64) * (math.pi / den)  # pi m / den
    if ends == "NN":
        q = torch.cos(ang(k * (2 * j + 1), 2 * n)) * math.sqrt(2.0 / n)
        q[0] *= math.sqrt(0.5)
        lam = ang(k[:, 0], n)
    elif ends == "DD":
        q = torch.sin(ang((k + 1) * (2 * j + 1), 2 * n)) * math.sqrt(2.0 / n)
        q[-1] *= math.sqrt(0.5)
        lam = ang(k[:, 0] + 1, n)
    elif ends in ("ND", "DN"):
        a = ang((2 * k + 1) * (2 * j + 1), 4 * n)
        q = (torch.cos(a) if ends == "ND" else torch.sin(a)) * math.sqrt(2.0 / n)
        lam = ang(2 * k[:, 0] + 1, 2 * n)
    else:
        # cosines of k = 0 .. n/2, then sines of k = 1 .. (n-1)/2
        h = n // 2
        m = torch.where(k <= h, k, k - h)
        a = ang(2 * m * j, n)
        q = torch.where(k <= h, torch.cos(a), torch.sin(a)) * math.sqrt(2.0 / n)
        q[0] *= math.sqrt(0.5)
        if n % 2 == 0:
            q[h] *= math.sqrt(0.5)
        lam = ang(2 * m[:, 0], n)
    s = torch.sin(0.5 * lam)
    return q, -4.0 * s * s  # 2 cos(lam) - 2


def _apply(q, a, dim):
    """q applied along a dimension of a (z, y, x) array, real or complex."""
    if a.is_complex():
        return torch.complex(_apply(q, a.real.contiguous(), dim), _apply(q, a.imag.contiguous(), dim))
    if dim == 2:
        return a @ q.T
    if dim == 1:
        return torch.matmul(q, a)
    return torch.matmul(q, a.reshape(a.shape[0], -1)).reshape(a.shape)


def _thomas(lam, r, zlo, zhi):
    """x_{k-1} + lam x_k + x_{k+1} = r_k with Dirichlet / Neumann ends, in place in r."""
    nz = r.shape[0]
    one = {"D": -1.0, "N": 1.0}
    c = torch.empty((nz,) + lam.shape, dtype=torch.float64, device=r.device)
    b = lam + one[zlo]
    c[0] = 1.0 / b
    r[0] *= c[0]
    for k in range(1, nz):
        b = lam - c[k - 1]
        if k == nz - 1:
            b = b + one[zhi]
        torch.reciprocal(b, out=c[k])
        r[k] -= r[k - 1]
        r[k] *= c[k]
    for k in range(nz - 2, -1, -1):
        r[k] -= c[k] * r[k + 1]
    return r


def _zero_column(col, nz, zlo, zhi, pin):
    """The kx = ky = 0 column, its first row replaced where it is pinned (the
    reference's x_0 = r_0; for periodic z x_0 + x_{nz-1} = (r_0 + r_{nz-1}) / 2)."""
    A = torch.zeros((nz, nz), dtype=torch.float64)
    i = torch.arange(nz)
    A[i, i] = -2.0
    A[i[1:], i[:-1]] = 1.0
    A[i[:-1], i[1:]] = 1.0
    r = col.cpu().clone()
    if zlo == "P":
        A[0, -1] = A[-1, 0] = 1.0
        if pin:
            A[0] = 0.0
            A[0, 0] = A[0, -1] = 1.0
            r[0] = 0.5 * (r[0] + r[-1])
    else:
        A[0, 0] += 1.0 if zlo == "N" else -1.0
        A[-1, -1] += 1.0 if zhi == "N" else -1.0
        if pin:
            A[0] = 0.0
            A[0, 0] = 1.0
    return torch.linalg.solve(A.to(r.dtype), r[:, None])[:, 0].to(col.device)


def _exact_one(nx, ny, nz, bc, f, faces, lift, pin_always):
    dev = f.device
    dx, dy, dz = 1.0 / nx, 1.0 / ny, 1.0 / nz
    w = [(dz / dx) ** 2, (dz / dy) ** 2, 1.0]
    b = f * (dz * dz)
    terms = {face: (2.0 * w[face // 2]) * g for face, g in faces.items()}  # Dirichlet: the ghost cell 2 g - u_0
    terms.update(lift)
    for face, g in terms.items():
        g = torch.as_tensor(g, device=dev)
        at = 0 if face % 2 == 0 else -1
        if face < 2:
            b[:, :, at] -= g
        elif face < 4:
            b[:, at, :] -= g
        else:
            b[at] -= g
    qx, ex = _basis(nx, bc[0:2], dev)
    qy, ey = _basis(ny, bc[2:4], dev)
    b = _apply(qy, _apply(qx, b, 2), 1)
    lam = -2.0 + ey[:, None] * w[1] + ex[None, :] * w[0]
    has_zero = all(bc[d:d + 2] in ("NN", "PP") for d in (0, 2))
    col = b[:, 0, 0].clone() if has_zero else None
    if has_zero:
        lam[0, 0] = -4.0  # solved separately
    if bc[4] == "P":
        qz, ez = _basis(nz, "PP", dev)
        b = _apply(qz, b, 0)
        b /= (lam + 2.0)[None] + ez[:, None, None]
        b = _apply(qz.T.contiguous(), b, 0)
    else:
        b = _thomas(lam, b, bc[4], bc[5])
    if has_zero:
        b[:, 0, 0] = _zero_column(col, nz, bc[4], bc[5], pin_always or "D" not in bc[4:6])
    b = _apply(qx.T.contiguous(), _apply(qy.T.contiguous(), b, 1), 2)
    return b if b.is_complex() else torch.complex(b, torch.zeros_like(b))


def exact(case, seed):
    fs = _inputs(case, seed, "cuda")
    refined = case.get("precision") == "refined"
    out = []
    for (nx, ny, nz, bc), f in zip(_grids(case), fs):
        faces = _faces(nx, ny, nz, bc, seed) if case.get("faces") else {}
        lift = _default_lift(nx, ny, nz, bc) if case["kind"] == "batch" else {}
        out.append(_exact_one(nx, ny, nz, bc, f, faces, lift, not refined))
    if case["kind"] == "batch":
        return out
    return out[0].cpu().numpy() if case["kind"] == "host" else out[0]
