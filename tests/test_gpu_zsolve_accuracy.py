"""The z solve's error on a nearly singular mode does not depend on how its
rows are split over lanes: one x/y mode with lambda = -(2 + e), e down to
1e-6, solved on the GPU with every lane count and row capacity and compared
with the same system (the same FP64 lambda) solved in 60 decimal digits.

A diagonal that an elimination forms by subtraction loses up to 2^-53 / e of
the solution (1e-10 here); carried as row sums nothing cancels, and what is
left is the rounding of the transforms, of the sweeps over a lane's rows and
of the right-hand side: relative L2 <= 32 * 2^-53 asked for, 3.6e-15."""
import math
from decimal import Decimal, getcontext
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 32 * 2.0 ** -53


def _thomas(lam, r, first, last):
    b = [lam] * len(r)
    b[0] += first
    b[-1] += last
    c, x = [], []
    for k, v in enumerate(r):
        d = 1 / (b[k] - (c[-1] if c else 0))
        x.append((v - (x[-1] if x else 0)) * d)
        c.append(d)
    for k in range(len(r) - 2, -1, -1):
        x[k] -= c[k] * x[k + 1]
    return x


def _exact(lam, r, ends):
    getcontext().prec = 60
    lam, r = Decimal(lam), [Decimal(float(v)) for v in r]
    if ends != "PP":
        one = {"D": -1, "N": 1}
        return np.array([float(v) for v in _thomas(lam, r, one[ends[0]], one[ends[1]])])
    # corners 1: T + u v^T with u = v = (1, 0, .., 0, 1), T's end rows lambda - 1
    y = _thomas(lam, r, -1, -1)
    z = _thomas(lam, [Decimal(int(k in (0, len(r) - 1))) for k in range(len(r))], -1, -1)
    s = (y[0] + y[-1]) / (1 + z[0] + z[-1])
    return np.array([float(v - s * q) for v, q in zip(y, z)])


def _check(bcxy, ends, nz, e, lanes):
    import pittpack_b200 as pp

    n = 16
    # the lowest mode of the D-D direction; the other one has a constant mode
    y = bcxy[2:4] == "DD"
    part = -2.0 + 2.0 * math.cos((0 + 1.0) * math.pi / n)
    h, dz = math.sqrt(-part / e) / nz, 1.0 / nz  # cell size of that direction: -part (dz / h)^2 = e
    box = [0.0, 1.0, 0.0, n * h, 0.0, 1.0] if y else [0.0, n * h, 0.0, 1.0, 0.0, 1.0]
    ratio = -(box[4] - box[5]) / nz / (-(0.0 - n * h) / n)
    lam = float(Fraction(-2) + Fraction(part) * Fraction(ratio * ratio))
    r = np.random.default_rng(nz).uniform(0.5, 1.5, nz)
    s = np.sin(math.pi * (np.arange(n) + 0.5) / n)
    mode = s[:, None] * np.ones(n) if y else np.ones(n)[:, None] * s
    X = (_exact(lam, r, ends) * dz * dz)[:, None, None] * mode
    with pp.make_Poisson(n, n, nz) as M:
        M.setOptions(dirichlet_lift=0)
        M.assignBoundary(bcxy + ends)
        M.setBox(box)
        M.assignRhs(r[:, None, None] * mode)
        for P in lanes:
            M.setTuning(zsolve_lanes=P)
            M.pittPack()
            err = np.linalg.norm(M.getSolution() - X) / np.linalg.norm(X)
            assert err <= TOL, (P, err)


@pytest.mark.parametrize("ends", ["NN", "DN", "ND", "DD", "PP"])
@pytest.mark.parametrize("bcxy", ["NNDD", "DDPP"])  # real and complex spectra
@pytest.mark.parametrize("nz", [9, 37, 60, 100, 160, 210, 300, 512])
def test_lanes(nz, bcxy, ends):
    for e in (1e-6, 1e-3, 3.0):
        _check(bcxy, ends, nz, e, [0] + [P for P in (1, 2, 4, 8, 16, 32) if P == 1 or P <= nz // 2])


@pytest.mark.parametrize("ends", ["NN", "DN", "PP"])
def test_long_systems(ends):
    # rows in shared memory, and blocks whose pivots take the division recurrence
    for nz, lanes in ((1500, (8, 32)), (9000, (8, 32))):
        _check("NNDD", ends, nz, 1e-6, lanes)
