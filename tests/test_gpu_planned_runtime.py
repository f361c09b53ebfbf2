"""The transform pass whose plan is read at run time (pp_mr.cuh), on grids large
enough that it is taken for lengths of factors 2, 3, 5 and 7 (350,000 points,
complex lines of three passes 8,000,000), and the generic kernel just below,
in x and in y, against the oracle: relative L2 <= 1e-12 in FP64, <= 1e-10 for
the refined solve."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_planned_lengths import solve

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

POINTS = 350000
# even (half length, M even and odd) and odd, every radix, two to four passes
LENGTHS = [9, 14, 18, 25, 27, 28, 30, 35, 42, 45, 56, 63, 70, 75, 98, 105, 112, 135, 175, 252, 315, 350, 490, 625, 700]
FAMS = {("x", 0): ["NNDD", "NDND", "PPPP"], ("x", 1): ["DDNN", "PPNN"],
        ("y", 0): ["DDNN", "NDND", "NNPP"], ("y", 1): ["NNDD", "DDPP"]}


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", ["x", "y"])
def test_lengths(axis, n):
    m = 61 if n % 2 else 64
    for q, bc in enumerate(FAMS[axis, n % 2]):
        # the first count of planes that takes the plan; the last one that does not, once
        nz = -(-POINTS // (n * m))
        for k in (nz, nz - 1)[:1 + (q == 0)]:
            nx, ny = (n, m) if axis == "x" else (m, n)
            f = np.random.default_rng(n + q).uniform(-1, 1, (k, ny, nx))
            Q = O.solve(O.problem(nx, ny, k, bc + "DN"), f)
            assert O.rel_l2(solve(nx, ny, k, bc + "DN", f, off=q % 2), Q) <= 1e-12, (bc, k)


@pytest.mark.parametrize("n", [18, 30, 45, 63, 98, 175, 350])
def test_refined(n):
    nx, ny, nz = n, 64, -(-POINTS // (n * 64))
    f = np.random.default_rng(n).uniform(-1, 1, (nz, ny, nx))
    Q = O.solve(O.problem(nx, ny, nz, "NNDDDN", compat_zero_mode=0), f)
    assert O.rel_l2(solve(nx, ny, nz, "NNDDDN", f, precision=1, max_sweeps=2, compat_zero_mode=0), Q) <= 1e-10


@pytest.mark.parametrize("nx,ny,nz,bc", [(189, 212, 200, "PPPPDD"), (200, 196, 206, "NNPPDN")])
def test_complex_lines_of_three_passes(nx, ny, nz, bc):
    assert nx * ny * nz >= 8000000
    f = np.random.default_rng(nx).uniform(-1, 1, (nz, ny, nx))
    Q = O.solve(O.problem(nx, ny, nz, bc), f)
    assert O.rel_l2(solve(nx, ny, nz, bc, f), Q) <= 1e-12
