"""Boundary data on every face through the planned kernel's forward x pass
(pp_mr.cuh), which subtracts it where the face's elements lie in the FFT
input: each family, lengths planned at compile time and (factors 11 and 13) at
run time, even and odd, partial tiles, unaligned buffers, real and complex
right-hand sides, against the oracle: relative L2 <= 1e-12."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_half_length import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bcxy", ["NNDD", "DDNN", "NDDD", "DNND", "PPDD", "PPPP"])
@pytest.mark.parametrize("nx", [50, 96, 200, 384, 44, 26, 33, 39, 143])
def test_faces(nx, bcxy):
    ny, nz = 19, 6
    rng = np.random.default_rng(nx)
    f, g = rng.uniform(-1, 1, (2, nz, ny, nx))
    bc = bcxy + "DN"
    faces = {face: rng.uniform(-1, 1, [(nz, ny), (nz, nx), (ny, nx)][face // 2]) for face in range(6) if bc[face] != "P"}
    pb = O.problem(nx, ny, nz, bc, dirichlet_lift=0, faces=faces)
    Q = O.solve(pb, f)
    for off in (0, 1):
        assert O.rel_l2(solve(nx, ny, nz, bc, f, off, faces=faces), Q) <= 1e-12
    if bcxy[:2] == bcxy[2:] or bcxy[0] != "P":
        assert O.rel_l2(solve(nx, ny, nz, bc, f + 1j * g, faces=faces), O.solve(pb, f, g)) <= 1e-12
