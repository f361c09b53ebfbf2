"""The contiguous x passes of lengths m 2^k that run the register kernel
(pp_lpm_takes): complex lines, half spectra (complex, and real after a
non-periodic y), DCT-II/III and DST-II/III, with a last partial tile, buffers
that start on and off 16 bytes, complex right-hand sides and face values,
against the oracle: relative L2 <= 1e-12."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_half_length import solve

pytestmark = pytest.mark.gpu

LENGTHS = [320, 480, 576, 640, 768, 960, 1152, 1280, 1536]


@pytest.mark.parametrize("bcxy", ["NNDD", "DDNN", "PPPP", "PPND", "NNPP"])
@pytest.mark.parametrize("nx", LENGTHS)
def test_real_rhs(nx, bcxy):
    ny, nz = 18 if bcxy[2] != "P" else 23, 5
    rng = np.random.default_rng(nx)
    f = rng.uniform(-1, 1, (nz, ny, nx))
    bc = bcxy + "DN"
    Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0), f)
    for off in (0, 1):
        assert O.rel_l2(solve(nx, ny, nz, bc, f, off), Q) <= 1e-12, off
    faces = {face: rng.uniform(-1, 1, [(nz, ny), (nz, nx), (ny, nx)][face // 2]) for face in range(6) if bc[face] != "P"}
    Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0, faces=faces), f)
    assert O.rel_l2(solve(nx, ny, nz, bc, f, faces=faces), Q) <= 1e-12


@pytest.mark.parametrize("bcxy", ["NNDD", "DDNN", "PPPP"])
@pytest.mark.parametrize("nx", LENGTHS)
def test_complex_rhs(nx, bcxy):
    ny, nz = 19 if bcxy[2] == "P" else 16, 5
    rng = np.random.default_rng(nx + 1)
    f, g = rng.uniform(-1, 1, (2, nz, ny, nx))
    Q = O.solve(O.problem(nx, ny, nz, bcxy + "DD", dirichlet_lift=0), f, g)
    assert O.rel_l2(solve(nx, ny, nz, bcxy + "DD", f + 1j * g), Q) <= 1e-12
