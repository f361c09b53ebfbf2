"""The half-length real transform pass (pp_rhalf.cuh): every length it takes,
in x and in y, each boundary family, with line counts that leave a partial
tile, buffers that start off the kernel's widest accesses, complex right-hand
sides (real families read the real part) and face values, against the oracle.

Tolerance: relative L2 <= 1e-12 in FP64 (the plain path's bar), 1e-10 for the
refined solve.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LENGTHS = [32, 64, 128, 256, 512, 1024]
# (x family, y family) with the length in x, then in y; PP-PP: half spectra in x
PAIRS = ["NNDD", "DDNN", "NDND", "DNDN", "PPPP", "NDPP", "NNPP"]


def solve(nx, ny, nz, bc, f, off=0, faces=None, **opts):
    import torch

    import pittpack_b200 as pp

    fd = torch.as_tensor(np.ascontiguousarray(f)).cuda()
    n = fd.numel()
    cplx = fd.is_complex()
    raw = torch.zeros(n + 4, dtype=fd.dtype, device="cuda")
    out = torch.zeros(n + 4, dtype=torch.complex128, device="cuda")
    raw[off:off + n] = fd.reshape(-1)
    with pp.make_Poisson(nx, ny, nz) as M:
        M.setOptions(dirichlet_lift=0, **opts)
        M.assignBoundary(bc)
        M.setBox([0, 1, 0, 1, 0, 1])
        for face, g in (faces or {}).items():
            M.setFaceValues(face, g)
        # an odd offset leaves the real RHS on an 8-byte boundary and P on a 16-byte one
        M.bindDeviceBuffers(raw.data_ptr() + off * raw.element_size(), cplx, out.data_ptr() + 16 * off)
        torch.cuda.synchronize()
        M.pittPack()
        M.synchronize()
    return out[off:off + n].cpu().numpy().reshape(nz, ny, nx)


@pytest.mark.parametrize("bcxy", PAIRS)
@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", ["x", "y"])
def test_lengths(axis, n, bcxy):
    # 37 lines (or 36, padded spectrum columns): a partial tile at every tile width
    nx, ny, nz = (n, 37, 9) if axis == "x" else (37, n, 9)
    rng = np.random.default_rng(n)
    f = rng.uniform(-1, 1, (nz, ny, nx))
    for off in (0, 1):
        Q = O.solve(O.problem(nx, ny, nz, bcxy + "DN", dirichlet_lift=0), f)
        assert O.rel_l2(solve(nx, ny, nz, bcxy + "DN", f, off), Q) <= 1e-12


@pytest.mark.parametrize("bcxy", ["NNDD", "DDND", "NDNN", "PPPP", "DDPP"])
@pytest.mark.parametrize("n", [32, 128, 512, 1024])
def test_complex_rhs_and_faces(n, bcxy):
    nx, ny, nz = n, 32, 6
    rng = np.random.default_rng(7 + n)
    f = rng.uniform(-1, 1, (nz, ny, nx))
    g = rng.uniform(-1, 1, (nz, ny, nx))
    bc = bcxy + "DD"
    Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0), f, g)
    assert O.rel_l2(solve(nx, ny, nz, bc, f + 1j * g), Q) <= 1e-12
    faces = {}
    for face in range(6):
        if bc[face] != "P":
            faces[face] = rng.uniform(-1, 1, [(nz, ny), (nz, nx), (ny, nx)][face // 2])
    Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0, faces=faces), f)
    assert O.rel_l2(solve(nx, ny, nz, bc, f, faces=faces), Q) <= 1e-12


@pytest.mark.parametrize("bcxy", ["NNDD", "DNND", "PPPP"])
@pytest.mark.parametrize("n", LENGTHS)
def test_refined(n, bcxy):
    # both directions in FP32, the epilogues of every sweep
    rng = np.random.default_rng(n + 3)
    for nx, ny in ((n, 34), (34, n)):
        nz = 12
        f = rng.uniform(-1, 1, (nz, ny, nx))
        Q = O.solve(O.problem(nx, ny, nz, bcxy + "DN", compat_zero_mode=0, dirichlet_lift=0), f)
        for off in (0, 1):
            P = solve(nx, ny, nz, bcxy + "DN", f, off, precision=1, max_sweeps=2, compat_zero_mode=0)
            assert O.rel_l2(P, Q) <= 1e-10
