"""The transform pass planned from the length (pp_mr.cuh): lengths planned at
compile time and at run time (on grids this small the even DCT / DST ones and those
with a factor 11 or 13; the others take the generic kernel here, and the plan in
test_gpu_planned_runtime.py),
even (half-length FFT) and odd (two lines per FFT), every radix, in x and in y, with partial tiles, buffers off the widest
accesses, padded spectrum columns and complex right-hand sides, against the
oracle: relative L2 <= 1e-12 in FP64, <= 1e-10 for the refined solve."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

COMPILED = [40, 48, 50, 54, 60, 72, 80, 90, 96, 100, 108, 120, 144, 150, 160, 162, 180, 192, 200, 216, 240, 250, 270,
            288, 300, 320, 324, 360, 384, 400, 432, 450, 480, 500, 540, 576, 600, 640, 720, 750, 768, 800, 864, 900,
            960, 1000, 1152, 1200, 1280, 1536]
# even: radices 2 .. 20 and their mixtures, M odd and even; odd; one past a tile of 8 lines
RUNTIME = [8, 10, 12, 14, 18, 20, 22, 24, 26, 28, 30, 36, 42, 44, 52, 56, 66, 70, 78, 98, 110, 126, 130, 154, 168, 182,
           242, 338, 490, 686, 1100, 1750, 2000, 2500, 5000,
           9, 11, 13, 15, 21, 25, 27, 33, 35, 39, 45, 49, 55, 63, 75, 77, 81, 91, 99, 105, 117, 121, 125, 135, 143, 169,
           225, 243, 343, 375, 625, 1125]
FAMS = ["NNDD", "DDNN", "NDDN", "PPPP", "NNPP"]


def solve(nx, ny, nz, bc, f, off=0, **opts):
    import torch

    import pittpack_b200 as pp

    fd = torch.as_tensor(np.ascontiguousarray(f)).cuda()
    n = fd.numel()
    raw = torch.zeros(n + 4, dtype=fd.dtype, device="cuda")
    out = torch.zeros(n + 4, dtype=torch.complex128, device="cuda")
    raw[off:off + n] = fd.reshape(-1)
    with pp.make_Poisson(nx, ny, nz) as M:
        M.setOptions(**opts)
        M.assignBoundary(bc)
        M.setBox([0, 1, 0, 1, 0, 1])
        M.bindDeviceBuffers(raw.data_ptr() + off * raw.element_size(), fd.is_complex(), out.data_ptr() + 16 * off)
        torch.cuda.synchronize()
        M.pittPack()
        M.synchronize()
    return out[off:off + n].cpu().numpy().reshape(nz, ny, nx)


@pytest.mark.parametrize("n", COMPILED + RUNTIME)
@pytest.mark.parametrize("axis", ["x", "y"])
def test_lengths(axis, n):
    nz = 5
    for q, bc in enumerate(FAMS):
        m = (19, 32, 21, 36, 33)[q]
        nx, ny = (n, m) if axis == "x" else (m, n)
        f = np.random.default_rng(n + q).uniform(-1, 1, (nz, ny, nx))
        if q == 3 and n % 4 == 0:
            f = f + 1j * np.random.default_rng(n).uniform(-1, 1, f.shape)
        fr, fi = (f.real.copy(), f.imag.copy()) if np.iscomplexobj(f) else (f, None)
        Q = O.solve(O.problem(nx, ny, nz, bc + "DN"), fr, fi)
        assert O.rel_l2(solve(nx, ny, nz, bc + "DN", f, off=q % 2), Q) <= 1e-12, bc


@pytest.mark.parametrize("n", [50, 60, 100, 250, 300, 576, 768, 1000, 42, 66, 130, 242, 45, 81, 125, 143])
@pytest.mark.parametrize("bc", ["NNDD", "NDDN", "PPPP"])
def test_refined(n, bc):
    nz = 10
    rng = np.random.default_rng(n)
    for nx, ny in ((n, 35), (36, n)):
        f = rng.uniform(-1, 1, (nz, ny, nx))
        Q = O.solve(O.problem(nx, ny, nz, bc + "DN", compat_zero_mode=0), f)
        P = solve(nx, ny, nz, bc + "DN", f, precision=1, max_sweeps=2, compat_zero_mode=0)
        assert O.rel_l2(P, Q) <= 1e-10


@pytest.mark.parametrize("nx,ny,nz,bc", [(200, 200, 24, "NNNNDD"), (300, 200, 40, "DDNDPP"), (100, 300, 33, "PPPPNN"),
                                         (250, 96, 75, "NDPPDN"), (75, 125, 50, "DDNNND")])
def test_decimal_grids(nx, ny, nz, bc):
    # many tiles, z-tiled and plain spectra, the Dirichlet lift of the default options
    f = np.random.default_rng(nx).uniform(-1, 1, (nz, ny, nx))
    Q = O.solve(O.problem(nx, ny, nz, bc), f)
    assert O.rel_l2(solve(nx, ny, nz, bc, f), Q) <= 1e-12
