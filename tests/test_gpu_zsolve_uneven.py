"""The z solve at any row count: two half blocks per lane with M, M - 1 or
M - 2 rows, every lane count that leaves a lane at least two rows, real and
complex spectra, each pair of z ends (periodic with and without the zero
mode), bulk-copied z-tiled and element-copied tiles, FP64 (relative L2 <= 1e-12
against the oracle) and FP32 spectra (refined solve, <= 1e-10)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

NZ = [3, 5, 8, 9, 10, 11, 13, 15, 17, 18, 19, 21, 23, 25, 27, 29, 31, 33, 37, 41, 50, 57, 63, 65, 75, 100, 129, 200, 301]


def _rhs(shape, seed, bc):
    f = np.random.default_rng(seed).uniform(-1, 1, shape)
    return f - f.mean() if "D" not in bc else f


@pytest.mark.parametrize("bc", ["NNNNDD", "NNNNPP", "DDNDPP", "NDNDDN", "PPPPPP", "PPPPND"])
@pytest.mark.parametrize("nz", NZ)
def test_lanes(nz, bc):
    import pittpack_b200 as pp

    nx, ny = 32, 16
    f = _rhs((nz, ny, nx), nz, bc)
    Q = O.solve(O.problem(nx, ny, nz, bc), f)
    with pp.make_Poisson(nx, ny, nz) as M:
        M.assignBoundary(bc)
        M.assignRhs(f)
        for lanes in (0, 1, 2, 4, 8, 16, 32):
            if lanes > 1 and lanes > nz // 2:
                continue
            for tile in (0, 1):
                M.setTuning(zsolve_lanes=lanes, zsolve_tile=tile)
                M.pittPack()
                assert O.rel_l2(M.getSolution(), Q) <= 1e-12, (lanes, tile)
        assert M.kernelTimeouts() == 0


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("bc", ["NNNNDD", "NDNDPP", "DDNDDN", "NNPPNN"])
@pytest.mark.parametrize("nz", NZ)
def test_bulk_tiles(nz, bc, precision):
    # ny = 64: the y pass has 8 lines a tile, real spectra too, so that the lanes
    # that leave a CTA its 8 systems copy their blocks of rows in bulk
    import pittpack_b200 as pp

    nx, ny = 24, 64
    f = _rhs((nz, ny, nx), nz, bc)
    Q = O.solve(O.problem(nx, ny, nz, bc, compat_zero_mode=1 - precision), f)
    with pp.make_Poisson(nx, ny, nz) as M:
        M.setOptions(precision=precision, max_sweeps=3, compat_zero_mode=1 - precision)
        M.assignBoundary(bc)
        M.assignRhs(f)
        for lanes in (0, 1, 2, 4, 8, 16, 32):
            if lanes > 1 and lanes > nz // 2:
                continue
            M.setTuning(zsolve_lanes=lanes)
            M.pittPack()
            assert O.rel_l2(M.getSolution().real, Q.real) <= (1e-10 if precision else 1e-12), lanes
        assert M.kernelTimeouts() == 0


@pytest.mark.parametrize("bc", ["NNNNDD", "PPPPPP", "NDPPDN"])
@pytest.mark.parametrize("nz", [9, 19, 25, 37, 50, 75, 129])
def test_refined(nz, bc):
    import pittpack_b200 as pp

    nx, ny = 32, 16
    f = _rhs((nz, ny, nx), nz + 1, bc)
    Q = O.solve(O.problem(nx, ny, nz, bc, compat_zero_mode=0), f)
    with pp.make_Poisson(nx, ny, nz) as M:
        M.setOptions(precision=1, max_sweeps=3, compat_zero_mode=0)
        M.assignBoundary(bc)
        M.assignRhs(f)
        for lanes in (0, 1, 2, 4):
            M.setTuning(zsolve_lanes=lanes)
            M.pittPack()
            assert O.rel_l2(M.getSolution().real, Q.real) <= 1e-10, lanes
