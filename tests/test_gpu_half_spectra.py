"""Periodic x with a non-periodic y and a real right-hand side: the x spectrum
is kept as half spectra, whose imaginary part the y transform drops (the
reference's quirk, src/signalProc.cpp:160-195), so that the inverse x pass
reads a real half spectrum.  Every kernel of that pass (powers of two,
lengths planned at compile time and at run time, 2048), whole z tiles and
padded columns, aligned and unaligned buffers, plain and refined solves, the
batch and the staged slabs, against the oracle: relative L2 <= 1e-12 in FP64,
a few FP32 roundings refined."""
import os

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_half_length import solve
from test_gpu_slab import _run

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

POW2 = [32, 64, 128, 256, 512, 1024, 2048]
PLANNED = [50, 96, 200, 500]  # at compile time
RUNTIME = [34, 42, 98, 154]   # at run time; 34 = 2 * 17 has no plan: the full spectrum
YS = ["NN", "DD", "ND", "DN"]


def _rhs(nx, ny, nz, seed=0):
    return np.random.default_rng(nx * ny + nz + seed).uniform(-1, 1, (nz, ny, nx))


@pytest.mark.parametrize("y", YS)
@pytest.mark.parametrize("nx", POW2 + PLANNED + RUNTIME)
def test_plain(nx, y):
    # ny: 8 lines a y tile (z-tiled spectrum), a planned length, no common tile
    for ny, nz, off in ((64, 11, 0), (48, 9, 1), (21 if y in ("NN", "DD") else 22, 7, 1)):
        bc = "PP" + y + "DN"
        f = _rhs(nx, ny, nz)
        Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0), f)
        assert O.rel_l2(solve(nx, ny, nz, bc, f, off), Q) <= 1e-12, (ny, off)


@pytest.mark.parametrize("bc", ["PPNNNN", "PPNNPP", "PPDDPP", "PPNDNN"])
def test_other_z_ends(bc):
    nx, ny, nz = 64, 48, 40
    f = _rhs(nx, ny, nz)
    if bc[2:4] == "NN":
        f -= f.mean()
    Q = O.solve(O.problem(nx, ny, nz, bc, dirichlet_lift=0), f)
    assert O.rel_l2(solve(nx, ny, nz, bc, f), Q) <= 1e-12


@pytest.mark.parametrize("y", YS)
@pytest.mark.parametrize("nx", [32, 256, 1024, 50, 200, 42])
def test_refined(nx, y):
    ny, nz = 40, 12
    bc = "PP" + y + "DN"
    f = _rhs(nx, ny, nz)
    # the part that is odd in x is dropped by every correction: the residual keeps
    # the right-hand side's, and u keeps what the FP32 transforms' rounding puts
    # there, so that the sweeps end at a few 2^-24 of the solution (0.2 .. 3 of
    # them where this was measured; 16 allowed)
    Q = O.solve(O.problem(nx, ny, nz, bc, compat_zero_mode=0, dirichlet_lift=0), f)
    for off in (0, 1):
        P = solve(nx, ny, nz, bc, f, off, precision=1, max_sweeps=2, compat_zero_mode=0)
        assert O.rel_l2(P.real, Q.real) <= 16 * 2.0 ** -24


@pytest.mark.parametrize("branches", [1, 4])
def test_batch(branches):
    import torch

    from pittpack_b200.batch import Batch

    grids = [(64, 32, 20, "PPNNDD"), (200, 60, 33, "PPDDDN"), (42, 36, 50, "PPNDDD"), (32, 64, 9, "NNPPDD"),
             (96, 50, 17, "PPDNND")]
    fs = [_rhs(*g[:3]) for g in grids]
    rhs = [torch.as_tensor(f).cuda() for f in fs]
    Ps = [torch.zeros(f.shape, dtype=torch.complex128, device="cuda") for f in fs]
    torch.cuda.synchronize()
    B = Batch([{"nx": nx, "ny": ny, "nz": nz, "bc": bc, "d_rhs": r.data_ptr(), "d_P": P.data_ptr()}
               for (nx, ny, nz, bc), r, P in zip(grids, rhs, Ps)], branches=branches, autotune=False)
    for _ in range(2):
        B.run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    B.close()
    for (nx, ny, nz, bc), f, P in zip(grids, fs, Ps):
        assert O.rel_l2(P.cpu().numpy(), O.solve(O.problem(nx, ny, nz, bc), f)) <= 1e-12, (nx, bc)


def _rank(rank, world, port, nx, ny, nz, bc, q):
    import torch
    import torch.distributed as dist

    from pittpack_b200.distributed import SlabPoisson

    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        with SlabPoisson(nx, ny, nz, bc) as S:
            q.put((rank, S.solve(_rhs(nx, ny, nz)[S.k0:S.k0 + S.nzl])))
    except Exception as e:  # reported to the parent
        q.put((rank, repr(e)))
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("nx,y", [(64, "NN"), (50, "DD")])
def test_slabs(nx, y):
    ny, nz, bc = 20, 13, "PP" + y + "DD"
    res = _run(_rank, 2, nx, ny, nz, bc)
    assert all(isinstance(r[1], np.ndarray) for r in res), res
    P = np.concatenate([r[1] for r in res], axis=0)
    assert O.rel_l2(P, O.solve(O.problem(nx, ny, nz, bc), _rhs(nx, ny, nz))) <= 1e-12
