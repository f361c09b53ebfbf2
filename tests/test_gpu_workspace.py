"""What a handle keeps on the device: four buffers of a complex number per
point and its tables.  Padding columns of the spectrum fit beside a real one
for nothing; a complex one (periodic y) gets room for them where the memory is
there, and the request server stays within its budget either way."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

TABLES = 1 << 20  # what the server allows for them


def _rhs(nx, ny, nz):
    return np.random.default_rng(nx + ny + nz).uniform(-1, 1, (nz, ny, nx))


@pytest.mark.parametrize("nx,ny,nz,bc", [(100, 128, 128, "NNDDDD"), (500, 96, 64, "DDNDNN"), (150, 120, 100, "NDNNPP")])
def test_real_spectra_are_padded_for_nothing(nx, ny, nz, bc):
    import pittpack_b200 as pp

    with pp.make_Poisson(nx, ny, nz) as M:
        M.assignBoundary(bc)
        assert M.workspaceBytes() <= 64 * nx * ny * nz + TABLES


def _served(nx, ny, nz, bc, room):
    """One request through a server whose budget is the plain buffers, the
    tables and a share 'room' of the buffers: (status, P, pooled bytes, budget)."""
    import torch

    from pittpack_b200.batch import Server

    plain = 64 * nx * ny * nz
    budget = plain + TABLES + int(room * plain) + 4096
    S = Server(streams=1, hbm_fraction=budget / torch.cuda.mem_get_info()[0])
    try:
        P = np.zeros((nz, ny, nx), dtype=np.complex128)
        st, _, _ = S.wait(S.submit(nx, ny, nz, bc, _rhs(nx, ny, nz), P))
        return st, P, S.stats()["pool_bytes"], budget
    finally:
        S.close()


@pytest.mark.parametrize("room", [0.0, 0.02, 0.1])
@pytest.mark.parametrize("nx,ny,nz,bc", [(100, 128, 128, "NNPPDD"), (100, 128, 128, "NNDDDD"), (180, 96, 100, "DDPPNN"),
                                         (100, 128, 128, "PPPPDD")])
def test_server_keeps_its_budget(nx, ny, nz, bc, room):
    st, P, pool, budget = _served(nx, ny, nz, bc, room)
    assert st == 0
    # (the budget is a rounded fraction of the free memory)
    assert pool <= budget + 64, (pool, budget)
    assert O.rel_l2(P, O.solve(O.problem(nx, ny, nz, bc), _rhs(nx, ny, nz))) <= 1e-12
    if bc[2] == "P" and room > 0.07:
        assert pool >= 64 * nx * ny * nz + 2 * 16 * 4 * ny * nz  # by four columns, to the next multiple of 8
