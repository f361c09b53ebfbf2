"""What a handle keeps on the device: four buffers of a complex number per
point and its tables.  Padding columns of the spectrum fit beside a real one
for nothing; a complex one (periodic y) gets room for them where the memory is
there."""
import pytest
pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

TABLES = 1 << 20


@pytest.mark.parametrize("nx,ny,nz,bc", [(100, 128, 128, "NNDDDD"), (500, 96, 64, "DDNDNN"), (150, 120, 100, "NDNNPP")])
def test_real_spectra_are_padded_for_nothing(nx, ny, nz, bc):
    import pittpack_b200 as pp

    with pp.make_Poisson(nx, ny, nz) as M:
        M.assignBoundary(bc)
        assert M.workspaceBytes() <= 64 * nx * ny * nz + TABLES
