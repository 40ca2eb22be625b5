"""mmc_demag_apply with caller scratch on any boundary of a complex value: a
buffer carved out of an arena at an 8-byte offset gives the aligned buffer's
field bit for bit at every length of the pipelined column pass (whose copies
are of 16 bytes) and beside them; anything less aligned is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILMS = [(20, 32, 1), (64, 64, 1), (16, 128, 1), (128, 256, 1), (20, 17, 0), (33, 100, 0), (48, 96, 1), (24, 512, 1)]


def field(torch, lat, m, offset):
    nb = lat.demag_scratch_bytes()
    arena = torch.zeros(nb + 64, dtype=torch.uint8, device="cuda")
    base = (-arena.data_ptr()) % 16 + offset
    h = torch.zeros_like(m)
    torch.cuda.synchronize()
    lat.demag_apply(m.data_ptr(), h.data_ptr(), arena.data_ptr() + base, nb, None)
    torch.cuda.synchronize()
    assert not arena[:base].any() and not arena[base + nb:].any()
    return h.cpu().numpy()


@pytest.mark.parametrize("nx,ny,pbc", FILMS)
def test_scratch_on_8_bytes(M, nx, ny, pbc):
    torch = pytest.importorskip("torch")
    c = M.Config.defaults(nx=nx, ny=ny, nz=1, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=pbc, pbc_y=pbc, pbc_z=0,
                          precision=32, randomseed=4)
    with M.Lattice(c) as lat:
        lat.build_demag()
        m = torch.tensor(lat.get_m(), dtype=torch.float32, device="cuda").contiguous()
        want = field(torch, lat, m, 0)
        assert np.abs(want).max() > 0
        assert np.array_equal(field(torch, lat, m, 8), want)


@pytest.mark.parametrize("prec,offset", [(32, 4), (64, 8)])
def test_less_aligned_scratch_is_refused(M, prec, offset):
    torch = pytest.importorskip("torch")
    c = M.Config.defaults(nx=16, ny=32, nz=1, pbc_x=1, pbc_y=1, pbc_z=0, precision=prec, randomseed=4)
    with M.Lattice(c) as lat:
        nb = lat.demag_scratch_bytes()
        arena = torch.zeros(nb + 64, dtype=torch.uint8, device="cuda")
        with pytest.raises(M.MmcError) as ei:  # refused on the host, before any launch
            lat.demag_apply(arena.data_ptr(), arena.data_ptr(), arena.data_ptr() + offset, nb, None)
        assert ei.value.status == M.ERR_INVALID
