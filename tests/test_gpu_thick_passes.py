"""Thick lattices: the one-direction y passes at every warp-shaped length (first
and last tile partly empty) and the short-line z pass at every length up to 16,
against the direct sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# y lengths 32 .. 1024 (periodic) and 32 (open, 13 -> 25 -> 32); z lengths 3 .. 15
SHAPES = [(34, 32, 2, 1), (16, 64, 3, 1), (10, 128, 4, 1), (6, 256, 5, 1), (4, 512, 2, 1), (4, 1024, 2, 1),
          (9, 13, 6, 0), (5, 8, 7, 0), (12, 10, 8, 0)]
# a convolution's rounding error relative to the field's norm is a small multiple
# of eps log2(n)
TOL = {64: 1e-13, 32: 2e-6}


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("nx,ny,nz,pbc", SHAPES)
def test_thick_field_matches_direct_sum(M, O, nx, ny, nz, pbc, prec):
    c = M.Config.defaults(nx=nx, ny=ny, nz=nz, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=pbc, pbc_y=pbc, pbc_z=0,
                          precision=prec, randomseed=3, cal_demag_flag=1, use_random_init=1)
    with M.Lattice(c) as lat:
        lat.build_demag()
        m = lat.get_m()
        lat.compute_demag()
        got, k = lat.field(M.TERM_DEMAG), lat.tensor()
    want = c.ms * O.demag_direct(c, k, m)
    assert np.linalg.norm(got - want) <= TOL[prec] * np.linalg.norm(want)
