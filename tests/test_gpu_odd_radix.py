"""Transform lengths with prime factors 7 .. 31: every radix in rows and in
columns, in first and later stages, with few lines (a butterfly shared by
several threads) and many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [(7, 11), (13, 17), (19, 23), (29, 31), (77, 62), (341, 7), (7, 341), (31, 145)]
# a convolution's rounding error relative to the field's norm is a small multiple
# of eps log2(n); the direct R-point sums add up to R products each
TOL = {64: 1e-13, 32: 3e-6}


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("nx,ny", SIDES)
def test_field_of_odd_lengths_matches_direct_sum(M, O, nx, ny, prec):
    c = M.Config.defaults(nx=nx, ny=ny, nz=1, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=1, pbc_y=1, pbc_z=0, precision=prec,
                          randomseed=3, cal_demag_flag=1, use_random_init=1)
    with M.Lattice(c) as lat:
        lat.build_demag()
        m = lat.get_m()
        lat.compute_demag()
        got, k = lat.field(M.TERM_DEMAG), lat.tensor()
    want = c.ms * O.demag_direct(c, k, m)
    assert np.linalg.norm(got - want) <= TOL[prec] * np.linalg.norm(want)
