"""The pass kernels and the row kernel with and without the stages of radix 7
and above: a length of radices 2 to 5 in one axis and an odd one in the other,
either way round, against the direct sum; and row-kernel sweeps against the
pass kernels'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [(48, 60), (100, 27), (75, 80), (48, 28), (28, 48), (20, 62), (44, 32), (32, 44)]
# a convolution's rounding error relative to the field's norm is a small multiple
# of eps log2(n); the direct R-point sums add up to R products each
TOL = {64: 1e-13, 32: 3e-6}


def cfg(M, nx, ny, prec, **kw):
    return M.Config.defaults(nx=nx, ny=ny, nz=1, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=1, pbc_y=1, pbc_z=0,
                             precision=prec, randomseed=3, **kw)


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("nx,ny", SIDES)
def test_field_matches_direct_sum(M, O, nx, ny, prec):
    c = cfg(M, nx, ny, prec)
    with M.Lattice(c) as lat:
        lat.build_demag()
        m = lat.get_m()
        lat.compute_demag()
        got, k = lat.field(M.TERM_DEMAG), lat.tensor()
    want = c.ms * O.demag_direct(c, k, m)
    assert np.linalg.norm(got - want) <= TOL[prec] * np.linalg.norm(want)


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("nx", [28, 44, 48, 60, 64])
def test_row_kernel_sweeps_equal_pass_kernels(M, nx, prec):
    cfgs = [cfg(M, nx, 36, prec, Temperature_start=150.0).copy(randomseed=r) for r in range(3)]
    with M.Batch(cfgs) as a, M.Batch(cfgs) as b:
        s = list(a.launch_shape())
        s[5], s[6] = 0, 0
        a.set_launch_shape(s)
        s[5] = 4
        b.set_launch_shape(s)
        a.run_sweeps(0, 0, 40)
        b.run_sweeps(0, 0, 40)
        assert all(np.array_equal(a.get_m(r), b.get_m(r)) for r in range(3))
