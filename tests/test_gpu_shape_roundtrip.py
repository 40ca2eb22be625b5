"""The launch shape a batch reports -- its default and the one the autotuner
chose -- is one that it accepts, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the pipelined column pass by default, the copying and in-place forms, the FP64
# passes, mixed radices, thick lattices with short and long z lines
BATCHES = [(32, 256, 32, 1, 24), (32, 64, 64, 1, 8), (32, 128, 128, 1, 24), (32, 64, 256, 1, 24), (32, 256, 256, 1, 8),
           (32, 20, 512, 1, 2), (32, 48, 48, 1, 4), (32, 64, 64, 4, 2), (32, 32, 32, 20, 2), (64, 256, 32, 1, 24),
           (64, 20, 64, 1, 8), (64, 128, 64, 1, 8), (64, 48, 40, 1, 4), (64, 32, 32, 3, 2)]


@pytest.mark.parametrize("prec,nx,ny,nz,R", BATCHES)
def test_reported_shapes_are_accepted(M, prec, nx, ny, nz, R):
    cfgs = [M.Config.defaults(nx=nx, ny=ny, nz=nz, pbc_x=1, pbc_y=1, pbc_z=0, precision=prec, randomseed=r,
                              Temperature_start=200.0) for r in range(R)]
    with M.Batch(cfgs) as a, M.Batch(cfgs) as b:
        default = list(a.launch_shape())
        a.set_launch_shape(default)
        a.autotune(4)
        tuned = list(a.launch_shape())
        assert 0 <= tuned[8] <= 3
        a.set_launch_shape(tuned)
        assert list(a.launch_shape()) == tuned
        a.run_sweeps(0, 0, 40)
        b.run_sweeps(0, 0, 40)
        assert all(np.array_equal(a.get_m(r), b.get_m(r)) for r in range(R))


@pytest.mark.parametrize("nx,ny,nz,R,rows", [(512, 48, 1, 1, 4), (1024, 16, 1, 1, 2), (512, 512, 1, 4, 8),
                                             (256, 48, 1, 1, 4)])
def test_long_lines_on_few_rows_spread_over_the_sms(M, nx, ny, nz, R, rows):
    """FP32 x passes of 512 and 1024 take half as many rows per CTA where full
    CTAs would not cover the SMs."""
    cfgs = [M.Config.defaults(nx=nx, ny=ny, nz=nz, pbc_x=1, pbc_y=1, pbc_z=0, precision=32) for _ in range(R)]
    with M.Batch(cfgs) as b:
        assert b.launch_shape()[0] == rows
