"""FP64 fields do not depend on the launch shape: the pass kernels of
power-of-two lengths spread a line over more threads where there are few lines,
and a film alone, in a batch, and in a part of the batch on a stream of its own
(the graphs of a long run, with one stream for the sweeps that are left) have
the same demag energy bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def energies(o):
    return [o.e_total, o.e_exchange, o.e_dmi, o.e_anisotropy, o.e_zeeman, o.e_demag, o.accepted]


# batches that take the other thread count than the single lattice in the x
# passes, the column passes or both; every length of both counts
@pytest.mark.parametrize("nx,ny,nz,R", [(64, 64, 1, 32), (32, 32, 1, 64), (128, 128, 1, 8), (32, 256, 1, 16),
                                        (256, 32, 1, 24), (20, 50, 1, 40), (64, 128, 3, 6)])
@pytest.mark.parametrize("streams", [1, 4])
def test_batch_equals_single_lattices(M, nx, ny, nz, R, streams):
    cfgs = [M.Config.defaults(nx=nx, ny=ny, nz=nz, pbc_x=int(nx != 20), pbc_y=int(ny != 50), pbc_z=0, precision=64,
                              dz=0.8e-9, Dind=4e-3, randomseed=30 + r) for r in range(R)]
    with M.Batch(cfgs) as b:
        shape = list(b.launch_shape())
        shape[9] = streams
        b.set_launch_shape(shape)
        start = [energies(o) for o in b.energy()]
        b.set_temperatures(np.full(R, 120.0))
        b.run_sweeps(0, 0, 40)  # a graph of 32 sweeps and 8 more
        end = [energies(o) for o in b.energy()]
        m = [b.get_m(r) for r in range(R)]
    for r in (0, R // 2, R - 1):
        with M.Lattice(cfgs[r].copy(sweep_engine=M.ENGINE_KERNELS)) as lat:
            assert energies(lat.energy()) == start[r]
            lat.run_sweeps(120.0, 0, 0, 40)
            assert energies(lat.energy()) == end[r]
            assert np.array_equal(lat.get_m(), m[r])
