"""The tile form of the Metropolis sweep (both colours in one launch) where its
CTAs cannot all start together: batches whose waves of CTAs end inside a replica,
fresh ones (the first launches of a process or a batch start unevenly), against
the scalar form; and runs of odd length, whose state lands in the other copy of
m, with tempering swaps and parts on streams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def batch(M, form, R, streams=1, **geom):
    cfgs = [M.Config.defaults(pbc_x=1, pbc_y=1, pbc_z=0, nz=1, precision=32, dz=0.8e-9, Dind=4e-3, Bextz=0.3,
                              randomseed=r, **geom) for r in range(R)]
    b = M.Batch(cfgs)
    s = list(b.launch_shape())
    s[6], s[9] = form, streams
    b.set_launch_shape(s)
    b.set_temperatures(np.geomspace(50, 900, R))
    return b


def states(b):
    return [b.get_m(r) for r in range(b.R)], [o.accepted for o in b.energy()]


@pytest.mark.parametrize("geom,R", [(dict(nx=256, ny=256), 64), (dict(nx=64, ny=64), 500),
                                    (dict(nx=512, ny=512), 9)])
def test_uneven_waves(M, geom, R):
    with batch(M, 0, R, **geom) as want:
        want.run_sweeps(0, 0, 200)
        m, acc = states(want)
    for _ in range(3):
        with batch(M, 1, R, **geom) as b:
            b.run_sweeps(0, 0, 200)
            got, acc1 = states(b)
        assert acc1 == acc
        assert all(np.array_equal(x, y) for x, y in zip(got, m))


@pytest.mark.parametrize("streams", [1, 3])
def test_odd_runs_and_swaps(M, streams):
    R, out = 12, []
    for form in (0, 1):
        with batch(M, form, R, streams, nx=64, ny=96) as b:
            b.set_ladders(np.arange(R, dtype=np.int32).reshape(2, -1), np.tile(np.geomspace(60, 400, 6), (2, 1)), 5, 11)
            for s0, n in ((0, 1), (1, 33), (34, 64), (98, 7)):
                b.run_sweeps(0, s0, n)
            out.append((states(b), [x.tolist() for x in b.ladder_state()], b.temperatures().tolist()))
    assert out[0][0][1] == out[1][0][1] and out[0][1:] == out[1][1:]
    assert all(np.array_equal(x, y) for x, y in zip(out[0][0][0], out[1][0][0]))
