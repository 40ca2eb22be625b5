"""Batches of thick lattices on colour-split rows: runs of 16 sweeps and more
against the same sweeps in shorter pieces, which stay in the natural order, with
replicas in parts on streams, with tempering swaps (whose energies are read from
split rows), and through the change of a run's order at both ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOMS = [dict(nx=64, ny=64, nz=4, pbc_x=1, pbc_y=1, pbc_z=0), dict(nx=64, ny=48, nz=2, pbc_x=0, pbc_y=1, pbc_z=1),
         dict(nx=60, ny=31, nz=3, pbc_x=0, pbc_y=0, pbc_z=0)]


def batch(M, geom, R, streams):
    cfgs = [M.Config.defaults(precision=32, dz=0.8e-9, Dind=3e-3, Bextz=0.2, randomseed=70 + r, **geom)
            for r in range(R)]
    b = M.Batch(cfgs)
    s = list(b.launch_shape())
    s[6], s[9] = 2, streams
    b.set_launch_shape(s)
    return b


def result(b):
    o = b.energy()
    return [b.get_m(r) for r in range(b.R)], [[e.e_total, e.e_demag, e.accepted] for e in o]


@pytest.mark.parametrize("streams", [1, 3])
@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: "x".join(str(g[k]) for k in ("nx", "ny", "nz")))
@pytest.mark.parametrize("swaps", [False, True])
def test_split_runs_equal_short_pieces(M, geom, streams, swaps):
    R, out = 6, []
    T = np.geomspace(60.0, 500.0, 3)
    for pieces in ([96, 20], [12] * 8 + [12, 8]):
        with batch(M, geom, R, streams) as b:
            if swaps:
                b.set_ladders(np.arange(R, dtype=np.int32).reshape(2, -1), np.tile(T, (2, 1)), 4, 5)
            else:
                b.set_temperatures(np.geomspace(50.0, 600.0, R))
            s0 = 0
            for n in pieces:
                b.run_sweeps(0, s0, n)
                s0 += n
            m, obs = result(b)
            out.append((m, obs, [x.tolist() for x in b.ladder_state()] if swaps else None, b.temperatures().tolist()))
    assert out[0][1:] == out[1][1:]
    assert all(np.array_equal(x, y) for x, y in zip(out[0][0], out[1][0]))
    if swaps:
        assert out[0][2][1][1] > 0  # some swaps were accepted
