"""The FP32 pass kernels round alike: the demag field that the last sweep left
behind is the same bit for bit from the film engine's transforms and from the
x passes and the pipelined column pass, and runs on colour-split rows leave m
and h as runs in the natural order do."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cfg(M, **kw):
    base = dict(nx=64, ny=64, nz=1, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=1, pbc_y=1, pbc_z=0, precision=32,
                randomseed=5, Bextz=0.3, Dind=4e-3)
    base.update(kw)
    return M.Config.defaults(**base)


# every (x, y) transform length of the passes; open and odd sides (cropped rows,
# zero-filled columns, a last tile of one column, odd row lengths)
FILMS = [dict(nx=32, ny=64), dict(nx=64, ny=32), dict(nx=128, ny=128), dict(nx=256, ny=256), dict(nx=64, ny=256),
         dict(nx=256, ny=64), dict(nx=20, ny=89, pbc_x=0, pbc_y=0), dict(nx=124, ny=12, pbc_x=0, pbc_y=0),
         dict(nx=100, ny=33, pbc_x=0, pbc_y=0), dict(nx=20, ny=128, pbc_x=0)]


@pytest.mark.parametrize("film", FILMS, ids=lambda f: "x".join(str(f[k]) for k in ("nx", "ny")))
def test_sweep_field_equals_film_engine(M, film):
    c = cfg(M, **film)
    with M.Lattice(c.copy(sweep_engine=M.ENGINE_KERNELS)) as a, M.Lattice(c.copy(sweep_engine=M.ENGINE_FUSED)) as b:
        a.run_sweeps(150.0, 2, 0, 9)
        b.run_sweeps(150.0, 2, 0, 9)
        assert np.array_equal(a.get_m(), b.get_m())
        assert np.array_equal(a.field(M.TERM_DEMAG), b.field(M.TERM_DEMAG))


@pytest.mark.parametrize("R", [1, 2, 9, 40])
def test_batched_columns_equal_single_lattice(M, R):
    """Chunks of the pipelined column pass that span tiles and replicas."""
    cfgs = [cfg(M, nx=128, ny=64, randomseed=50 + r) for r in range(R)]
    with M.Batch(cfgs) as b:
        assert b.launch_shape()[8] == 2
        b.set_temperatures(np.full(R, 120.0))
        b.run_sweeps(0, 0, 20)
        got = [b.get_m(r) for r in (0, R - 1)]
    for r, want in zip((0, R - 1), got):
        with M.Lattice(cfgs[r].copy(sweep_engine=M.ENGINE_FUSED)) as lat:
            lat.run_sweeps(120.0, 0, 0, 20)
            assert np.array_equal(lat.get_m(), want)


SPLIT = [dict(nx=512, ny=256, nz=4), dict(nx=8, ny=512, nz=128, pbc_x=0, pbc_z=1),
         dict(nx=260, ny=512, nz=4, pbc_x=0)]


@pytest.mark.parametrize("geom", SPLIT, ids=["periodic", "narrow_open_x", "open_x"])
def test_split_rows_leave_m_and_h_in_order(M, geom):
    """16 sweeps and more run on colour-split rows; in pieces of fewer they do not."""
    c = cfg(M, **geom)
    with M.Lattice(c) as a, M.Lattice(c) as b:
        a.run_sweeps(90.0, 1, 0, 18)
        for s0 in (0, 9):
            b.run_sweeps(90.0, 1, s0, 9)
        assert np.array_equal(a.get_m(), b.get_m())
        assert np.array_equal(a.field(M.TERM_DEMAG), b.field(M.TERM_DEMAG))
        assert a.energy().accepted == b.energy().accepted


def test_stopped_run_restores_the_row_order(M):
    """A stop request in the middle of a run: m is left in its natural order
    (unit vectors of which a zero-temperature-like energy can be evaluated), so
    a second lattice given that m continues identically."""
    cfgs = [cfg(M, nx=256, ny=256, randomseed=r) for r in range(8)]
    with M.Batch(cfgs) as b, M.Batch(cfgs) as d:
        assert b.launch_shape()[6] == 2
        b.build_demag()
        threading.Timer(0.3, lambda: M.lib().mmc_batch_request_stop(b.h)).start()
        with pytest.raises(M.MmcError) as ei:
            b.run_sweeps(0, 0, 10 ** 7)
        assert ei.value.status == M.ERR_INTERRUPTED
        for r in range(8):
            d.set_m(r, b.get_m(r))
        eb, ed = b.energy(), d.energy()
        # neighbours in the wrong places would change the exchange energy by its own size
        assert [o.e_total for o in eb] == [o.e_total for o in ed]
        b.run_sweeps(1, 0, 24)
        d.run_sweeps(1, 0, 24)
        assert all(np.array_equal(b.get_m(r), d.get_m(r)) for r in range(8))
        assert all(o.e_exchange < 0.8 * ref.e_exchange for o, ref in zip(b.energy(), _random_energies(M, cfgs)))


def _random_energies(M, cfgs):
    with M.Batch(cfgs) as b:
        return b.energy()
