"""The FP64 sweep's FP32 filter: decisions equal the oracle's FP64 formula bit
for bit where the filter's bound is wide or cannot hold (low and very high
temperatures, m far from unit length), at the edges of the list kernel's CTAs
and for every colouring.  No tolerance: the filter may only confirm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOMS = {
    "one_cell": dict(nx=1, ny=1),
    "cta_edge_127": dict(nx=127, ny=2, pbc_x=0),  # 64 cells of a colour per row: one CTA, one cell missing
    "cta_edge_258x1": dict(nx=258, ny=1, pbc_x=0),         # 129 cells of a colour: one past the CTA's 128
    "three_colours": dict(nx=15, ny=9),
    "thick": dict(nx=7, ny=5, nz=4, pbc_x=0, pbc_y=1),
    "fused_film": dict(nx=16, ny=12, sweep_engine=2),
}


def cfg(M, **kw):
    base = dict(nx=16, ny=16, nz=1, dx=1e-9, dy=1e-9, dz=0.8e-9, pbc_x=1, pbc_y=1, pbc_z=0, precision=64,
                randomseed=11, Bextx=0.02, Bexty=-0.01, Bextz=0.3, anisUx=0.1, anisUy=0.0, anisUz=1.0,
                sweep_engine=1)
    base.update(kw)
    if base["nz"] > 1 or base["nx"] % 2 and base["pbc_x"]:
        base["sweep_engine"] = 0
    return M.Config.defaults(**base)


@pytest.mark.parametrize("T", [0.5, 90.0, 1e7])
@pytest.mark.parametrize("scale", [1.0, 40.0])
@pytest.mark.parametrize("geom", sorted(GEOMS))
def test_decisions_equal_oracle(M, O, geom, scale, T):
    c = cfg(M, **GEOMS[geom])
    with M.Lattice(c) as lat:
        m0 = lat.get_m() * scale
        lat.set_m(m0)
        k = lat.tensor()
        lat.run_sweeps(T, 3, 0, 25)
        got = lat.get_m()
        accepted = lat.energy().accepted
    m = m0.copy()
    acc = O.sweeps(c, k, T, 3, 0, 25, m, demag_mode=1)
    assert accepted == acc
    assert np.array_equal(got, m)


def test_huge_and_non_finite_values_reach_the_formula(M, O):
    """Values beyond FP32's range, infinities and NaN: the filter is unsure and
    the FP64 formula decides, as in the oracle.  Without demag, so that a bad
    cell stays where it is."""
    c = cfg(M, nx=24, ny=10, cal_demag_flag=0)
    with M.Lattice(c) as lat:
        m0 = lat.get_m()
        for i, v in enumerate((1e39, -1e60, 1e-320, np.inf, -np.inf, np.nan)):
            m0[i % 3, 31 * i + 5] = v
        lat.set_m(m0)
        lat.run_sweeps(200.0, 1, 0, 12)
        got = lat.get_m()
        accepted = lat.energy().accepted
    m = m0.copy()
    acc = O.sweeps(c, None, 200.0, 1, 0, 12, m, demag_mode=1)
    assert accepted == acc
    assert np.array_equal(got, m, equal_nan=True)


def test_two_trials_per_thread_equal_single_lattice(M):
    """A launch large enough for two trials per thread (80 x 96 x 90 cells)."""
    cfgs = [cfg(M, nx=96, ny=90, randomseed=100 + r) for r in range(80)]
    with M.Batch(cfgs) as b:
        b.set_temperatures(np.full(80, 150.0))
        b.run_sweeps(0, 0, 3)
        got = [b.get_m(r) for r in (0, 41, 79)]
    for r, want in zip((0, 41, 79), got):
        with M.Lattice(cfgs[r]) as lat:
            lat.run_sweeps(150.0, 0, 0, 3)
            assert np.array_equal(lat.get_m(), want)
