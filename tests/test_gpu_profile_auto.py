"""mmc_profile_fused on films that AUTO runs on the pass kernels: the film engine
is set up for the call, its sweeps are the handle's sweeps, and the handle goes
on with its own engine."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n", [(32, 64), (64, 32)])
def test_profile_of_an_auto_film(M, prec, n):
    c = M.Config.defaults(nx=n, ny=n, nz=1, pbc_x=1, pbc_y=1, pbc_z=0, precision=prec, randomseed=9, Bextz=0.3)
    with M.Lattice(c) as a, M.Lattice(c) as b:
        assert a.engine() == (M.ENGINE_KERNELS, 0, 0)
        st = a.profile_fused(150.0, 1, 0, 17).astype(np.int64)
        assert (np.diff(st[:, :, 0], axis=1) >= 0).all() and st[0, 0, 0] > 0
        assert a.engine()[0] == M.ENGINE_KERNELS and a.engine()[2] > 0
        b.run_sweeps(150.0, 1, 0, 17)
        assert np.array_equal(a.get_m(), b.get_m())
        a.run_sweeps(150.0, 1, 17, 70)
        b.run_sweeps(150.0, 1, 17, 70)
        assert np.array_equal(a.get_m(), b.get_m())
        assert a.energy().as_dict() == b.energy().as_dict()


def test_profile_is_refused_where_the_engine_cannot_run(M):
    c = M.Config.defaults(nx=64, ny=64, nz=1, pbc_x=1, pbc_y=1, pbc_z=0, precision=32)
    for other in (c.copy(sweep_engine=M.ENGINE_KERNELS), c.copy(nx=15, pbc_x=0), c.copy(nz=2)):
        with M.Lattice(other) as lat, pytest.raises(M.MmcError) as ei:
            lat.profile_fused(150.0, 0, 0, 4)
        assert ei.value.status == M.ERR_STATE
