"""The staged vectorised Metropolis form (3) makes the scalar form's decisions
over enough trials to see the rounding of one product: two trials in 1e10 depend
on whether the second exchange product is rounded before it is added."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pbc,ny", [(2, 256), (0, 250)])
def test_band_form_decides_as_the_scalar_form(M, pbc, ny):
    R, sweeps = 64, 10000  # 4e10 trials: seven replicas of the periodic film differed with the product apart
    cfgs = [M.Config.defaults(nx=256, ny=ny, nz=1, pbc_x=pbc, pbc_y=pbc, pbc_z=0, precision=32, dz=0.8e-9, ms=1.6e6,
                              Aex=16e-12, Dind=6e-3, Ku1=2e6, Bextz=0.3, randomseed=r) for r in range(R)]
    got = []
    for form in (0, 3):
        with M.Batch(cfgs) as b:
            s = list(b.launch_shape())
            s[6] = form
            b.set_launch_shape(s)
            b.set_temperatures(np.geomspace(50, 1200, R))
            b.run_sweeps(0, 0, sweeps)
            got.append(([b.get_m(r) for r in range(R)], [o.accepted for o in b.energy()]))
    assert got[0][1] == got[1][1]
    assert all(np.array_equal(x, y) for x, y in zip(got[0][0], got[1][0]))
