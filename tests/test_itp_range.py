"""The chemical potential of gpe_itp where its products leave FP32's range."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


# block scales where psi and H psi are of ordinary size, where their products overflow FP32
# (psi 1e11, H psi 1e29) and where they vanish (1e-17, 1e-37)
@pytest.mark.parametrize("bs,dt", [(0.3, 2e-4), (1e-9, 1e-21), (1e10, 1e18)])
@pytest.mark.parametrize("name,C", [("bcc", 1), ("bcc", 3), ("fcc", 5)])
def test_chemical_potential_range(gpu, name, C, bs, dt):
    """Against a sum in extended precision over the stored psi and H psi: 1e-12 of the sum of
    magnitudes."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, precision=capi.FP32, dims=(6, 5, 4), block_scale=bs, dt=dt, trap_lambda=(0.0, 0.0, 0.0),
                         lattice=lat)
    psi = states.normalize(0.2 * states.random_state(capi.buffer_shape(lat, p), seed=5), lat, p)
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_ODD, psi)
        mu = s.itp(1)
        a, b = s.download(s.current).astype(np.longdouble), s.download(capi.HPSI).astype(np.longdouble)
    dv = np.longdouble(p.block_scale ** 3 * lat.volume)
    assert np.isfinite(a).all() and np.isfinite(b).all() and abs(b).max() > 0
    assert abs(mu - (a * b).sum() * dv) <= 1e-12 * abs(a * b).sum() * dv
