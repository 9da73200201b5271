"""The numbers of a recorded FP32 run (overlap with the target, magnetisation) for targets
and states so large or small that products of FP32 values overflow or vanish."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("amp,target_amp", [(0.2, 1.0), (0.2, 1e-36), (0.2, 1e20), (0.2, 1e30), (1e-12, 1e-25), (1e-25, 0.2),
                                            (1e-25, 1e-25), (1e-36, 1e30)])
@pytest.mark.parametrize("name,C", [("bcc", 1), ("bcc", 3), ("fcc", 5)])
def test_final_numbers(gpu, name, C, amp, target_amp):
    """Against sums in extended precision over the state left behind: 1e-12 of the sums of
    magnitudes (some 1e3 terms, each to 2^-47 at worst)."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, precision=capi.FP32, dims=(6, 5, 4), block_scale=0.3, dt=2e-4, trap_offset=10.0,
                         c0=120.0, c2=-7.0, c4=3.0, lattice=lat)
    shape = capi.buffer_shape(lat, p)
    psi = amp * states.random_state(shape, seed=3)
    target = (target_amp * states.random_state(shape, seed=4)).astype(np.float32).astype(np.float64)
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_ODD, psi)
        out = s.adjoint_forward(np.zeros((2, 4)), target)
        last = s.download(s.current)
    inner = (slice(1, -1),) * 3
    dv = np.longdouble(p.block_scale ** 3 * lat.volume)
    u, t = (v[inner].astype(np.longdouble) for v in (last, target))
    u, t = u[..., 0] + 1j * u[..., 1], t[..., 0] + 1j * t[..., 1]
    overlap = (t.conj() * u).sum() * dv
    assert abs(out[0] + 1j * out[1] - overlap) <= 1e-12 * (abs(t) * abs(u)).sum() * dv
    if C > 1:
        n = abs(u) ** 2
        if C == 3:
            across = np.sqrt(np.longdouble(2)) * (u[..., 0].conj() * u[..., 1] + u[..., 1].conj() * u[..., 2])
            along = n[..., 0] - n[..., 2]
        else:
            across = (2 * (u[..., 0].conj() * u[..., 1] + u[..., 3].conj() * u[..., 4])
                      + np.sqrt(np.longdouble(6)) * (u[..., 1].conj() * u[..., 2] + u[..., 2].conj() * u[..., 3]))
            along = 2 * (n[..., 0] - n[..., 4]) + n[..., 1] - n[..., 3]
        want = np.array([across.real.sum(), across.imag.sum(), along.sum()]) * dv
        assert np.max(np.abs(out[2:] - want)) <= 1e-12 * 2 * n.sum() * dv
