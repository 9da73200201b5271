"""gpe_observe of FP32 states whose values leave the range of the sums in FP32 words: one
large value among ordinary ones, and states so small that their squares vanish.  Such a
state is summed in FP64."""
import numpy as np
import pytest

from oracle import oracle
from spacetime_gb300 import capi
from spacetime_gb300.stepper import Stepper
from test_observe_columns import _params, _ramp, _state

pytestmark = pytest.mark.gpu

CASES = [("bcc", 3, (5, 3, 7)), ("fcc", 5, (3, 2, 5)), ("c15", 1, (2, 2, 3)), ("cube", 3, (20, 9, 4))]


def _check(lat, p, psi):
    """1e-12 of each number's scale, as for states within the range."""
    ramp = _ramp(capi.make_fields(bq=0.3, bb=(0.1, -0.2, 0.5)))
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_EVEN, psi)
        s.set_ramp(ramp, 0.0)
        got = s.observe(capi.PSI_EVEN, t=0.0)
    want = oracle.observe(lat, p, oracle.ramp_eval(ramp, 0.0), 0.0, psi)
    norm = want["norm"]
    box = 0.3 * max(d * w for d, w in zip(p.dims, lat.block_width))
    for k, scale in (("norm", norm), ("energy", abs(want["h_expect"]) + abs(want["energy"])), ("h_expect", abs(want["h_expect"])),
                     ("spin_norm", 2 * norm), ("max_abs", want["max_abs"])):
        assert abs(got[k] - want[k]) <= 1e-12 * scale, k
    for k, scale in (("magnetization", 2 * norm), ("com", box * norm)):
        assert np.max(np.abs(np.array(got[k]) - np.array(want[k]))) <= 1e-12 * scale, k


@pytest.mark.parametrize("big", [1e10, 1e20, 1e30])
@pytest.mark.parametrize("name,C,dims", CASES)
def test_one_large_value(gpu, name, C, dims, big):
    lat = capi.Lattice(name)
    p = _params(lat, C, capi.FP32, dims)
    psi = _state(lat, p, 17)
    psi[2, 1, 2, 0, C - 1, 1] = np.float32(big)
    _check(lat, p, psi)


@pytest.mark.parametrize("amp", [1e-20, 1e-25, 1e-36])
@pytest.mark.parametrize("name,C,dims", CASES)
def test_vanishing_squares(gpu, name, C, dims, amp):
    lat = capi.Lattice(name)
    p = _params(lat, C, capi.FP32, dims)
    _check(lat, p, _state(lat, p, 17, amp))
