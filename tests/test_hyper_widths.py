"""The hyperbolic interleaved step's group widths on both sides of the state size that decides
them (9 MB a psi slot: rows of 24 and 40 cells in groups of 32 and 16 below, of 8 from there
on), bit for bit against the gather kernel."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,C,dims", [("bcc", 5, (24, 28, 27)), ("bcc", 5, (24, 28, 28)), ("bcc", 5, (40, 22, 21)),
                                         ("bcc", 5, (40, 22, 22)), ("bcc", 3, (23, 37, 36)), ("bcc", 3, (23, 37, 37)),
                                         ("c15", 3, (40, 8, 8)), ("c15", 3, (40, 9, 8)), ("c15", 5, (7, 16, 15)),
                                         ("c15", 5, (7, 16, 16))])
def test_widths_equal_gather(gpu, name, C, dims):
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, scheme=capi.SCHEME_HYPERBOLIC, precision=capi.FP32, dims=dims, block_scale=0.3, dt=2e-4,
                         trap_offset=100.0, c0=120.0, c2=-7.0, c4=3.0, sigma=0.01, lattice=lat)
    psi = 0.2 * states.random_state(capi.buffer_shape(lat, p), seed=9)
    out = []
    for kernel in (capi.KERNEL_GATHER, capi.KERNEL_INTERLEAVED):
        with Stepper(lat, p) as s:
            s.set_tuning(capi.TUNE_KERNEL, kernel)
            s.upload(capi.PSI_ODD, psi)
            s.start()
            s.step(17)
            out.append([s.download(k) for k in range(4)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
