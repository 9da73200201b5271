"""The hyperbolic interleaved step with both edges of a node loaded together, and one after the
other (spin-1 in groups of 8 cells from 9 MB a psi slot on), bit for bit against the gather
kernel: every group width, the smallest grids, both sides of the line."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,C,dims", [("bcc", 3, (8, 62, 63)), ("bcc", 3, (8, 63, 63)), ("bcc", 3, (6, 6, 6)), ("bcc", 3, (1, 1, 1)),
                                         ("bcc", 3, (10, 9, 3)), ("bcc", 3, (33, 5, 4)), ("bcc", 1, (8, 63, 63)), ("bcc", 1, (17, 3, 5)),
                                         ("c15", 3, (7, 20, 19)), ("c15", 3, (7, 20, 20)), ("c15", 1, (5, 5, 5)), ("c15", 1, (31, 2, 3)),
                                         ("bcc227", 3, (8, 3, 2)), ("bcc227", 1, (40, 2, 2))])
def test_edges_equal_gather(gpu, name, C, dims):
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, scheme=capi.SCHEME_HYPERBOLIC, precision=capi.FP32, dims=dims, block_scale=0.3, dt=2e-4,
                         trap_offset=100.0, c0=120.0, c2=-7.0 if C > 1 else 0.0, sigma=0.01, lattice=lat)
    psi = 0.2 * states.random_state(capi.buffer_shape(lat, p), seed=11)
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
