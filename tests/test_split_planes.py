"""The split scheme's calls of 16 or more steps on planes of cells in a line against the same
steps in the handle's layout (the gather kernel on request), bit for bit."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


# rows that end on a group of 32 cells, before and after it; lines of less than a group
@pytest.mark.parametrize("name,dims", [("c15", (36, 2, 2)), ("c15", (2, 3, 2)), ("bcc", (32, 3, 2)), ("bcc", (33, 2, 3)),
                                       ("bcc", (31, 2, 2)), ("bcc", (12, 3, 3)), ("bcc", (8, 2, 2)), ("bcc227", (40, 3, 2)),
                                       ("bcc", (1, 1, 1)), ("bcc", (64, 2, 2))])
@pytest.mark.parametrize("n", [16, 17])
def test_planes_equal_handle_layout(gpu, name, dims, n):
    """psi and q after two calls (the second from the first's result) in every bit, halo
    cells included; the launches of a call: two per step and the layout changes."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=1, scheme=capi.SCHEME_SPLIT, precision=capi.FP32, dims=dims, block_scale=0.3, dt=1e-3,
                         trap_offset=3.0, trap_lambda=(1.0, 1.1, 1.3), c0=300.0, sigma=0.01, lattice=lat)
    psi = 0.2 * states.random_state(capi.buffer_shape(lat, p), seed=1)
    q = 0.2 * states.random_state(capi.buffer_shape(lat, p, True), seed=2)
    out = []
    for kernel in (capi.KERNEL_GATHER, capi.KERNEL_AUTO):
        with Stepper(lat, p) as s:
            s.set_tuning(capi.TUNE_KERNEL, kernel)
            s.upload(capi.PSI_EVEN, psi)
            s.upload(capi.Q_EVEN, q)
            s.start()
            n0 = s.launches
            s.step(n)
            assert s.launches - n0 == 2 * n + (4 if kernel == capi.KERNEL_AUTO else 0)
            s.step(n)
            out.append((s.download(capi.PSI_EVEN), s.download(capi.Q_EVEN)))
    for a, b in zip(*out):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
