"""gpe_itp over several iterations, whose normalisations are folded into the next one's
reads, against single iterations, each of which stores its normalised state."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


# each row shape and its kernels: interleaved (32, 16 and 8 cells a group), fixed rows, the
# grid-stride kernel of a single cell
@pytest.mark.parametrize("n", [2, 3, 18])
@pytest.mark.parametrize("name,C,dims", [("bcc", 3, (33, 4, 3)), ("bcc", 3, (40, 3, 2)), ("bcc", 5, (12, 3, 2)), ("fcc", 3, (35, 3, 2)),
                                         ("bcc", 1, (9, 8, 3)), ("fcc", 1, (6, 5, 4)), ("cube", 3, (20, 9, 7)),
                                         ("bcc", 3, (1, 1, 1))])
def test_iterations_equal_single_ones(gpu, name, C, dims, n):
    """Every bit: an iteration reads the same rounded values, normalised in memory or on the
    way in."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, precision=capi.FP32, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=100.0,
                         trap_lambda=(1.0, 1.1, 1.3), c0=120.0, c2=-7.0, c4=3.0, lattice=lat)
    psi = states.normalize(0.2 * states.random_state(capi.buffer_shape(lat, p), seed=5), lat, p)
    out = []
    for calls in ([n], [1] * n):
        with Stepper(lat, p) as s:
            s.upload(capi.PSI_ODD, psi)
            for k in calls:
                mu = s.itp(k)
            out.append((s.download(s.current), s.download(1 - s.current), s.download(capi.HPSI)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
