"""The interleaved layout's group widths (32, 16 or 8 cells, chosen by the row length):
rows that end on a group's edge, one cell before and after it, and inside it, bit for
bit against the gather kernels."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


# widths chosen: X = 1..8 -> 8, 12 -> 16, 23..25 -> 8 / 8 / 32, 31..32 -> 32, 40 -> 8, 41 -> 16, 48 -> 16, 72 -> 16 (8 for C = 5)
@pytest.mark.parametrize("X", [1, 7, 8, 12, 23, 24, 25, 31, 32, 40, 41, 48, 72])
@pytest.mark.parametrize("name,C,scheme", [("bcc", 3, 0), ("fcc", 3, 0), ("bcc", 5, 0), ("bcc", 5, 1), ("c15", 3, 1)])
def test_widths_equal_gather(gpu, name, C, scheme, X):
    """18 steps leave every slot bit for bit as the gather kernel does (both kernels
    share their arithmetic, written out in explicit multiply-adds)."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, scheme=scheme, precision=capi.FP32, dims=(X, 3, 2), block_scale=0.3, dt=2e-4,
                         trap_offset=100.0, c0=120.0, c2=-7.0, c4=3.0, sigma=0.01 if scheme else 0.0, lattice=lat)
    psi = 0.2 * states.random_state(capi.buffer_shape(lat, p), seed=9)
    out = []
    for kernel in (capi.KERNEL_GATHER, capi.KERNEL_INTERLEAVED):
        with Stepper(lat, p) as s:
            s.set_tuning(capi.TUNE_KERNEL, kernel)
            s.upload(capi.PSI_ODD, psi)
            s.start()
            s.step(18)
            out.append([s.download(k) for k in ((0, 1, 2, 3) if scheme else (0, 1))])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
