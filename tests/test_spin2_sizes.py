"""The FP32 spin-2 gather step on both sides of the grid size from which it runs four blocks per
SM (2^20 nodes): the same states as the interleaved kernel's, bit for bit, and near FP64's."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu


# 1 044 900 and 1 069 200 nodes, 1 033 600 and 1 088 000
@pytest.mark.parametrize("name,dims", [("bcc", (43, 45, 45)), ("bcc", (44, 45, 45)), ("c15", (20, 19, 20)), ("c15", (20, 20, 20))])
def test_step_across_the_limit(gpu, name, dims):
    lat = capi.Lattice(name)
    kw = dict(components=5, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=10.0, c0=120.0, c2=-7.0, c4=3.0, lattice=lat)
    p = capi.make_params(precision=capi.FP32, **kw)
    psi = (0.2 * states.random_state(capi.buffer_shape(lat, p), seed=9)).astype(np.float32).astype(np.float64)
    out = []
    for prec, kernel in ((capi.FP32, capi.KERNEL_GATHER), (capi.FP32, capi.KERNEL_INTERLEAVED), (capi.FP64, capi.KERNEL_AUTO)):
        with Stepper(lat, capi.make_params(precision=prec, **kw)) as s:
            s.set_tuning(capi.TUNE_KERNEL, kernel)
            s.upload(capi.PSI_ODD, psi)
            s.start()
            s.step(2)
            out.append(s.download(s.current))
    np.testing.assert_array_equal(out[0], out[1])
    # some ten roundings of 6e-8 per step
    assert float(np.max(np.abs(out[0] - out[2]))) <= 2e-6 * float(np.max(np.abs(out[2])))


@pytest.mark.parametrize("dims", [(46, 46, 47), (47, 46, 47)])
def test_cube_step_across_the_limit(gpu, dims):
    """Rows of 6 entries: one block more per SM from 100000 nodes on (99 452 and 101 614)."""
    lat = capi.Lattice("cube")
    kw = dict(components=5, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=10.0, c0=120.0, c2=-7.0, c4=3.0, lattice=lat)
    psi = 0.2 * states.random_state(capi.buffer_shape(lat, capi.make_params(precision=capi.FP32, **kw)), seed=9)
    psi = psi.astype(np.float32).astype(np.float64)
    out = []
    for prec in (capi.FP32, capi.FP64):
        with Stepper(lat, capi.make_params(precision=prec, **kw)) as s:
            s.upload(capi.PSI_ODD, psi)
            s.start()
            s.step(2)
            out.append(s.download(s.current))
    assert float(np.max(np.abs(out[0] - out[1]))) <= 2e-6 * float(np.max(np.abs(out[1])))
