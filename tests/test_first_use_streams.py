"""Buffers that a handle allocates and clears on first use are ready for the stream of the
call that needs them, while other work holds up the default stream."""
import ctypes as C

import numpy as np
import pytest
import torch

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu

SEED = np.array([0.7, -0.4, 0.2, -0.1, 0.3])
BUSY = 400_000_000  # cycles of work on the default stream, a fifth of a second


def _stepper(lat, p, stream):
    s = Stepper(lat, p)
    if stream is not None:
        s.stream = C.c_void_p(stream.cuda_stream)
    return s


def _setup(prec):
    lat = capi.Lattice("bcc")
    p = capi.make_params(components=3, precision=prec, dims=(24, 3, 2), block_scale=0.3, dt=2e-4, trap_offset=10.0,
                         c0=120.0, c2=-7.0, lattice=lat)
    shape = capi.buffer_shape(lat, p)
    return lat, p, states.normalize(states.random_state(shape, seed=3), lat, p), states.normalize(
        states.random_state(shape, seed=4), lat, p)


@pytest.mark.parametrize("prec", [capi.FP32, capi.FP64])
def test_h_psi_of_the_first_iteration(gpu, prec):
    lat, p, psi, _ = _setup(prec)
    out = []
    for stream in (None, torch.cuda.Stream()):
        with _stepper(lat, p, stream) as s:
            s.upload(capi.PSI_ODD, psi)
            torch.cuda.synchronize()
            if stream is not None:
                torch.cuda._sleep(BUSY)
            mu = s.itp(1)
            torch.cuda.synchronize()
            out.append((mu, s.download(s.current), s.download(capi.HPSI)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert np.any(out[0][2])


@pytest.mark.parametrize("prec", [capi.FP32, capi.FP64])
def test_adjoint_records_on_a_stream(gpu, prec):
    """Every state kept, then checkpoints allocated by a handle that has its other buffers, then
    more states, each against a handle of its own on the default stream."""
    lat, p, psi, target = _setup(prec)
    records = [(17, 0), (17, 4), (40, 0), (40, 6)]

    def run(s, n, stride):
        fields = 0.5 * np.random.default_rng(n).standard_normal((n, 4))
        s.upload(capi.PSI_ODD, psi)
        out = s.adjoint_forward(fields, target, stride)
        return out, s.adjoint_backward(SEED), s.download(s.current)

    got = []
    with _stepper(lat, p, torch.cuda.Stream()) as s:
        for r in records:
            torch.cuda.synchronize()
            torch.cuda._sleep(BUSY)
            got.append(run(s, *r))
            torch.cuda.synchronize()
    for r, g in zip(records, got):
        with _stepper(lat, p, None) as s:
            want = run(s, *r)
        for a, b in zip(g, want):
            np.testing.assert_array_equal(a, b)
