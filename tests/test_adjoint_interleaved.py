"""The recorded run and its reverse in the interleaved layout (FP32 runs long enough for
the interleaved step kernel) against the FP64 adjoint, for every row shape and group
width, ragged rows, and the checkpoint strides where a state is a checkpoint, half of
one, or neither."""
import numpy as np
import pytest

from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu

SEED = np.array([0.7, -0.4, 0.2, -0.1, 0.3])


def _gradient(lat, prec, C, dims, n, stride, kernel, flags=0):
    p = capi.make_params(components=C, precision=prec, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=10.0,
                         trap_lambda=(1.0, 1.1, 1.3), c0=120.0, c2=-7.0, c4=3.0, alpha=2.0, flags=flags, lattice=lat)
    shape = capi.buffer_shape(lat, p)
    psi = states.normalize(states.random_state(shape, seed=3), lat, p).astype(np.float32).astype(np.float64)
    target = states.normalize(states.random_state(shape, seed=4) + 0.5 * psi, lat, p).astype(np.float32).astype(np.float64)
    fields = 0.5 * np.random.default_rng(5).standard_normal((n, 4))
    with Stepper(lat, p) as s:
        s.set_tuning(capi.TUNE_KERNEL, kernel)
        s.upload(capi.PSI_ODD, psi)
        out = s.adjoint_forward(fields, target, stride)
        g = s.adjoint_backward(SEED)
        g2 = s.adjoint_backward(SEED)   # again from the same record
        last, before = s.download(s.current), s.download(1 - s.current)
    assert np.array_equal(g, g2)
    return out, g, last, before


def _close(a, b, tol):
    return float(np.max(np.abs(a - b))) <= tol * float(np.max(np.abs(b)))


@pytest.mark.parametrize("name,C,dims", [("bcc", 3, (33, 3, 2)), ("bcc", 3, (40, 2, 3)), ("bcc", 3, (12, 4, 3)),
                                         ("fcc", 3, (35, 3, 2)), ("a15", 3, (5, 2, 2)), ("bcc", 1, (9, 3, 2)),
                                         ("bcc", 5, (34, 2, 2)), ("bcc", 3, (1, 1, 1))])
def test_interleaved_adjoint_against_fp64(gpu, name, C, dims):
    """FP32 storage and arithmetic over 18 steps against the FP64 adjoint: 2e-5 of the
    largest gradient and state (some 1e2 roundings of 6e-8)."""
    lat = capi.Lattice(name)
    flags = capi.FLAG_QUADRATIC_ZEEMAN | capi.FLAG_THREE_BODY_LOSS if C == 3 else capi.FLAG_THREE_BODY_LOSS
    ref = _gradient(lat, capi.FP64, C, dims, 18, 0, capi.KERNEL_GATHER, flags)
    got = _gradient(lat, capi.FP32, C, dims, 18, 0, capi.KERNEL_INTERLEAVED, flags)
    for a, b in zip(got, ref):
        assert _close(a, b, 2e-5)


@pytest.mark.parametrize("stride", [1, 2, 3, 5, 8, 16, 17, 18, 0])
def test_interleaved_adjoint_strides(gpu, stride):
    """Every stride gives the gradient, the numbers and the final pair of states of
    stride N bit for bit."""
    lat = capi.Lattice("bcc")
    ref = _gradient(lat, capi.FP32, 3, (24, 3, 2), 17, 17, capi.KERNEL_AUTO)
    got = _gradient(lat, capi.FP32, 3, (24, 3, 2), 17, stride, capi.KERNEL_AUTO)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


def test_one_handle_many_records(gpu):
    """One handle's records one after the other -- every state kept (no stride given), more
    of them, checkpoints, fewer states -- give what a handle of their own gives, bit for bit."""
    lat = capi.Lattice("bcc")
    p = capi.make_params(components=3, precision=capi.FP32, dims=(24, 3, 2), block_scale=0.3, dt=2e-4, trap_offset=10.0,
                         c0=120.0, c2=-7.0, lattice=lat)
    shape = capi.buffer_shape(lat, p)
    psi = states.normalize(states.random_state(shape, seed=3), lat, p)
    target = states.normalize(states.random_state(shape, seed=4), lat, p)

    def run(s, n, stride):
        fields = 0.5 * np.random.default_rng(n).standard_normal((n, 4))
        s.upload(capi.PSI_ODD, psi)
        out = s.adjoint_forward(fields, target, stride)
        return out, s.adjoint_backward(SEED), s.adjoint_backward(2 * SEED), s.download(s.current)

    records = [(17, 0), (40, 0), (40, 6), (19, 0), (7, 0), (18, 18), (40, 0)]
    with Stepper(lat, p) as s:
        got = [run(s, *r) for r in records]
    for (n, _), g in zip(records, got):
        with Stepper(lat, p) as s:
            want = run(s, n, 1)
        for a, b in zip(g, want):
            assert np.array_equal(a, b), n
