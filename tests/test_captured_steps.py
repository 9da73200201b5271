"""Steps recorded in CUDA graphs: a handle's calls captured by the caller (their launches overlap,
so the graph's edges are programmatic ones) and a batch's replays in the interleaved layout mixed
with members stepped on their own -- against the same steps without a graph."""
import ctypes as C

import numpy as np
import pytest
import torch

from spacetime_gb300 import capi, states
from spacetime_gb300.batch import Batch
from spacetime_gb300.stepper import Stepper
from test_batch import SPECS, _close, _compare, _pair

pytestmark = pytest.mark.gpu

# (lattice, C, dims, scheme, precision, kernel, steps of a call): gather, columns (FP64), the
# interleaved kernels with their layout changes, hyperbolic gather, split scheme in the handle's
# layout and on planes
CASES = [("bcc", 1, (9, 8, 7), 0, capi.FP32, capi.KERNEL_AUTO, 6), ("bcc", 3, (9, 8, 7), 0, capi.FP64, capi.KERNEL_AUTO, 4),
         ("fcc", 3, (33, 4, 3), 0, capi.FP32, capi.KERNEL_AUTO, 16), ("bcc", 5, (24, 4, 3), 0, capi.FP32, capi.KERNEL_AUTO, 18),
         ("bcc", 3, (9, 8, 7), 1, capi.FP32, capi.KERNEL_GATHER, 6), ("c15", 3, (7, 3, 2), 1, capi.FP32, capi.KERNEL_AUTO, 16),
         ("c15", 1, (5, 4, 3), 2, capi.FP32, capi.KERNEL_AUTO, 4), ("bcc", 1, (33, 4, 3), 2, capi.FP32, capi.KERNEL_AUTO, 16)]


def _stepper(case):
    name, comps, dims, scheme, prec, kernel, _ = case
    lat = capi.Lattice(name)
    p = capi.make_params(components=comps, scheme=scheme, precision=prec, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=100.0,
                         trap_lambda=(1.0, 1.1, 1.3), c0=120.0, c2=-7.0 if comps > 1 else 0.0, c4=3.0 if comps == 5 else 0.0,
                         sigma=0.01 if scheme else 0.0, lattice=lat)
    s = Stepper(lat, p)
    s.set_tuning(capi.TUNE_KERNEL, kernel)
    s.upload(capi.PSI_EVEN if scheme == 2 else capi.PSI_ODD, 0.2 * states.random_state(capi.buffer_shape(lat, p), seed=7))
    s.start()
    return s


def _slots(s, scheme):
    return [s.download(k) for k in ((0, 1, 2, 3) if scheme == 1 else (capi.PSI_EVEN, capi.Q_EVEN) if scheme == 2 else (0, 1))]


def _capture_and_replay(s, call, times):
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    s.stream = C.c_void_p(stream.cuda_stream)
    call()   # allocates what the call needs
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    with torch.cuda.stream(stream):
        for _ in range(times):
            graph.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize("case", CASES)
def test_captured_call_replayed(gpu, case):
    n = case[-1]
    a, b = _stepper(case), _stepper(case)
    try:
        _capture_and_replay(a, lambda: a.step(n), 3)
        for _ in range(4):
            b.step(n)
        for x, y in zip(_slots(a, case[3]), _slots(b, case[3])):
            np.testing.assert_array_equal(x, y)
    finally:
        _close([a, b])


@pytest.mark.parametrize("case", [CASES[0], CASES[2], CASES[1]])
def test_captured_imaginary_time_replayed(gpu, case):
    a, b = _stepper(case), _stepper(case)
    try:
        _capture_and_replay(a, lambda: a.itp(18, want_mu=False), 2)
        for _ in range(3):
            b.itp(18, want_mu=False)
        for k in (capi.PSI_EVEN, capi.PSI_ODD, capi.HPSI):
            np.testing.assert_array_equal(a.download(k), b.download(k))
    finally:
        _close([a, b])


def test_interleaved_batch_replays_between_single_steps(gpu):
    """12 captured steps are long enough for the interleaved layout (4 layout changes a member)."""
    prec = capi.FP32
    mem, ref = _pair(prec)
    stream = torch.cuda.Stream()
    sp = C.c_void_p(stream.cuda_stream)
    try:
        with Batch(mem) as b:
            b.stream = sp
            b.set_tuning(capi.BATCH_STEPS_PER_LAUNCH, 5)
            b.capture(12, sp)
            n_il = sum(1 for s in SPECS if s[1] == 3 and s[0] != "c15")
            for _ in range(2):
                before = b.launches
                b.replay()
                assert b.launches - before == 3 + 4 * n_il
            for m in mem:
                m.step(1)
            b.replay()
        for r in ref:
            r.step(37)
        _compare(mem, ref, prec)
    finally:
        _close(mem + ref)
