"""gpe_observe and gpe_node_fields_reduce with FP64 node terms: the sums over columns of
cells (pairs of FP32 values for FP32 storage) against the FP64 oracle and against sums
in more than 64 bits, at the column lengths, row shapes and amplitudes where they can go
wrong, and what they make of empty and non-finite nodes."""
import math

import numpy as np
import pytest

from oracle import oracle
from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu

# (lattice, C, dims): rows of 4, 4 and 8, 6 entries; one cell, columns of one plane, of an odd
# number and longer than 64
CASES = [("bcc", 3, (1, 1, 1)), ("bcc", 3, (5, 3, 67)), ("bcc", 1, (4, 5, 9)), ("bcc", 5, (6, 2, 33)),
         ("fcc", 3, (3, 4, 11)), ("fcc", 5, (3, 2, 5)), ("cube", 3, (20, 9, 70)), ("cube", 1, (33, 3, 1)),
         ("c15", 1, (2, 2, 3)), ("c15", 5, (2, 1, 2)), ("a15", 3, (2, 3, 4)), ("z", 3, (2, 2, 3))]


def _params(lat, C, prec, dims, **kw):
    return capi.make_params(components=C, precision=prec, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=100.0,
                            trap_lambda=(1.0, 1.1, 1.3), c0=120.0, c2=-7.0, c4=3.0, lattice=lat, **kw)


def _state(lat, p, seed, amp=0.2):
    psi = amp * states.random_state(capi.buffer_shape(lat, p), seed=seed)
    return psi.astype(np.float32).astype(np.float64)


def _ramp(f):
    return capi.make_ramp(bq_segments=[(f.bq, 1e9, capi.RAMP_CONSTANT)], bb_segments=[(tuple(f.bb), 1e9, capi.RAMP_CONSTANT)])


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("amp", [1e-9, 0.2, 1e9])
@pytest.mark.parametrize("name,C,dims", CASES)
def test_observe_against_oracle(gpu, name, C, dims, amp, prec):
    """1e-12 of each number's scale (sums of at most 6e4 nodes' terms, each to 2^-47 at
    worst); amplitudes outside the pairs' range are summed in FP64."""
    lat = capi.Lattice(name)
    p = _params(lat, C, prec, dims, flags=capi.FLAG_QUADRUPOLE_OFFSET, quad_center=(0.1, -0.2, 0.05))
    psi = _state(lat, p, 61, amp)
    ramp = _ramp(capi.make_fields(bq=0.3, bb=(0.1, -0.2, 0.5)))
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_EVEN, psi)
        s.set_ramp(ramp, 0.0)
        got = s.observe(capi.PSI_EVEN, t=0.0)
    want = oracle.observe(lat, p, oracle.ramp_eval(ramp, 0.0), 0.0, psi)
    norm = want["norm"]
    box = 0.3 * max(d * w for d, w in zip(dims, lat.block_width))
    for k, scale in (("norm", norm), ("energy", abs(want["h_expect"]) + abs(want["energy"])), ("h_expect", abs(want["h_expect"])),
                     ("spin_norm", 2 * norm), ("max_abs", want["max_abs"])):
        assert abs(got[k] - want[k]) <= 1e-12 * scale, k
    for k, scale in (("magnetization", 2 * norm), ("com", box * norm)):
        assert np.max(np.abs(np.array(got[k]) - np.array(want[k]))) <= 1e-12 * scale, k


def test_sums_hold_64_bits(gpu):
    """FP32 storage: norm, centre of mass and spin against sums of the stored values
    without rounding (math.fsum of exact products).  1e-15: a few units in the last
    place, from the FP64 additions across threads and blocks."""
    lat = capi.Lattice("bcc")
    p = _params(lat, 3, capi.FP32, (12, 10, 14))
    psi = _state(lat, p, 3)
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_EVEN, psi)
        got = s.observe(capi.PSI_EVEN)
        dens = s.node_fields_reduce(capi.PSI_EVEN, capi.FIELD_DENSITY)[0]
    v = psi[1:-1, 1:-1, 1:-1]
    dv = p.block_scale ** 3 * lat.volume
    norm = math.fsum((v * v).ravel()) * dv   # squares of 24-bit values are exact in FP64
    assert abs(got["norm"] - norm) <= 1e-15 * norm and abs(dens - norm) <= 1e-15 * norm
    mz = math.fsum((v[..., 0, :] ** 2).ravel().tolist() + (-v[..., 2, :] ** 2).ravel().tolist()) * dv
    assert abs(got["magnetization"][2] - mz) <= 1e-15 * norm


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("amp", [1e-12, 1e-5, 0.2, 1e9])
@pytest.mark.parametrize("C", [1, 3, 5])
def test_field_sums_against_fields(gpu, C, amp, prec):
    """The integrated DENSITY and SPIN fields against numpy's integrals of the node
    fields (gpe_node_fields, FP64 per node): 1e-12 of the density's."""
    lat = capi.Lattice("bcc")
    p = _params(lat, C, prec, (7, 6, 5))
    dv = p.block_scale ** 3 * lat.volume
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_ODD, _state(lat, p, 8, amp))
        d = s.node_fields_reduce(capi.PSI_ODD, capi.FIELD_DENSITY)
        want = s.node_fields(capi.PSI_ODD, capi.FIELD_DENSITY).sum() * dv
        assert abs(d[0] - want) <= 1e-12 * want
        if C > 1:
            f = s.node_fields(capi.PSI_ODD, capi.FIELD_SPIN).reshape(-1, 5)
            got = s.node_fields_reduce(capi.PSI_ODD, capi.FIELD_SPIN)
            ref = np.array([f[:, 0].sum(), (f[:, 4] * f[:, 1]).sum(), (f[:, 4] * f[:, 2]).sum(), (f[:, 4] * f[:, 3]).sum(),
                            f[:, 4].sum()]) * dv
            scale = np.array([ref[0], ref[4], ref[4], np.abs(f[:, 4] * f[:, 3]).sum() * dv, ref[4]])
            assert np.all(np.abs(got - ref) <= 1e-12 * scale)


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
def test_empty_and_nonfinite_nodes(gpu, prec):
    """A node without density has no spin direction: the reduction over SPIN is NaN in
    its first three numbers, as the sum of the node fields is.  A NaN or an infinity
    anywhere in a column is found."""
    lat = capi.Lattice("bcc")
    p = _params(lat, 3, prec, (4, 3, 6))
    psi = _state(lat, p, 8)
    psi[3, 2, 2, 5] = 0.0
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_ODD, psi)
        r = s.node_fields_reduce(capi.PSI_ODD, capi.FIELD_SPIN)
        assert np.isnan(r[:3]).all() and np.isfinite(r[3:]).all()
        s.observe(capi.PSI_ODD)
        s.upload(capi.PSI_ODD, np.zeros_like(psi))
        o = s.observe(capi.PSI_ODD)
        assert o["norm"] == 0.0 and o["energy"] == 0.0 and o["max_abs"] == 0.0
        for bad in (math.nan, math.inf):
            psi[5, 3, 4, 11, 1, 1] = bad
            s.upload(capi.PSI_ODD, psi)
            with pytest.raises(capi.GpeError) as e:
                s.observe(capi.PSI_ODD)
            assert e.value.status == 5  # GPE_ERR_NONFINITE
