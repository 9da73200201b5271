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


@pytest.mark.parametrize("name,C,dims", [("bcc", 1, (12, 13, 14)), ("bcc", 3, (13, 12, 15)), ("bcc", 5, (12, 12, 13)),
                                         ("c15", 3, (4, 5, 6))])
def test_sums_of_one_sign_have_no_bias(gpu, name, C, dims):
    """Norm, centre of mass and spin against sums in extended precision over eight clouds: what
    is left is the rounding of the sums' last FP64 additions and of the product with the cell
    volume, 2e-16 at most each time and of either sign (a bias of the pairs' low words, whose
    squares round down more often than up, is 3e-16 to 8e-16)."""
    lat = capi.Lattice(name)
    p = _params(lat, C, capi.FP32, dims)
    wide = np.longdouble
    dv = wide(p.block_scale * p.block_scale * p.block_scale * lat.volume)
    inner = (slice(1, -1),) * 3
    errors = []
    with Stepper(lat, p) as s:
        for seed in range(8):
            rng = np.random.default_rng(seed)
            psi = np.zeros(capi.buffer_shape(lat, p))
            shape = psi[inner].shape[:-1]
            # densities of a cloud from its edge to its middle, every node's phases its own
            phase = rng.uniform(-np.pi, np.pi, shape)
            psi[inner] = 0.07 * np.sqrt(rng.uniform(0, 1, shape))[..., None] * np.stack([np.cos(phase), np.sin(phase)], -1)
            psi = psi.astype(np.float32).astype(np.float64)
            s.upload(capi.PSI_EVEN, psi)
            got = s.observe(capi.PSI_EVEN)
            re, im = psi[inner][..., 0].astype(wide), psi[inner][..., 1].astype(wide)
            n = re * re + im * im
            x = wide(p.p0[0]) + wide(p.block_scale) * (np.arange(dims[0]).astype(wide)[:, None] * wide(lat.block_width[0])
                                                       + lat.pos[:, 0].astype(wide))
            norm, com = n.sum() * dv, (n.sum(-1) * x).sum() * dv
            e = [(wide(got["norm"]) - norm) / norm, (wide(got["com"][0]) - com) / ((n.sum(-1) * abs(x)).sum() * dv)]
            if C > 1:
                def pair(a, b):
                    return np.stack([re[..., a] * re[..., b] + im[..., a] * im[..., b],
                                     re[..., a] * im[..., b] - im[..., a] * re[..., b]])
                if C == 3:
                    across, along = np.sqrt(wide(2)) * (pair(0, 1) + pair(1, 2)), n[..., 0] - n[..., 2]
                else:
                    across = 2 * (pair(0, 1) + pair(3, 4)) + np.sqrt(wide(6)) * (pair(1, 2) + pair(2, 3))
                    along = 2 * (n[..., 0] - n[..., 4]) + n[..., 1] - n[..., 3]
                size = np.sqrt((across ** 2).sum(0) + along ** 2).sum() * dv
                e.append((wide(got["spin_norm"]) - size) / size)
            errors.append([float(v) for v in e])
    assert np.all(np.abs(np.mean(errors, axis=0)) <= 2e-16), np.mean(errors, axis=0)
