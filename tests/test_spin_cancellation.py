"""Spin sums of FP32 states whose spin cancels within a node -- nematic and cyclic spinors,
turned every way -- against extended precision.  The same spinor sits on every node, so that
a rounding is the same everywhere and does not average out."""
import numpy as np
import pytest

from spacetime_gb300 import capi
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu

SPINORS = {3: [(0, 1, 0)], 5: [(0, 0, 1, 0, 0), (0.5 ** 0.5, 0, 0, 0, 0.5 ** 0.5), ((1 / 3) ** 0.5, 0, 0, (2 / 3) ** 0.5, 0)]}


def _turned(C, zeta, seed):
    """The spinor under a seeded rotation and phase, as FP32 values."""
    F = (C - 1) // 2
    m = np.arange(F, -F - 1, -1)
    up = np.diag(np.sqrt(F * (F + 1) - m[1:] * (m[1:] + 1.0)), 1)
    fx, fy, fz = (up + up.T) / 2, (up - up.T) / 2j, np.diag(m)
    rng = np.random.default_rng(seed)
    n = rng.standard_normal(3)
    w, v = np.linalg.eigh(n[0] * fx + n[1] * fy + n[2] * fz)
    z = np.exp(1j * rng.uniform(0, 6)) * (v @ (np.exp(-1j * w * rng.uniform(1, 4)) * (v.conj().T @ np.array(zeta, complex))))
    return np.stack([z.real, z.imag], -1).astype(np.float32).astype(np.float64)


def _spin(z):
    """(F_x, F_y, F_z) of one spinor in extended precision."""
    c = z[:, 0].astype(np.longdouble) + 1j * z[:, 1].astype(np.longdouble)
    n = abs(c) ** 2
    if len(c) == 3:
        f = np.sqrt(np.longdouble(2)) * (c[0].conj() * c[1] + c[1].conj() * c[2])
        return np.array([f.real, f.imag, (z[0].astype(np.longdouble) ** 2 - z[2].astype(np.longdouble) ** 2).sum()])
    f = 2 * (c[0].conj() * c[1] + c[3].conj() * c[4]) + np.sqrt(np.longdouble(6)) * (c[1].conj() * c[2] + c[2].conj() * c[3])
    return np.array([f.real, f.imag, 2 * (n[0] - n[4]) + n[1] - n[3]])


@pytest.mark.parametrize("C,k", [(3, 0), (5, 0), (5, 1), (5, 2)])
def test_spin_of_unpolarised_states(gpu, C, k):
    """1e-15 of the density: FP64 terms round three partial sums of at most that size by 1.1e-16
    each (pairs of FP32 words: by 1.8e-15 to 7e-15)."""
    lat = capi.Lattice("bcc")
    p = capi.make_params(components=C, precision=capi.FP32, dims=(2, 2, 1), block_scale=0.3, dt=1e-4, lattice=lat)
    dv = np.longdouble(p.block_scale ** 3 * lat.volume) * 48
    with Stepper(lat, p) as s:
        for seed in range(40):
            z = _turned(C, SPINORS[C][k], seed)
            psi = np.zeros(capi.buffer_shape(lat, p))
            psi[1:-1, 1:-1, 1:-1] = z
            s.upload(capi.PSI_ODD, psi)
            got, fields = s.observe(capi.PSI_ODD), s.node_fields_reduce(capi.PSI_ODD, capi.FIELD_SPIN)
            rho, f = (z.astype(np.longdouble) ** 2).sum(), _spin(z)
            tol = 1e-15 * float(rho * dv)
            assert abs(got["spin_norm"] - np.sqrt((f * f).sum()) * dv) <= tol
            assert np.max(np.abs(np.array(got["magnetization"]) - f * dv)) <= tol
            if C == 3:  # F_x and F_y of the normalised spinor, F_z times the density
                g = f * np.array([1, 1, rho])
                want = np.append(np.sqrt((g * g).sum()), g) * dv
                assert np.max(np.abs(fields[:4] - want)) <= tol


@pytest.mark.parametrize("C,k", [(3, 0), (5, 0), (5, 1), (5, 2)])
def test_adjoint_numbers_of_unpolarised_states(gpu, C, k):
    """The recorded run's magnetisation, and Im <T|u> where T is near u, to 1e-15 of the density."""
    lat = capi.Lattice("bcc")
    # no couplings and a time step too short to move an FP32 value: the state stays as uploaded
    p = capi.make_params(components=C, precision=capi.FP32, dims=(2, 2, 1), block_scale=0.3, dt=1e-30, lattice=lat)
    dv = np.longdouble(p.block_scale ** 3 * lat.volume) * 48
    with Stepper(lat, p) as s:
        for seed in range(20):
            z, t = _turned(C, SPINORS[C][k], seed), _turned(C, SPINORS[C][k], seed) * np.float32(0.75)
            psi, target = np.zeros(capi.buffer_shape(lat, p)), np.zeros(capi.buffer_shape(lat, p))
            psi[1:-1, 1:-1, 1:-1], target[1:-1, 1:-1, 1:-1] = z, t
            s.upload(capi.PSI_ODD, psi)
            out = s.adjoint_forward(np.zeros((1, 4)), target)
            assert np.array_equal(s.download(s.current)[1, 1, 1, 0], z)
            t = t.astype(np.float32).astype(np.longdouble)
            rho = (z.astype(np.longdouble) ** 2).sum()
            im = (t[:, 0] * z[:, 1] - t[:, 1] * z[:, 0]).sum()
            want = np.append(im, _spin(z)) * dv
            assert np.max(np.abs(out[1:] - want)) <= 1e-15 * float(rho * dv)
