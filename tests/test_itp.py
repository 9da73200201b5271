"""gpe_itp over several iterations: all but the last run without their H psi, the
normalisation folded into the next one's reads (FP32), from 16 iterations on in the
interleaved layout where that is the handle's kernel; every slot the call leaves is
compared with the FP64 oracle's loop of itp + normalise."""
import numpy as np
import pytest

from oracle import oracle
from spacetime_gb300 import capi, states
from spacetime_gb300.stepper import Stepper

pytestmark = pytest.mark.gpu

# (lattice, C, dims): the fixed-node kernel of each row shape, grids of one block and
# of one cell (the grid-stride kernel), groups of 32 and 16 cells, ragged rows
CASES = [("bcc", 3, (33, 4, 3)), ("bcc", 1, (9, 8, 3)), ("bcc", 5, (40, 3, 2)), ("fcc", 3, (35, 3, 2)),
         ("fcc", 1, (6, 5, 4)), ("cube", 3, (20, 9, 7)), ("c15", 3, (5, 2, 2)), ("a15", 5, (3, 2, 2)),
         ("bcc", 3, (1, 1, 1))]


@pytest.mark.parametrize("prec", [capi.FP64, capi.FP32])
@pytest.mark.parametrize("n", [1, 2, 5, 18])
@pytest.mark.parametrize("name,C,dims", CASES)
def test_itp_iterations(gpu, name, C, dims, n, prec):
    """FP64 to 1e-12 and FP32 to 2e-5 of the state's scale (the tolerances of the
    single-step parity tests: dt times the largest energy is 0.06 here, so an iterate's
    rounding shrinks from one iteration to the next instead of adding up)."""
    lat = capi.Lattice(name)
    p = capi.make_params(components=C, precision=prec, dims=dims, block_scale=0.3, dt=2e-4, trap_offset=100.0,
                         trap_lambda=(1.0, 1.1, 1.3), c0=120.0, c2=-7.0, c4=3.0, lattice=lat)
    psi = states.normalize(0.2 * states.random_state(capi.buffer_shape(lat, p), seed=5), lat, p)
    with Stepper(lat, p) as s:
        s.upload(capi.PSI_ODD, psi)
        mu = s.itp(n)
        assert s.current == (capi.PSI_EVEN if n % 2 else capi.PSI_ODD)
        other = capi.PSI_ODD if s.current == capi.PSI_EVEN else capi.PSI_EVEN
        got, got_old, got_h = s.download(s.current), s.download(other), s.download(capi.HPSI)
    cur, hp = psi.copy(), np.zeros_like(psi)
    for _ in range(n):
        old, cur = cur, np.zeros_like(psi)
        oracle.parabolic_step(lat, p, capi.make_fields(), 0.0, oracle.ITP, cur, old, hp)
        oracle.normalize(lat, p, cur)
    tol = 1e-12 if prec == capi.FP64 else 2e-5
    for a, b in ((got, cur), (got_old, old), (got_h, hp)):
        assert float(np.max(np.abs(a - b))) <= tol * float(np.max(np.abs(b)))
    mu_ref = float(np.sum(cur * hp)) * p.block_scale ** 3 * lat.volume
    assert mu == pytest.approx(mu_ref, rel=1e-11 if prec == capi.FP64 else 1e-5)
