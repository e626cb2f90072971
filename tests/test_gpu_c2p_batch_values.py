"""Every state of a con2prim batch, beyond one pass of the capped grid too: repeated
states convert to the same bits wherever they sit, and the first copies to the
oracle's values."""
import numpy as np
import pytest
import torch

import oracle as O
from states import make_c2p_batch

pytestmark = pytest.mark.gpu

CFG = dict(GAMMA=4.0 / 3.0, P_MAX=1e3, V_MAX=0.9999, N_PASSIVE=0, PASSIVE_OFFSET=9)
M = 4999
# within the first pass of 148 * 32 blocks of 128, at its end, and well into a second
COUNTS = [M, 148 * 32 * 128 + 1, 148 * 32 * 128 + 3 * M]


def _conserved(n):
    """Jet-like states with the field across the velocity (one root), repeated."""
    q = make_c2p_batch(5, M)
    q[0] = 0.1 * (1.0 + q[0] / 10.0)
    q[4] = 0.01 * (1.0 + q[4] / 10.0)
    q[1:4] *= 0.9
    v, b = q[1:4], q[5:8]
    b *= 0.1 / np.maximum(1.0, np.linalg.norm(b, axis=0))
    b -= v * ((v * b).sum(0) / (v * v).sum(0))
    U = O.p2c(O.params_from_config("rmhd", CFG), q)
    return U, np.ascontiguousarray(np.tile(U, (1, -(-n // M)))[:, :n])


def _check(got, U, ref):
    n = got.shape[1]
    assert np.array_equal(got, np.tile(got[:, :M], (1, -(-n // M)))[:, :n])
    # |f| < 1e-10 max(1, tau) fixes Z to ~1.5e-10 max(1, tau) (f' >= 0.7), so v to
    # that over Z + B^2, rho to W^2 (<= 6) of it and p absolutely
    tol = 2e-9 * np.maximum(1.0, U[4])
    assert np.all(np.abs(got[:5, :M] - ref[:5]) <= tol * np.maximum(1.0, np.abs(ref[:5])))
    assert np.array_equal(got[5:, :M], ref[5:])


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("recon", ["muscl", "ppm"])  # the regrouped and the reference's order
def test_reference_batch(n, recon):
    from astrofd_b200.core import rmhd_core
    rmhd_core.configure(dict(CFG, RECON=recon, RIEMANN="hlle", PRECISION="fp64"))
    U, big = _conserved(n)
    ref = O.c2p(O.params_from_config("rmhd", CFG), U)
    _check(rmhd_core.engine().c2p_array(torch.from_numpy(big).cuda()).cpu().numpy(), U, ref)


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("listed", [True, False])
def test_learned_batch(n, listed):
    from astrofd_b200 import learned_c2p as LC
    e = LC.c2p_engine()
    U, big = _conserved(n)
    ref = O.c2p(O.params_from_config("rmhd", CFG), U)
    params = torch.as_tensor(LC.load(), dtype=torch.float32).cuda()
    q, st = LC.c2p_learned(e, torch.from_numpy(big).cuda(), params, listed=listed)
    assert st["status"] == 0 and st["cells"] == n
    _check(q.cpu().numpy(), U, ref)
