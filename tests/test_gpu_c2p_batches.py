"""con2prim batches at the edges of their launches: the counters, which every
warp adds up before its one atomic, and the converted states, against the
oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from states import make_c2p_batch

pytestmark = pytest.mark.gpu

CFG = dict(GAMMA=4.0 / 3.0, P_MAX=1e3, V_MAX=0.9999, N_PASSIVE=0, PASSIVE_OFFSET=9)
# one lane, a warp less and plus one, a block and a tile plus one, several
# tiles, and one state more than one pass of the capped grid (148 * 32 blocks)
COUNTS = [1, 31, 33, 129, 4097, 148 * 32 * 128 + 1]


def _states(n):
    """Jet-like states with the field across the velocity, where the equation
    has one root."""
    q = make_c2p_batch(5, min(n, 5000))
    q[0] = 0.1 * (1.0 + q[0] / 10.0)
    q[4] = 0.01 * (1.0 + q[4] / 10.0)
    q[1:4] *= 0.9
    v, b = q[1:4], q[5:8]
    b *= 0.1 / np.maximum(1.0, np.linalg.norm(b, axis=0))
    b -= v * ((v * b).sum(0) / (v * v).sum(0))
    return np.ascontiguousarray(np.tile(q, (1, -(-n // q.shape[1])))[:, :n])


@pytest.mark.parametrize("n", COUNTS)
def test_reference_batch(n):
    from astrofd_b200.core import rmhd_core
    rmhd_core.configure(CFG)
    prm = O.params_from_config("rmhd", CFG)
    U = O.p2c(prm, _states(n))
    m = min(n, 5000)
    ref = O.c2p(prm, np.ascontiguousarray(U[:, :m]))
    rmhd_core.c2p_stats(reset=True)
    got = rmhd_core.engine().c2p_array(torch.from_numpy(U).cuda()).cpu().numpy()
    st = rmhd_core.c2p_stats(reset=True)
    assert st["cells"] == n
    assert st["newton"] + st["bisection"] == n
    # |f| < 1e-10 max(1, tau) fixes Z to ~1.5e-10 max(1, tau) (f' >= 0.7), so v
    # to that over Z + B^2, rho to W^2 (<= 6) of it and p absolutely
    tol = 2e-9 * np.maximum(1.0, U[4, :m])
    assert np.all(np.abs(got[:5, :m] - ref[:5]) <= tol * np.maximum(1.0, np.abs(ref[:5])))
    # the repeated states convert to the same bits wherever they sit
    assert np.array_equal(got[:, n - n % m - (m if n % m == 0 else 0):][:, :1], got[:, :1])


@pytest.mark.parametrize("n", COUNTS)
def test_learned_batch_counters(n):
    from astrofd_b200 import learned_c2p as LC
    e = LC.c2p_engine()
    U = torch.from_numpy(O.p2c(O.params_from_config("rmhd", CFG), _states(n))).cuda()
    params = torch.as_tensor(LC.load(), dtype=torch.float32).cuda()
    for listed in (True, False):
        _, st = LC.c2p_learned(e, U, params, listed=listed)
        assert st["status"] == 0 and st["wait_timeouts"] == 0
        assert st["cells"] == n
        assert st["learned_polish"] + st["learned_fallback"] == n
        assert st["polish_steps"] <= 2 * n
