"""Finite cells of 1e308, whose differences have no reciprocal in float64's normal range:
what lies two cells away is as the oracle gives it."""
import numpy as np
import pytest
import torch

import oracle as O
from states import make_state

pytestmark = pytest.mark.gpu

BASE = {"srhd": dict(GAMMA=5.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, PASSIVE_OFFSET=5),
        "rmhd": dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, GLM_CH=1.0, GLM_CP=0.1,
                     PASSIVE_OFFSET=9, RESISTIVE_ENABLED=False, RESISTIVITY=0.0)}


@pytest.mark.parametrize("physics,recon,riemann,var", [
    ("srhd", "muscl", "hlle", 0), ("srhd", "muscl", "hllc", 0), ("srhd", "ppm", "hllc", 0),
    ("rmhd", "muscl", "hlle", 8), ("rmhd", "muscl", "hlld", 8), ("rmhd", "muscl", "hlle", 0)])
@pytest.mark.parametrize("value", [1e308, 4.6e307, 1e280])
@pytest.mark.parametrize("seed", [3, 4])
def test_two_cells_away(physics, recon, riemann, var, value, seed):
    from astrofd_b200.core import rmhd_core, srhd_core
    pr = make_state(seed, (9, 8, 10), 3, physics, stripes=False)
    at = (7, 6, 8)
    pr[(var,) + at] = value
    cfg = dict(BASE[physics], RECON=recon, LIMITER="vanleer", RIEMANN=riemann, N_PASSIVE=0,
               FLUX_MODE="conservative", PRECISION="fp64", STAGE_KERNEL="split", C2P_GUESS="reference")
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(cfg)
    f = {"muscl": getattr(m, "compute_rhs_muscl", None) or m.compute_rhs_rmhd, "ppm": m.compute_rhs_ppm}[recon]
    got = f(torch.from_numpy(pr).cuda(), *pr.shape[1:], 0.1, 0.1, 0.1).cpu().numpy()
    ref = O.rhs(O.params_from_config(physics, cfg), pr, 0.1, 0.1, 0.1)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    ok = np.isfinite(ref)
    ok[(slice(None),) + tuple(slice(i - 1, i + 2) for i in at)] = False
    for v in range(pr.shape[0]):
        x, y = got[v][ok[v]], ref[v][ok[v]]
        # the bar of the fixture comparison: FMA and division rounding
        assert np.abs(x - y).max() <= 1e-11 * max(np.abs(y).max(), 1e-3)
