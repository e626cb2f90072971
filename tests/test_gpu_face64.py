"""The float64 face kernels (astrofd_b200/csrc/face64.cu) against the oracle at
the sizes where their thread layouts end: rows of 31 z faces per warp, walks of
1 to 16 x or y faces per thread, blocks with one updated cell; and states
whose WENO5 denominators leave the range of the shared division, which the
general per-face evaluation takes over."""
import numpy as np
import pytest
import torch

import oracle as O
import parity as PT
from states import make_state

pytestmark = pytest.mark.gpu

BASE = {"srhd": dict(GAMMA=5.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, PASSIVE_OFFSET=5),
        "rmhd": dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, GLM_CH=1.0, GLM_CP=0.1,
                     PASSIVE_OFFSET=9, RESISTIVE_ENABLED=False, RESISTIVITY=0.0)}


def _both(physics, recon, riemann, pr, d, flux_mode="reference"):
    from astrofd_b200.core import rmhd_core, srhd_core
    cfg = dict(BASE[physics], RECON=recon, LIMITER="vanleer", RIEMANN=riemann, N_PASSIVE=0,
               FLUX_MODE=flux_mode, PRECISION="fp64")
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(cfg)
    f = {"muscl": getattr(m, "compute_rhs_muscl", None) or m.compute_rhs_rmhd,
         "ppm": m.compute_rhs_ppm, "weno": m.compute_rhs_weno}[recon]
    got = f(torch.from_numpy(pr).cuda(), *pr.shape[1:], *d).cpu().numpy()
    return got, O.rhs(O.params_from_config(physics, cfg), pr, *d)


# (4, 5, 30) .. (3, 3, 63): z rows of 31, 32, 33, 62, 63 and 64 faces;
# (1, 1, 1): one cell; the larger blocks walk several faces per thread in x and y
@pytest.mark.parametrize("n", [(4, 5, 30), (4, 5, 31), (5, 4, 32), (3, 3, 61), (3, 3, 62),
                               (3, 3, 63), (1, 1, 1), (70, 66, 65)])
@pytest.mark.parametrize("physics,recon,riemann", [("rmhd", "weno", "hlld"), ("rmhd", "ppm", "hlle"),
                                                   ("rmhd", "muscl", "hlld"), ("srhd", "weno", "hlle"),
                                                   ("srhd", "ppm", "hllc"), ("srhd", "muscl", "hllc")])
def test_rhs_at_the_edges_of_the_thread_layouts(n, physics, recon, riemann):
    ng = 3 if recon != "muscl" else 2
    pr = make_state(7, n, ng, physics, stripes=False)
    got, ref = _both(physics, recon, riemann, pr, (1.0 / n[0], 0.9 / n[1], 1.1 / n[2]))
    # the bar of the fixture comparison: FMA and division rounding
    assert PT.normwise(got, ref) < 1e-11


@pytest.mark.parametrize("physics,var", [("rmhd", 8), ("srhd", 4)])
@pytest.mark.parametrize("value", [1e60, 1e75])
def test_weno_denominators_out_of_range(physics, var, value):
    """A spike of 1e60 puts squared indicators at 1e240 and their products out
    of float64's range (1e75: the squares themselves at the edge of it), where
    the reference's separate quotients still give a result."""
    pr = make_state(8, (6, 7, 34), 3, physics, stripes=False)
    pr[var, 5, 5, 10:20:3] = value
    got, ref = _both(physics, "weno", "hlle", pr, (0.1, 0.1, 0.1))
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert ok.mean() > 0.9
    for v in range(ref.shape[0]):
        s = np.abs(ref[v][ok[v]]).max()
        assert np.abs(got[v][ok[v]] - ref[v][ok[v]]).max() <= 1e-11 * s
