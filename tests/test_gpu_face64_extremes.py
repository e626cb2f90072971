"""Finite cells beyond the range of the float64 faces' reciprocals: the reference
clamps such a velocity to zero (v_max over an infinite square root), and its face then
has that state's wave speeds, whichever side the flux is taken from."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu

BASE = {"srhd": dict(GAMMA=5.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, PASSIVE_OFFSET=5),
        "rmhd": dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, GLM_CH=1.0, GLM_CP=0.1,
                     PASSIVE_OFFSET=9, RESISTIVE_ENABLED=False, RESISTIVITY=0.0)}


@pytest.mark.parametrize("physics,recon,riemann", [("srhd", "muscl", "hlle"), ("srhd", "muscl", "hllc"),
                                                   ("srhd", "ppm", "hllc"), ("srhd", "weno", "hlle"),
                                                   ("rmhd", "muscl", "hlle"), ("rmhd", "muscl", "hlld"),
                                                   ("rmhd", "ppm", "hlle")])
@pytest.mark.parametrize("direction", [0, 1, 2])
@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_huge_velocity_beside_supersonic_flow(physics, recon, riemann, direction, sign):
    from astrofd_b200.core import rmhd_core, srhd_core
    rng = np.random.default_rng(4)
    nm = 5 if physics == "srhd" else 9
    pr = np.zeros((nm, 12, 13, 14))
    pr[0] = 1.0 + 0.1 * rng.random(pr.shape[1:])
    pr[1 + direction] = sign * 0.9
    pr[4] = 0.01
    if nm == 9:
        pr[5:8] = 0.01
    pr[1 + (direction + 1) % 3, 6, 6, 6] = 1e200
    cfg = dict(BASE[physics], RECON=recon, LIMITER="minmod", RIEMANN=riemann, N_PASSIVE=0,
               FLUX_MODE="conservative", PRECISION="fp64", STAGE_KERNEL="split", C2P_GUESS="reference")
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(cfg)
    f = {"muscl": getattr(m, "compute_rhs_muscl", None) or m.compute_rhs_rmhd,
         "ppm": m.compute_rhs_ppm, "weno": m.compute_rhs_weno}[recon]
    got = f(torch.from_numpy(pr).cuda(), *pr.shape[1:], 0.1, 0.1, 0.1).cpu().numpy()
    ref = O.rhs(O.params_from_config(physics, cfg), pr, 0.1, 0.1, 0.1)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    ok = np.isfinite(ref)
    for v in range(nm):
        # FMA and division rounding, as in the comparison with the reference's fixtures
        scale = max(np.abs(ref[v][ok[v]]).max(), 1.0)
        assert np.abs(got[v][ok[v]] - ref[v][ok[v]]).max() <= 1e-11 * scale
