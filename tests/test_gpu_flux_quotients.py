"""Float64 right-hand sides divide the flux differences by the cell widths to the last bit:
with the other two widths at 1e300 the right-hand side at width 1 is the flux
difference itself (where that is not zero), and at any width h the IEEE quotient of it."""
import numpy as np
import pytest
import torch

from states import make_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("physics,recon,riemann,flux_mode", [
    ("srhd", "muscl", "hlle", "reference"), ("srhd", "ppm", "hllc", "reference"),
    ("srhd", "weno", "hlle", "reference"), ("rmhd", "muscl", "hlld", "reference"),
    ("rmhd", "ppm", "hlle", "reference"), ("rmhd", "weno", "hlld", "conservative"),
    ("rmhd", "weno", "hlld", "reference")])
def test_quotients(physics, recon, riemann, flux_mode, axis):
    from astrofd_b200.core import rmhd_core, srhd_core
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, GLM_CH=1.0, GLM_CP=0.1, RECON=recon,
                     LIMITER="mc", RIEMANN=riemann, FLUX_MODE=flux_mode, PRECISION="fp64", N_PASSIVE=0,
                     PASSIVE_OFFSET=5 if physics == "srhd" else 9, RESISTIVE_ENABLED=False, RESISTIVITY=0.0,
                     STAGE_KERNEL="split", C2P_GUESS="reference"))
    pr = make_state(6, (13, 12, 14), 3, physics, stripes=False)
    nm = 5 if physics == "srhd" else 8  # psi's own damping does not divide
    t = torch.from_numpy(pr).cuda()

    def rhs(h):
        d = [1e300] * 3
        d[axis] = h
        return m.engine().rhs(t, *t.shape[1:], *d).cpu().numpy()[:nm]

    one = rhs(1.0)
    there = np.abs(one) > 1e-200  # elsewhere the other directions' 1e-300 is all there is
    assert np.isfinite(one).all() and there.mean() > 0.2
    for h in (0.1, 1.0 / 61, 1.0 / 128, 3.0, 0.7, 1.1e-3):
        assert np.array_equal(rhs(h)[there], (one / h)[there]), h
