"""The float64 face kernel's walks: a face's value does not depend on how its
direction is cut into segments, so the right-hand side of a block whose threads walk 15
faces (18 in the carried x pass, which is alone; a shorter last segment in y) equals
that of its parts, cut elsewhere, bit for bit; and the schemes that use this kernel against the oracle at the ends of its
thread layouts."""
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
D = (0.02, 0.021, 0.019)
SCHEMES = [("rmhd", "weno", "hlld", "conservative"), ("rmhd", "weno", "hlle", "reference"),
           ("rmhd", "ppm", "hlld", "conservative"), ("rmhd", "ppm", "hlle", "reference"),
           ("rmhd", "muscl", "hlld", "reference"), ("srhd", "ppm", "hllc", "reference"),
           ("srhd", "weno", "hlle", "reference")]


def _rhs(physics, recon, riemann, flux_mode, pr):
    from astrofd_b200.core import rmhd_core, srhd_core
    cfg = dict(BASE[physics], RECON=recon, LIMITER="vanleer", RIEMANN=riemann, N_PASSIVE=0,
               FLUX_MODE=flux_mode, PRECISION="fp64", STAGE_KERNEL="split", C2P_GUESS="reference")
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(cfg)
    f = {"muscl": getattr(m, "compute_rhs_muscl", None) or m.compute_rhs_rmhd,
         "ppm": m.compute_rhs_ppm, "weno": m.compute_rhs_weno}[recon]
    return f(pr, *pr.shape[1:], *D), cfg


def test_the_block_below_reaches_the_longest_walks():
    """Faces of the walk, over the blocks resident at a time (4 per SM for RMHD, 8 for
    SRHD, 148 SMs), as launch() divides them."""
    for e, faces in (((131, 133), 71), ((70, 133), 132)):
        per = -(-e[0] * e[1] // 128)
        assert per * faces // (148 * 4) >= 16
        assert per * faces // (148 * 8) >= 8


@pytest.mark.parametrize("scheme", SCHEMES, ids=["-".join(s) for s in SCHEMES])
def test_parts_of_a_block(scheme):
    ng = 2 if scheme[1] == "muscl" else 3
    pr = torch.from_numpy(make_state(11, (70, 131, 133), ng, scheme[0], stripes=False)).cuda()
    whole, _ = _rhs(*scheme, pr)
    h, S = 3, pr.shape[1:]
    # x and y cut, full rows in z: the carried speeds of a cell come from its
    # predecessor in the row, or from the row before it (left out below)
    for x0, x1, y0, y1 in ((0, 17, 0, 40), (5, 71, 30, 47), (50, S[0], 90, S[1]), (31, 40, 0, S[1])):
        part, _ = _rhs(*scheme, pr[:, x0:x1, y0:y1].contiguous())
        inner = (slice(None), slice(h + 1, x1 - x0 - h), slice(h + 1, y1 - y0 - h), slice(h, S[2] - h))
        outer = (slice(None), slice(x0 + h + 1, x1 - h), slice(y0 + h + 1, y1 - h), slice(h, S[2] - h))
        assert torch.equal(part[inner], whole[outer])
        assert float(part[inner].abs().max()) > 0.0


@pytest.mark.parametrize("n", [(4, 5, 30), (5, 4, 32), (3, 3, 62), (3, 3, 63), (1, 1, 1), (33, 34, 31)])
@pytest.mark.parametrize("scheme", SCHEMES[:4], ids=["-".join(s) for s in SCHEMES[:4]])
def test_against_the_oracle(scheme, n):
    pr = make_state(7, n, 3, scheme[0], stripes=False)
    got, cfg = _rhs(*scheme, torch.from_numpy(pr).cuda())
    ref = O.rhs(O.params_from_config(scheme[0], cfg), pr, *D)
    # the bar of the fixture comparison: FMA and division rounding
    assert PT.normwise(got.cpu().numpy(), ref) < 1e-11
