"""The list of float32 faces to recompute in float64: one list for the passes of the
three directions, in the order they run, so that one direction can use all of it."""
import ctypes as C

import numpy as np
import pytest
import torch

import parity as PT
from astrofd_b200 import _lib
from astrofd_b200.core import rmhd_core
from states import make_state

pytestmark = pytest.mark.gpu

N, NG = (14, 14, 20), 3
PLANES = (5, 11, 17)  # ghost-inclusive; at least two cells apart and from the updated range's ends
CFG = dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, GLM_CH=1.0, GLM_CP=0.1, PASSIVE_OFFSET=9, N_PASSIVE=0,
           RESISTIVE_ENABLED=False, RESISTIVITY=0.0, RECON="weno", LIMITER="mc", RIEMANN="hlle",
           FLUX_MODE="conservative", STAGE_KERNEL="split", C2P_GUESS="reference")


def _block(axes):
    """psi with planes of 1e12 across the given axes: the squared smoothness indicators
    (1e24, squared again) overflow float32 where all three stencils of a face's left or
    right value contain the plane, that is at the plane's two faces."""
    pr = make_state(9, N, NG, "rmhd", stripes=False)
    pr[8] = 0.0
    for ax in axes:
        for k in PLANES[:2] if ax < 2 else PLANES:
            s = [8] + [slice(None)] * 3
            s[1 + ax] = k
            pr[tuple(s)] = 1e12
    return pr


def test_one_direction_may_fill_the_list():
    L = _lib.load()
    rmhd_core.configure(dict(CFG, PRECISION="mixed"))
    pr = torch.from_numpy(_block([2])).cuda()
    nc = pr[0].numel()
    cap = nc // 16 + 1024
    g = _lib.AstroGrid(*pr.shape, 0.1, 0.1, 0.1)
    p = rmhd_core.engine().p
    nb = L.astro_rhs_workspace_bytes(C.byref(p), C.byref(g))
    w = torch.full((nb,), 0xFF, dtype=torch.uint8, device="cuda")
    rhs = torch.empty_like(pr)
    assert L.astro_rhs(C.byref(p), C.byref(g), C.c_void_p(pr.data_ptr()), C.c_void_p(rhs.data_ptr()),
                       C.c_void_p(w.data_ptr()), nb, None) == 0
    torch.cuda.synchronize()
    # the workspace: three flux blocks of 9 float32 rows, then the counters, then the list
    off = 3 * ((9 * nc * 4 + 255) // 256 * 256)
    words = w[off:off + 256 + 4 * cap].cpu().numpy().view(np.uint32)
    # two zero words, then the counts of z, x and y
    listed, lst = int(words[2]), words[64:]
    assert words[[0, 1, 3, 4]].tolist() == [0, 0, 0, 0]
    assert cap // 3 < listed <= cap
    e = (N[0], N[1], N[2] + 1)  # z faces
    c = sorted(k + o - NG for k in PLANES for o in (0, 1))
    want = (np.arange(e[0] * e[1])[:, None] * e[2] + np.array(c)[None]).reshape(-1)
    # all of the planes' faces, but for the few where supersonic flow takes the flux of
    # the finite side alone
    assert listed > 0.95 * want.size
    assert np.unique(lst[:listed]).size == listed and np.isin(lst[:listed], want).all()
    assert np.all(lst[listed:] == 0xFFFFFFFF)


@pytest.mark.parametrize("axes", [[2], [0], [1], [0, 2], [0, 1, 2]])
def test_every_listed_or_searched_face_is_recomputed(axes):
    """With planes across several axes the later passes find the list full.  A face left
    as it was would not be finite; density, momentum and energy do not depend on psi."""
    pr = torch.from_numpy(_block(axes)).cuda()
    out = {}
    for prec in ("mixed", "fp64"):
        rmhd_core.configure(dict(CFG, PRECISION=prec))
        out[prec] = rmhd_core.compute_rhs_weno(pr, *pr.shape[1:], 0.1, 0.1, 0.1).cpu().numpy()
    assert np.isfinite(out["fp64"]).all() and np.isfinite(out["mixed"]).all()
    # float32 faces: 2^-24 of the largest flux, times W^2 <= 50 and ten for the
    # cancellation of the flux difference
    assert PT.normwise(out["mixed"][:5], out["fp64"][:5]) < 1e-4
