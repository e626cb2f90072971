"""Blocks and workspaces that only hold float64 values (8-byte aligned): the mixed
path's wide copies then give way to single values, with the same results."""
import ctypes as C

import numpy as np
import pytest
import torch

from astrofd_b200 import _lib
from states import make_state

pytestmark = pytest.mark.gpu


def _params(physics):
    p = _lib.AstroParams()
    p.physics, p.recon, p.riemann, p.limiter = physics, 2, 1, 0
    p.passive_offset = 5 if physics == _lib.SRHD else 9
    p.gamma = 4.0 / 3.0 if physics == _lib.RMHD else 5.0 / 3.0
    p.srhd_gamma = 5.0 / 3.0
    p.p_max, p.v_max, p.glm_ch, p.glm_cp = 2.0, 0.9999, 1.0, 0.1
    p.flux_mode = _lib.FLUX_CONSERVATIVE
    p.precision = _lib.PREC_MIXED
    return p


def _shifted(nbytes, shift):
    return torch.empty(nbytes + shift, dtype=torch.uint8, device="cuda")[shift:]


@pytest.mark.parametrize("physics", [_lib.SRHD, _lib.RMHD])
# 11 x 10 x 9 cells: the copies are no multiple of four values long
@pytest.mark.parametrize("n", [(5, 4, 3), (6, 5, 4)])
def test_eight_byte_alignment(physics, n):
    L = _lib.load()
    pr = make_state(3, n, 3, "srhd" if physics == _lib.SRHD else "rmhd", stripes=False)
    g = _lib.AstroGrid(*pr.shape, 0.1, 0.12, 0.14)
    p = _params(physics)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    nr = L.astro_rhs_workspace_bytes(C.byref(p), C.byref(g))
    ns = L.astro_step_workspace_bytes(C.byref(p), C.byref(g))
    results = []
    for block_shift, work_shift in ((0, 0), (8, 0), (0, 8), (8, 8)):
        src = _shifted(pr.nbytes, block_shift)
        src.copy_(torch.from_numpy(pr.view(np.uint8).reshape(-1)))
        out, rhs = _shifted(pr.nbytes, block_shift), _shifted(pr.nbytes, block_shift)
        w = _shifted(max(nr, ns), work_shift)
        assert w.data_ptr() % 16 == work_shift and src.data_ptr() % 16 == block_shift
        ptr = [C.c_void_p(t.data_ptr()) for t in (src, rhs, out, w)]
        assert L.astro_rhs(C.byref(p), C.byref(g), ptr[0], ptr[1], ptr[3], nr, stream) == 0
        assert L.astro_step(C.byref(p), C.byref(g), ptr[0], ptr[2], 1e-3, 3, ptr[3], ns, None,
                            stream) == 0
        results.append((rhs.cpu(), out.cpu()))
    for r in results[1:]:
        assert torch.equal(r[0], results[0][0]) and torch.equal(r[1], results[0][1])
