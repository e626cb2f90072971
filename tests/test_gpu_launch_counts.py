"""The launch count and the kernel timing's launches count face passes that ran:
one per kernel in float64 (per direction, with its listed faces, in float32),
none for a block without updated cells."""
import ctypes as C

import pytest
import torch

from astrofd_b200 import _lib
from astrofd_b200.core import rmhd_core, srhd_core
from states import make_state

pytestmark = pytest.mark.gpu


def _setup(physics, recon, riemann, flux_mode="reference", precision="fp64"):
    m = srhd_core if physics == "srhd" else rmhd_core
    m.configure(dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, N_PASSIVE=0, RECON=recon,
                     PASSIVE_OFFSET=5 if physics == "srhd" else 9, RIEMANN=riemann,
                     RESISTIVE_ENABLED=False, RESISTIVITY=0.0, C2P_GUESS="reference",
                     STAGE_KERNEL="split", FLUX_MODE=flux_mode, PRECISION=precision))
    return m


def face_launches(physics, recon, riemann, flux_mode="reference", precision="fp64", n=(6, 5, 7)):
    """face launches of one SSPRK2 step, per stage"""
    m = _setup(physics, recon, riemann, flux_mode, precision)
    pr = torch.from_numpy(make_state(3, n, 3, physics, stripes=False)).cuda()
    _, _, launches = m.engine().step_profiled(pr, 0.1, 0.1, 0.1, 1e-3, 2, torch.empty_like(pr))
    assert launches[0] % 2 == 0
    return launches[0] // 2


@pytest.mark.parametrize("args,count", [
    (("srhd", "weno", "hllc"), 1),
    (("rmhd", "weno", "hlld", "conservative"), 1),
    (("rmhd", "weno", "hlle"), 2),   # z and y, then x with the carried speeds
    (("rmhd", "weno", "hlld"), 4),   # z, x, carried x, y
    (("rmhd", "ppm", "hlld"), 4),
    (("srhd", "weno", "hllc", "reference", "mixed"), 3),
    (("rmhd", "weno", "hlld", "reference", "mixed"), 4),
])
def test_face_launches_of_a_stage(args, count):
    assert face_launches(*args) == count


# 7 x 7 x 6 cells: no updated cell, so no float64 face.  The float32 passes have one
# z face (its pass, and for all three directions the one of the listed faces) and
# the float32 copy.
@pytest.mark.parametrize("args,count", [
    (("srhd", "weno", "hllc"), 0),
    (("rmhd", "weno", "hlle"), 0),
    (("rmhd", "weno", "hlld"), 0),
    (("rmhd", "weno", "hlld", "conservative"), 0),
    (("srhd", "weno", "hllc", "reference", "mixed"), 3),
    (("rmhd", "weno", "hlld", "reference", "mixed"), 2),
])
def test_no_updated_cells(args, count):
    L = _lib.load()
    m = _setup(*args)
    nm = 5 if args[0] == "srhd" else 9
    pr = torch.from_numpy(make_state(3, (1, 1, 1), 3, args[0], stripes=False)[:, :, :, :6].copy()).cuda()
    rhs = torch.empty((nm,) + tuple(pr.shape[1:]), dtype=torch.float64, device="cuda")
    g = _lib.AstroGrid(*pr.shape, 0.1, 0.1, 0.1)
    p = m.engine().p
    nb = L.astro_rhs_workspace_bytes(C.byref(p), C.byref(g))
    w = torch.empty(nb, dtype=torch.uint8, device="cuda")
    before = L.astro_launch_count()
    assert L.astro_rhs(C.byref(p), C.byref(g), C.c_void_p(pr.data_ptr()), C.c_void_p(rhs.data_ptr()),
                       C.c_void_p(w.data_ptr()), nb, None) == 0
    assert L.astro_launch_count() - before == count + 1  # and the update
    torch.cuda.synchronize()
    assert float(rhs.abs().max()) == 0.0
