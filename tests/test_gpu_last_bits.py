"""Float64 blocks whose schemes amplify a last bit (a contact speed beside speeds
that are not its face's, divided by their unbounded difference) keep the general
face evaluation, the quotients of the flux differences and the reference's con2prim
order on every path to them, not in the plain steps alone.  Their face kernels tell
the two evaluations apart: one per direction and one for the carried x faces."""
import ctypes as C

import numpy as np
import pytest
import torch

from astrofd_b200 import _lib
from astrofd_b200.core import grmhd_core, rmhd_core
from astrofd_b200.workloads import rmhd_jet
from states import make_state

pytestmark = pytest.mark.gpu

N = (9, 8, 11)


def _setup(recon, riemann, flux_mode="reference"):
    rmhd_core.configure(dict(GAMMA=4.0 / 3.0, P_MAX=2.0, V_MAX=0.9999, N_PASSIVE=0, PASSIVE_OFFSET=9,
                             RECON=recon, RIEMANN=riemann, LIMITER="mc", RESISTIVE_ENABLED=False,
                             RESISTIVITY=0.0, C2P_GUESS="reference", STAGE_KERNEL="split",
                             FLUX_MODE=flux_mode, PRECISION="fp64"))
    return torch.from_numpy(make_state(5, N, 3, "rmhd", stripes=False)).cuda()


def _launches(f):
    L = _lib.load()
    before = L.astro_launch_count()
    out = f()
    return out, L.astro_launch_count() - before


@pytest.mark.parametrize("recon", ["weno", "ppm"])
@pytest.mark.parametrize("riemann,flux_mode,faces", [("hlld", "reference", 4), ("hlle", "reference", 2),
                                                     ("hlld", "conservative", 1)])
def test_gr_steps(recon, riemann, flux_mode, faces):
    pr = _setup(recon, riemann, flux_mode)
    d = (0.1, 0.1, 0.1)
    plain = rmhd_core.step_ssprk3(pr, *d, 1e-3)
    grmhd_core.configure(dict(GR_METRIC="minkowski", GR_MASS=0.0, ORTHONORMAL_FLUX=True))
    gr, n = _launches(lambda: grmhd_core.step_ssprk3(pr, *d, 1e-3, 0, 3))
    assert n == 3 * (faces + 2)  # and the update and the con2prim of each stage
    # the con2prim runs in another kernel: the same operations, compiled apart
    scale = plain.abs().flatten(1).amax(1).clamp_min(1e-300)
    assert float(((gr - plain).abs().flatten(1).amax(1) / scale).max()) < 1e-9


@pytest.mark.parametrize("recon", ["weno", "ppm"])
@pytest.mark.parametrize("riemann,flux_mode,faces", [("hlld", "reference", 4), ("hlle", "reference", 2),
                                                     ("hlld", "conservative", 1)])
@pytest.mark.parametrize("entry", ["rhs", "static", "gr"])
def test_right_hand_sides(entry, recon, riemann, flux_mode, faces):
    L = _lib.load()
    pr = _setup(recon, riemann, flux_mode)
    shape, d = tuple(pr.shape[1:]), (0.1, 0.1, 0.1)
    plain, n = _launches(lambda: rmhd_core.engine().rhs(pr, *shape, *d))
    if entry == "static":
        out = torch.empty_like(pr)
        g = _lib.AstroGrid(*pr.shape, *d)
        rc, n = _launches(lambda: L.astro_rhs_static(
            C.byref(rmhd_core.engine().p), C.byref(g), C.c_void_p(pr.data_ptr()),
            C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert rc == 0 and torch.equal(out, plain)
    elif entry == "gr":
        grmhd_core.configure(dict(GR_METRIC="minkowski", GR_MASS=0.0, ORTHONORMAL_FLUX=True))
        out, n = _launches(lambda: grmhd_core.compute_rhs_grmhd(pr, *d, 0, 3))
        assert torch.equal(out, plain)
    assert n == faces + 1  # and the update


@pytest.mark.parametrize("riemann,flux_mode", [("hlle", "conservative"), ("hlld", "conservative"),
                                               ("hlle", "reference")])
@pytest.mark.parametrize("recon", ["ppm", "weno"])
def test_a_loop_over_right_hand_sides_and_batches_is_the_step(recon, riemann, flux_mode):
    """PPM's flattening compares neighbouring cells, whose pressures differ by the
    conversion's rounding alone where they began equal: the batch conversion keeps
    the order of operations that the configured step's has.  What remains is the
    conversion's tolerance of 1e-10 max(1, tau)."""
    ng, n = 3, 32
    pr = _setup(recon, riemann, flux_mode)
    pr = torch.from_numpy(np.ascontiguousarray(rmhd_jet(n, ng)[:9])).cuda()
    e, shape, d = rmhd_core.engine(), tuple(pr.shape[1:]), (1.0 / n,) * 3
    dt = 0.2 / n
    step = rmhd_core.step_ssprk3(pr, *d, dt)

    def rhs(q):
        return e.rhs(q, *shape, *d).reshape(9, -1)

    def prims(U):
        return e.c2p_array(U).reshape(pr.shape)

    U0 = e.p2c_array(pr)
    U1 = U0 + dt * rhs(pr)
    q = prims(U1)
    U2 = 0.75 * U0 + 0.25 * (U1 + dt * rhs(q))
    q = prims(U2)
    loop = prims(U0 / 3.0 + 2.0 / 3.0 * (U2 + dt * rhs(q)))
    scale = step.abs().flatten(1).amax(1).clamp_min(1e-300)
    assert float(((loop - step).abs().flatten(1).amax(1) / scale).max()) < 1e-8


@pytest.mark.parametrize("recon,flux_mode,faces", [("muscl", "reference", 3), ("muscl", "conservative", 3),
                                                   ("ppm", "conservative", 3), ("weno", "conservative", 3),
                                                   ("weno", "reference", 4)])
def test_hlld_full_with_any_speeds(recon, flux_mode, faces):
    """"hlld_full" also divides by D (s - v) - Bn^2; so with its own speeds too."""
    pr = _setup(recon, "hlld_full", flux_mode)
    shape, d = tuple(pr.shape[1:]), (0.1, 0.1, 0.1)
    _, n = _launches(lambda: rmhd_core.engine().rhs(pr, *shape, *d))
    assert n == faces + 1
    _, n = _launches(lambda: rmhd_core.step_ssprk2(pr, *d, 1e-3))
    assert n == 2 * (faces + 1)
