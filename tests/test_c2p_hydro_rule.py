"""The hydro con2prim stops a fixed point that runs away after its first step
(s_c2p, astrofd_b200/csrc/physics.cuh).  On the CPU: that rule against the
reference's 60 steps, over physical and unphysical conserved states.  On the
GPU: the conversion against the oracle's, which takes all 60 steps."""
import numpy as np
import pytest

import oracle as O

SM = 1e-12


def _states(n, gamma, kind, seed):
    """Conserved SRHD states: rho 1e-6..100, p 1e-9..100, W up to `kind`'s
    range; "odd" scales D and tau away from any physical state, some negative."""
    r = np.random.default_rng(seed)
    rho, p = 10.0 ** r.uniform(-6, 2, n), 10.0 ** r.uniform(-9, 2, n)
    W = {"slow": 1.0 + 10.0 ** r.uniform(-16, -2, n), "rest": np.ones(n)}.get(
        kind, 10.0 ** r.uniform(0, 2.2, n))
    d = r.normal(size=(3, n))
    d *= np.sqrt(1.0 - 1.0 / W ** 2) / np.linalg.norm(d, axis=0)
    w = (rho + gamma / (gamma - 1.0) * p) * W * W
    U = np.vstack([rho * W, w * d, w - p - rho * W])
    if kind == "odd":
        U[0] *= 10.0 ** r.uniform(-3, 1, n) * np.where(r.random(n) < 0.05, -1, 1)
        U[4] *= 10.0 ** r.uniform(-3, 1, n) * np.where(r.random(n) < 0.1, -1, 1)
    return U


def _fixed_point(U, gamma, p_max, v_max, rule):
    D, S2, tau = U[0], (U[1:4] ** 2).sum(0), U[4]
    E = tau + D
    p0 = np.clip((gamma - 1.0) * (E - D), SM, p_max)
    p, ok, stop = p0.copy(), np.zeros(D.shape, bool), np.zeros(D.shape, bool)
    for it in range(60):
        Wm = E + p
        v2 = S2 / (Wm * Wm + SM)
        v2 = np.where(v2 >= v_max ** 2, v_max ** 2 - 1e-14, v2)
        W = 1.0 / np.sqrt(1.0 - v2)
        rho = D / W
        h = 1.0 + gamma / (gamma - 1.0) * p / np.maximum(rho, SM)
        dp = np.clip(-(Wm - rho * h * W * W), -0.5 * p, 0.5 * p)
        pn = np.clip(p + dp, SM, p_max)
        hit = np.abs(dp) < 1e-12 * np.maximum(1.0, pn)
        live = ~(ok | stop)
        if rule and it == 0:
            stop |= ~hit & (dp > 0.0) & (D > 2.0 * SM * W)
            live = ~stop
        p = np.where(live, pn, p)
        ok |= live & hit
    return np.where(ok, p, p0), stop


@pytest.mark.parametrize("kind", ["jet", "slow", "rest", "odd"])
@pytest.mark.parametrize("gamma,p_max", [(4.0 / 3.0, 2.0), (5.0 / 3.0, 2.0), (5.0 / 3.0, 1e9),
                                         (1.05, 1e3), (1.9, 1e3)])
def test_a_runaway_start_ends_where_sixty_steps_end(kind, gamma, p_max):
    U = _states(10000, gamma, kind, 11)
    full, _ = _fixed_point(U, gamma, p_max, 0.9999, rule=False)
    fast, stopped = _fixed_point(U, gamma, p_max, 0.9999, rule=True)
    assert np.array_equal(full, fast)
    if kind == "jet":
        assert stopped.mean() > 0.5


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["jet", "slow", "rest", "odd"])
@pytest.mark.parametrize("p_max", [2.0, 1e9])
def test_device_conversion_equals_the_oracles(kind, p_max):
    import torch
    from astrofd_b200.core import srhd_core
    cfg = dict(GAMMA=5.0 / 3.0, P_MAX=p_max, V_MAX=0.9999, N_PASSIVE=0, PASSIVE_OFFSET=5)
    U = _states(20001, 5.0 / 3.0, kind, 12)
    ref = O.c2p(O.params_from_config("srhd", cfg), U)
    srhd_core.configure(cfg)
    got = srhd_core.engine().c2p_array(torch.from_numpy(U).cuda()).cpu().numpy()
    # both stop within 1e-12 max(1, p) of the same value (p0, or the converged
    # p); v = S / (E + p) then differs by as much relative to E + p, and
    # 1 - v^2 loses W^2 of it (W^2 <= 5000 at V_MAX)
    tol = 4e-12 * np.maximum(1.0, ref[4])
    assert np.all(np.abs(got[4] - ref[4]) <= tol)
    rel = tol / np.maximum(U[4] + U[0] + ref[4], 1e-300) + 1e-15
    W2 = 1.0 / (1.0 - (ref[1:4] ** 2).sum(0))
    same = (U[4] + U[0] + ref[4]) > 1e-9  # below, E + p is floored away
    assert np.all((np.abs(got[1:4] - ref[1:4]) <= 2.0 * rel)[:, same])
    assert np.all((np.abs(got[0] - ref[0]) <= 4.0 * W2 * rel * np.maximum(ref[0], SM))[same])
