"""Conversions of component tensors: the successive rows of one block go to the
device as they lie, every other arrangement through a stacked copy; both give the
same values and leave the inputs alone."""
import numpy as np
import pytest
import torch

from states import make_c2p_batch

pytestmark = pytest.mark.gpu


def _arrangements(q):
    n = q.shape[1]
    wide = torch.zeros((9, n + 3), dtype=q.dtype, device=q.device)
    wide[:, :n] = q
    pairs = q.repeat_interleave(2, dim=1)
    odd = torch.zeros(9 * n + 1, dtype=q.dtype, device=q.device)[1:].view(9, n)
    odd.copy_(q)
    return {"rows": list(q), "odd offset": list(odd), "row pitch": [wide[v, :n] for v in range(9)],
            "strided": [pairs[v, ::2] for v in range(9)],
            "separate": [q[v].clone() for v in range(9)],
            "blocks": [q[v].reshape(n // 6, 3, 2) for v in range(9)],
            "transposed": [q[v].reshape(n // 6, 6).t().contiguous().t() for v in range(9)]}


@pytest.mark.parametrize("kind", ["rows", "odd offset", "row pitch", "strided", "separate", "blocks",
                                  "transposed"])
def test_arrangements_agree(kind):
    from astrofd_b200.core import rmhd_core
    rmhd_core.configure(dict(GAMMA=4.0 / 3.0, P_MAX=1e3, V_MAX=0.9999))
    q = torch.from_numpy(make_c2p_batch(3, 600)).cuda()
    ref_u = rmhd_core.engine().p2c_array(q * 1.0)
    keep = q.clone()
    comps = _arrangements(q)[kind]
    U = rmhd_core.prim_to_cons_rmhd(*comps, gamma=4.0 / 3.0)
    assert torch.equal(q, keep)
    for v in range(9):
        assert U[v].shape == comps[v].shape
        assert torch.equal(U[v].reshape(-1), ref_u[v])
    comps = _arrangements(ref_u)[kind]
    back = rmhd_core.cons_to_prim_rmhd(*comps)
    want = rmhd_core.engine().c2p_array(ref_u * 1.0)
    for v in range(9):
        assert torch.equal(back[v].reshape(-1), want[v])


def test_swapped_components_are_not_taken_for_rows():
    from astrofd_b200.core import srhd_core
    srhd_core.configure({})
    q = torch.from_numpy(make_c2p_batch(4, 66)[:5]).cuda()
    q[1:4] *= 0.5
    a = srhd_core.prim_to_cons(q[0], q[2], q[1], q[3], q[4])
    b = srhd_core.prim_to_cons(*[c.clone() for c in (q[0], q[2], q[1], q[3], q[4])])
    for x, y in zip(a, b):
        assert torch.equal(x, y)


def test_single_precision_components_are_refused_as_before():
    from astrofd_b200 import _lib
    from astrofd_b200.core import srhd_core
    q = torch.zeros((5, 8), device="cuda")
    with pytest.raises(_lib.AstroError):
        srhd_core.prim_to_cons(*q)
