"""Conversions of lazily negated views (torch keeps the sign in a bit beside the
memory) give what the views' values give."""
import numpy as np
import pytest
import torch

from states import make_c2p_batch

pytestmark = pytest.mark.gpu


def test_negated_rows_of_one_block():
    from astrofd_b200.core import srhd_core
    srhd_core.configure({})
    q = make_c2p_batch(4, 66)[:5]
    q[1:4] *= 0.5
    plain = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    rows = list(torch._neg_view(-plain))
    assert all(r.is_neg() for r in rows)
    for a, b in zip(srhd_core.prim_to_cons(*rows), srhd_core.prim_to_cons(*plain)):
        assert torch.equal(a, b)
