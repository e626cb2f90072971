"""The training kernel at the edges of its 128-sample tiles, and with parameter
and gradient blocks that are only 4-byte aligned (its 16-byte loads and
reductions then give way to single values), against the CPU restatement."""
import numpy as np
import pytest
import torch

import mlp_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 148 * 128 + 5])
def test_gradients(n, shift):
    from astrofd_b200 import _lib, learned_c2p as LC, runtime as rt
    L = _lib.load()
    rng = np.random.default_rng(n)
    flat = LC.init_params(seed=3)
    X = rng.normal(size=(n, 5)).astype(np.float32)
    T = rng.normal(size=(n, 2)).astype(np.float32)
    nt = L.astro_mlp_trainable()
    p = torch.zeros(flat.size + shift, device="cuda")[shift:]
    p.copy_(torch.from_numpy(flat))
    g = torch.zeros(nt + shift, device="cuda")[shift:]
    loss = torch.zeros(1, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, t = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    _lib.check(L.astro_mlp_train_grad(rt.ptr(p), rt.ptr(x), rt.ptr(t), n, rt.ptr(g), rt.ptr(loss),
                                      rt.ptr(status), rt.stream_handle()), "train_grad")
    assert int(status.item()) == 0
    ref_loss, ref = MO.loss_and_grads(LC.unpack(flat), X, T)
    assert abs(float(loss.item()) - ref_loss) <= 1e-4 * ref_loss
    off, _ = LC.offsets()
    got = g.cpu().numpy()
    for name, want in ref.items():
        o, shp = off[name]
        have = got[o:o + int(np.prod(shp))].reshape(shp)
        # the restatement rounds the same operands to bfloat16; an activation on
        # a rounding boundary moves by 2^-8 of itself, one among the many summed
        scale = max(np.abs(want).max(), 1e-30)
        assert np.abs(have - want).max() <= 2.0 ** -6 * scale, name
