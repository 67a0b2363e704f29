"""A member's failed product is visible in the ensemble's results and raised where they reach the host."""

import numpy as np
import pytest
import torch

from pylblrtm_b200 import _lib, surrogate

pytestmark = pytest.mark.gpu


# Products of all members together (four of one architecture) and one by one (two architectures); the
# gate's vector form (200 channels, four members) and the scalar one (201 channels, seven members).
# The failure is a set error word: no wait runs out here.
@pytest.mark.parametrize("n_out,hidden", [(200, [128] * 4), (201, [128] * 7), (200, [128, 256])])
def test_failed_product_is_seen(cuda, n_out, hidden, monkeypatch):
    nets = [surrogate.MLP(61, n_out, hidden=h, depth=2, seed=i) for i, h in enumerate(hidden)]
    gs = surrogate.GatedSurrogate(nets, gate=1e9)
    raw = torch.randn((150, 61), generator=torch.Generator().manual_seed(1)).cuda()
    words, real = set(), _lib.call

    def spy(name, *args):
        if name in ("lbl_gemm_bf16", "lbl_ensemble_forward"):
            words.add(args[-2])
        return real(name, *args)

    monkeypatch.setattr(_lib, "call", spy)
    mean, est, flag = gs.ensemble(raw)
    gs.check()
    assert words == {gs.err.data_ptr()}
    assert torch.isfinite(mean).all() and torch.isfinite(est).all() and not flag.any()
    pred = gs.predictions(raw).double()
    np.testing.assert_allclose(mean.cpu().numpy(), pred.mean(0).cpu().numpy(), rtol=1e-5)
    gs.err.fill_(1)
    bad_mean, bad_est, bad_flag = gs.ensemble(raw)
    assert torch.isnan(bad_mean).all() and torch.isnan(bad_est).all() and bad_flag.all()
    with pytest.raises(RuntimeError, match="timed out"):
        gs.check()
    with pytest.raises(RuntimeError, match="timed out"):
        surrogate.calibrate_gate(gs, raw.cpu().numpy(), np.zeros((150, n_out), np.float32))
    gs.err.zero_()
    again = gs.ensemble(raw)
    assert all(torch.equal(a, b) for a, b in zip(again, (mean, est, flag)))
