"""The router's network on feature rows that start at any float of a larger buffer."""
import numpy as np
import pytest

import route_ref as R
import tlfr

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    torch = pytest.importorskip("torch")
    gen = torch.Generator().manual_seed(seed)
    feats = torch.randn((n, R.F), generator=gen) * 2 + 1
    labels = (torch.rand(n, generator=gen) < 0.4).float()
    return torch, feats.cuda(), labels.cuda()


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_feature_rows_at_any_float(offset):
    """Probabilities, gradient and a training step of rows 4 * offset bytes into a buffer
    equal those of the same rows at its start: sixteen rows are one tile of one warp, so
    every sum has one order."""
    n = 16
    torch, feats, labels = _rows(1000, 5)
    shifted = torch.empty(feats.numel() + offset, device="cuda")
    shifted[offset:] = feats.flatten()
    torch.cuda.synchronize()
    at = [feats.data_ptr(), shifted.data_ptr() + 4 * offset]
    got = []
    for ptr in at:
        router = tlfr.Router(0, seed=11)
        prob = torch.empty(feats.shape[0], device="cuda")
        router.predict(ptr, feats.shape[0], prob.data_ptr())
        grad, loss = router.gradient(ptr, labels.data_ptr(), n)
        last = router.train(ptr, labels.data_ptr(), n, steps=1, batch=n, lr=1e-3)
        got.append((prob.cpu().numpy(), grad, np.float32([loss, last]), router.params()))
        router.close()
    for a, b in zip(*got):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
