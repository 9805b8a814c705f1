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


@pytest.mark.parametrize("n,repeat", [(100003, 1), (1 << 18, 1), (1 << 18, 16)])
def test_gradient_of_many_rows(n, repeat):
    """Several groups of rows per block, against the BF16 network in 64 bits.  Repeating
    the rows a power of two times changes no rounding but that of the sums.  Bound: an
    accumulator goes through 32 truncating mma, each losing half a unit in the last place
    of a sum that grows to its end (32 * 2^-24 / 2, 1e-6), and 5e-7 for the sums in FP32
    and for activations that round to BF16 the other way (1/sqrt(n))."""
    torch, feats, labels = _rows(n, 7)
    router = tlfr.Router(0, seed=11, mean=np.full(R.F, 1, np.float32), inv_std=np.full(R.F, 0.5, np.float32))
    f, y = feats.repeat(repeat, 1), labels.repeat(repeat)
    torch.cuda.synchronize()
    grad, _ = router.gradient(f.data_ptr(), y.data_ptr(), n * repeat)
    want = R.gradient(router.params(), feats.cpu().numpy(), labels.cpu().numpy())
    router.close()
    assert np.linalg.norm(grad - want) <= 1.5e-6 * np.linalg.norm(want)
