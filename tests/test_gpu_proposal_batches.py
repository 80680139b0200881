"""The proposal's backward kernel at batch sizes around its grid: one window,
one more than the streaming multiprocessors, and batches that leave the last
round partly empty, for every head width, against the numpy oracle (the bound
of the other gradient tests: the activations are rounded to BF16)."""
import numpy as np
import pytest

from oracle import proposal_ref as R
from tests.test_proposal import GRAD_RTOL, _labels, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,n", [(0, 1), (1, 149), (5, 301), (7, 2), (7, 149)])
def test_gradient_batches(method, n):
    import torch
    from localizer_b200 import proposal as P
    net = P.Proposal(method, 0, seed=8)
    rng = np.random.default_rng(n)
    rois = P.synth_rois(n, elliptic=method in (5, 7), seed=n)
    lab = _labels(rng, n, net.nout)
    lam = rng.uniform(0.5, 2.0, net.nout).astype(np.float32)
    g, loss = net.gradient(rois, torch.from_numpy(lab).cuda(), lam)
    net.status()
    win = rois.cpu().numpy().view(np.uint16)
    ref_loss, ref_g = R.loss_and_grad(net.weights().astype(np.float64), win, lab.astype(np.float64), lam, net.nout)
    assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
    gg = g.cpu().numpy()
    for name, (a, b) in R.segments(net.nout).items():
        assert _rel(gg[a:b], ref_g[a:b]) < GRAD_RTOL, name
    net.close()
