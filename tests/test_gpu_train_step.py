"""The fused training step where it can go wrong: one row, a partial tile, more
tiles than SMs (persistent loop), splits of several 256-row stages, few band
groups.  Bounds as the gradient test of the network: per parameter block 1.5e-2
against the bf16-mimicking oracle, losses 1e-4."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from oracle import cvnet_oracle as NO

from test_gpu_cvnet import make_labels, random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,G", [(1, 5), (129, 1), (1500, 6), (20000, 8)])
def test_gradient_sizes(rows, G):
    net = D.CvNet(D.cvnet_default_config(ridge=0.05, n_groups=16))
    p = random_params(7)
    scales = np.array([2.0, 1.3, 0.8], np.float32)
    net.set_params(p, scales)
    feats = NO.bf16(np.random.default_rng(1).uniform(-1, 1, (rows, NO.NFEAT)).astype(np.float32))
    lab = make_labels(rows, G, 2)
    g, loss = net.gradient(feats, lab)
    gm, lm, _ = NO.gradient(p, feats, lab, scales, 0.05, mimic=True)
    np.testing.assert_allclose(loss[1:], lm, rtol=1e-4)
    edges = [NO.OFF_W1, NO.OFF_B1, NO.OFF_W2, NO.OFF_B2, NO.OFF_W3, NO.OFF_B3, NO.OFF_W4, NO.OFF_B4, NO.NPARAM]
    for a, b in zip(edges[:-1], edges[1:]):
        assert np.linalg.norm(g[a:b] - gm[a:b]) <= 1.5e-2 * np.linalg.norm(gm[a:b]), (a, b)
    net.close()


def test_training_is_the_same_whatever_the_split():
    """A batch of 17 x 256 + 128 rows (a split of two stages, an idle one at the
    end) steps like Adam on the gradient the same rows give alone."""
    rows, G = 4480, 4
    net = D.CvNet(D.cvnet_default_config(n_groups=16))
    p = random_params(9)
    scales = np.array([1.5, 0.7, 1.1], np.float32)
    net.set_params(p, scales)
    feats = NO.bf16(np.random.default_rng(4).uniform(-1, 1, (rows, NO.NFEAT)).astype(np.float32))
    lab = make_labels(rows, G, 6)
    whole, _ = net.gradient(feats, lab)
    halves = [net.gradient(feats[s], lab[s])[0] for s in (slice(0, 2240), slice(2240, rows))]
    mean = 0.5 * (halves[0] + halves[1])
    # f32 accumulation in another order; dO of a half is rounded to bf16 twice as large
    assert np.linalg.norm(whole - mean) <= 1e-3 * np.linalg.norm(whole)
    net.close()
