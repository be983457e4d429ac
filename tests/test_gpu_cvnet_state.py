"""What a network holds between calls: inputs and permutations on their way to
the device, chained training steps, work buffers shared by several solvers."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from oracle import cvnet_oracle as NO

from test_gpu_cvnet import make_labels, random_params, small_table, table_solver
from test_gpu_parity import packet_index, smooth_field

pytestmark = pytest.mark.gpu


def test_gradients_of_inputs_that_are_still_being_copied():
    """Calls one after the other on inputs of several megabytes: each has its
    own inputs complete before its kernels start."""
    net = D.CvNet(D.cvnet_default_config(ridge=0.05, n_groups=16))
    scales = np.array([2.0, 1.3, 0.8], np.float32)
    rng = np.random.default_rng(1)
    sets = []
    for seed, rows in ((2, 60000), (3, 3000), (4, 40000)):
        feats = NO.bf16(rng.uniform(-1, 1, (rows, NO.NFEAT)).astype(np.float32))
        sets.append((random_params(seed), feats, make_labels(rows, 8, seed)))
    ref = []
    for p, f, y in sets:
        net.set_params(p, scales)
        net.gradient(f, y)
        ref.append(net.gradient(f, y))
    for _ in range(3):
        for (p, f, y), (g, loss) in zip(sets, ref):
            net.set_params(p, scales)
            g1, loss1 = net.gradient(f, y)
            np.testing.assert_array_equal(g, g1)
            np.testing.assert_array_equal(loss, loss1)
    net.close()


def training_net(batch, data=None, **kw):
    """A network with the 1536 rows of one small solve (data: their features
    and labels, [rows][67] and [rows][G][8])."""
    s = table_solver(small_table(), 12, 32, 4, sampler=D.SAMPLER_RQMC, nvar=4, local_sampling=1, control_variate=1,
                     cv_moments=1, seed=5)
    x = (0.1 + 0.05 * np.random.default_rng(3).uniform(-1, 1, (4, 32, 12))).astype(np.float32)
    s.set_fields(smooth_field(12, 32, 4, 450, 1700, 8), x)
    s.set_rays(16)
    s.solve(timeout_s=60)
    net = D.CvNet(D.cvnet_default_config(n_groups=8, batch=batch, seed=9, **kw))
    net.add_training_data(s)
    if data is not None:
        rows = lambda a: a.transpose(0, 4, 2, 3, 1, *range(5, a.ndim)).reshape(1536, 4, *a.shape[5:])  # tally order
        m = rows(s.cv_moments()) / 16
        var = rows(s.group_results()[1]) * 16
        pack = packet_index(s).transpose(2, 0, 1).ravel()
        steps = s.item_steps().reshape(4, -1)[:, pack].T / 16
        cov = [m[..., 3] - m[..., 0] ** 2, m[..., 4] - m[..., 1] ** 2, m[..., 5] - m[..., 2] ** 2,
               m[..., 6] - m[..., 0] * m[..., 1], m[..., 7] - m[..., 0] * m[..., 2], m[..., 8] - m[..., 1] * m[..., 2]]
        for q in range(3):
            cov[q] = np.maximum(cov[q], 0.0)
        data += [net.features(s), np.stack(cov + [var, steps], -1).astype(np.float32)]
    s.close()
    return net


@pytest.mark.parametrize("batch,passes", [(128, 6), (1024, 3)])
def test_passes_of_one_call_equal_passes_of_several(batch, passes):
    """The order of a pass is shuffled while the pass before is still only
    enqueued; every pass uses its own."""
    a, b = training_net(batch), training_net(batch)
    la = a.train(passes)
    for _ in range(passes):
        lb = b.train(1)
    np.testing.assert_array_equal(a.params()[0], b.params()[0])
    np.testing.assert_array_equal(la, lb)
    a.close()
    b.close()


def test_chained_steps_are_adam_steps_on_the_gradient():
    """Steps whose kernels are placed while the ones before still run: the
    parameters follow Adam on the gradient of the same rows, moments carried
    along, and both copies of the weights follow the parameters.

    Row order and the labels' last places differ between the two gradients,
    about 2e-5 of a typical element, so about that share of the elements may
    step the other way: 2 sqrt(2e-5) = 9e-3 of the step's norm, bound 2e-2."""
    data = []
    net = training_net(2048, data, ridge=0.02)
    feats, lab = data
    p0 = random_params(9)
    net.set_params(p0)
    scales = net.params()[1]
    other = D.CvNet(D.cvnet_default_config(n_groups=8, ridge=0.02))
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    p, m, v = p0.astype(np.float64), 0.0, 0.0
    for step in (1, 2, 3):
        other.set_params(p.astype(np.float32), scales)
        g = other.gradient(feats, lab)[0].astype(np.float64)
        m = b1 * m + (1 - b1) * g
        v = b2 * v + (1 - b2) * g * g
        upd = lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
        net.train(1)
        now = net.params()[0].astype(np.float64)
        assert np.linalg.norm(upd) > 0.5 * lr * np.sqrt(upd.size)  # nearly every element steps
        assert np.linalg.norm((p - now) - upd) <= 2e-2 * np.linalg.norm(upd), step
        p = now
    # three steps in one call give what three calls gave
    again = training_net(2048, None, ridge=0.02)
    again.set_params(p0)
    again.train(3)
    np.testing.assert_array_equal(again.params()[0], net.params()[0])
    other.set_params(net.params()[0], scales)
    np.testing.assert_array_equal(again.gradient(feats, lab)[0], other.gradient(feats, lab)[0])
    np.testing.assert_array_equal(again.eval(feats), other.eval(feats))
    for n in (net, other, again):
        n.close()


def test_one_network_applied_to_several_solvers():
    """Applied to two solvers one after the other, each with its own stream, and
    trained right after: the work buffers and weights of one are not changed
    under the other."""
    tb = small_table()
    net = training_net(128)
    net.set_params(random_params(13))
    p0 = net.params()[0]

    def solver(seed):
        s = table_solver(tb, 48, 64, 32, sampler=D.SAMPLER_RQMC, nvar=4, local_sampling=1, control_variate=1, seed=seed)
        x = (0.1 + 0.05 * np.random.default_rng(seed).uniform(-1, 1, (32, 64, 48))).astype(np.float32)
        s.set_fields(smooth_field(48, 64, 32, 450, 1700, seed), x)
        return s

    solvers = [solver(s) for s in (1, 2)]
    ref = []
    for s in solvers:
        net.apply(s, mean_rays=16, min_rays=4, max_rays=64)
        ref.append((s.cv_beta(), s.rays_per_item()))
    for _ in range(5):
        for s in solvers:
            net.apply(s, mean_rays=16, min_rays=4, max_rays=64)
        net.train(1)
        for s, (beta, rays) in zip(solvers, ref):
            np.testing.assert_array_equal(s.cv_beta(), beta)
            np.testing.assert_array_equal(s.rays_per_item(), rays)
        net.set_params(p0)
    for s in solvers:
        s.close()
    net.close()
