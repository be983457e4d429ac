"""What a network holds between calls: inputs and permutations on their way to
the device, chained training steps, work buffers shared by several solvers."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from oracle import cvnet_oracle as NO

from test_gpu_cvnet import make_labels, random_params, small_table, table_solver
from test_gpu_parity import smooth_field

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


def training_net(batch, **kw):
    """A network with the 1536 rows of one small solve."""
    s = table_solver(small_table(), 12, 32, 4, sampler=D.SAMPLER_RQMC, nvar=4, local_sampling=1, control_variate=1,
                     cv_moments=1, seed=5)
    x = (0.1 + 0.05 * np.random.default_rng(3).uniform(-1, 1, (4, 32, 12))).astype(np.float32)
    s.set_fields(smooth_field(12, 32, 4, 450, 1700, 8), x)
    s.set_rays(16)
    s.solve(timeout_s=60)
    net = D.CvNet(D.cvnet_default_config(n_groups=8, batch=batch, seed=9, **kw))
    net.add_training_data(s)
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
