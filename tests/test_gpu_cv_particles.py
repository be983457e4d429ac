"""E[Y] of the control variate with particles: the node sums against the
per-sample float64 sums of the definition (the tolerance of the gas's own test:
the cells' FP32 table fractions, 1e-4)."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from dnsmc_gb300 import synth

from test_capi import alias_distribution
from test_gpu_parity import smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nX,groups", [(4, 3), (1, 1), (2, 2)])
def test_means_with_particles_match_their_definition(nX, groups):
    nq, nT, ni, nj, nk = 4, 20, 11, 20, 5
    tb = synth.ck_table(nbands=7, nq=nq, nT=nT, nX=max(nX, 4), seed=13)
    kk = np.ascontiguousarray(tb["k"][..., 2] if nX == 1 else tb["k"][..., :nX])
    s = D.Solver(D.default_config(model=D.MODEL_TABLE, imax=ni, jmax=nj, kmax=nk, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=1,
                                  T_west=420, T_east=380, eps_west=0.7, seed=17, n_groups=groups, control_variate=1))
    s.set_table(kk, tb["wvc"], tb["T0"], tb["dT"], dnu=tb["dnu"], wq=tb["wq"], X0=tb["X0"], dX=tb["dX"])
    T = smooth_field(ni, nj, nk, 450, 1700, 23)
    rng = np.random.default_rng(2)
    x = None if nX == 1 else rng.uniform(0.01, 0.07, T.shape).astype(np.float32)
    fv = rng.uniform(0.0, 2e-5, T.shape).astype(np.float32)
    part = (np.linspace(1e4, 6e4, 7).astype(np.float32), np.linspace(2e4, 1e4, 7).astype(np.float32), 0.4)
    s.set_fields(T, x)
    s.set_particles(*part)
    s.set_particle_field(fv)
    s.set_rays(8)
    s.solve(timeout_s=60)
    cv, smp, t = s.cv_data(), s.sampling(), s.table()
    Tg = tb["T0"] + tb["dT"] * np.arange(nT)
    Xg = tb["X0"] + tb["dX"] * np.arange(nX)
    scale = np.abs(cv["muY"]).max()
    for (i, j, k) in ((0, 0, 0), (5, 9, 1), (10, 19, 4)):
        for g in range(groups):
            p = alias_distribution(smp, g)
            a, e_ = int(smp["group_start"][g]), int(smp["group_start"][g + 1])
            acc = accB = 0.0
            for e in range(a, e_):
                b, gq = smp["band"][e], smp["gq"][e]
                kx = t["k"][b, gq, :, 0] if nX == 1 else [np.interp(x[k, j, i], Xg, t["k"][b, gq, it]) for it in range(nT)]
                ki = np.interp(T[k, j, i], Tg, kx) + float(fv[k, j, i]) * float(part[0][b])
                ib = np.interp(T[k, j, i], Tg, t["Ib"][b])
                sid = b * nq + gq
                C = smp["W"][e] * p[e - a]
                acc += C * ki * (ib - cv["Jhat"][0, sid, i, 0])
                accB += C * ki * (ib - cv["sur"][0, sid, i, 1]) * cv["Jhat"][0, sid, i, 1]
            mu = cv["muY"][0, g, k, j, i]
            assert abs(mu[0] - acc) <= 1e-4 * abs(acc) + 1e-9 * scale
            assert abs(mu[1] - accB) <= 1e-4 * abs(accB) + 1e-9 * scale
    s.close()
