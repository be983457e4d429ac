"""The correlated-k table generator on the GPU (dnsmc_ck_from_lbl) against
the oracle's restatement (orc_ck_from_lbl), which is itself checked against
the reference's compiled correlatedKT (tests/test_ckgen.py).

The bin counts and the g-function are integer and fixed-order work, the bin
values products: the GPU's k at the g-points equals the oracle's but for the
rare interval whose k^0.1 falls within a rounding of a bin edge (the device's
and the host's power functions may round differently); the band means agree
to rounding.  A generated table then drives a solve.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

import dnsmc_gb300 as D
from dnsmc_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_gpu_generator_matches_the_oracle():
    T = np.linspace(400.0, 2000.0, 9)
    spec = synth.lbl_spectrum(T, (0.05, 0.15, 0.3), nbands=5, band_width=20.0, lines_per_band=30, seed=11)
    gq, wq = synth.gauss_legendre_half(16)
    kq, kavg = D.ck_from_lbl(spec, gq, n_pwrk=10000)
    ko, ao = O.ck_from_lbl(spec, gq, n_pwrk=10000)
    assert (kq == ko).mean() > 0.99
    np.testing.assert_allclose(kq, ko, rtol=1e-5)
    np.testing.assert_allclose(kavg, ao, rtol=1e-9)
    assert (np.diff(kq, axis=1) >= 0).all()


def test_generated_table_drives_a_solve():
    T = np.linspace(300.0, 2100.0, 10)
    X = np.array([0.0, 0.1, 0.2, 0.3])
    spec = synth.lbl_spectrum(T, X, nbands=4, band_width=25.0, lines_per_band=30, seed=5)
    gq, wq = synth.gauss_legendre_half(16)
    kq, _ = D.ck_from_lbl(spec, gq, n_pwrk=10000)
    ni, nj, nk = 16, 32, 8
    s = D.Solver(D.default_config(model=D.MODEL_TABLE, imax=ni, jmax=nj, kmax=nk, Lx=2.0, Ly=2 * math.pi,
                                  Lz=math.pi, stretched_x=0, T_west=400.0, T_east=400.0, n_groups=2, seed=3,
                                  sampler=D.SAMPLER_RQMC, nvar=2, local_sampling=1))
    s.set_table(kq, spec["wvc"].astype(np.float32), float(T[0]), float(T[1] - T[0]),
                dnu=np.full(4, 25.0, np.float32), wq=wq.astype(np.float32), X0=0.0, dX=0.1)
    d = synth.ck_channel(32, 2)
    Tf = np.ascontiguousarray(d["T"][:nk, :, :ni])
    xf = np.ascontiguousarray(d["x"][:nk, :, :ni])
    s.set_fields(Tf, xf)
    s.set_rays(32)
    Q, S = s.solve(timeout_s=120)
    assert np.isfinite(Q).all() and np.abs(Q).max() > 0 and s.status() == 0
    s.close()


@pytest.mark.parametrize("n_pwrk", [2, 3, 777, 10000, 50000])
def test_bins_of_awkward_spectra(n_pwrk):
    """Points are binned in FP32 where that decides the bin: bands that are flat
    to 1e-13, that span sixty decades, hold zeros and subnormals, two points,
    or lie beyond FP32's range, against the oracle (bounds as above)."""
    rng = np.random.default_rng(4)
    n = 4001
    smooth = np.exp(3.0 * np.sin(np.linspace(0, 40, n)))
    rows = [smooth, 0.3 * (1 + 1e-13 * rng.integers(0, 9, n)), 10.0 ** rng.uniform(-30, 30, n),
            np.where(rng.random(n) < 0.2, 0.0, smooth), smooth * 1e-35, smooth * 1e-310, smooth * 1e60,
            1.0 + 1e-5 * smooth, np.full(n, 2.5)]
    k = np.stack(rows)[:, None, :]
    spec = dict(kappa=k, wv0=1000.0, dwv=0.01, first=np.array([0, 1500, 3999], np.int64),
                count=np.array([1501, 2500, 2], np.int32), wv_left=np.array([1000.0, 1015.0, 1039.99]),
                wv_right=np.array([1015.0, 1040.0, 1040.0]))
    gq, _ = synth.gauss_legendre_half(16)
    kq, kavg = D.ck_from_lbl(spec, gq, n_pwrk=n_pwrk)
    ko, ao = O.ck_from_lbl(spec, gq, n_pwrk=n_pwrk)
    np.testing.assert_allclose(kq, ko, rtol=1e-5)
    np.testing.assert_allclose(kavg, ao, rtol=1e-9)


@pytest.mark.parametrize("nT,nX", [(5, 3), (3, 1), (1, 14)])
def test_spectra_copied_in_parts_equal_single_rows(nT, nX):
    """From 8 MB on the spectra are copied and reduced in parts; every (T, x)
    row equals the row generated alone, and a bad value in the last part is
    refused."""
    per = 9000 if nT * nX > 3 else 88000
    nb = 9 if nT * nX > 3 else 4
    n = nb * per + 1
    assert nT * nX * n * 8 >= 8 << 20 and n * 8 < 8 << 20
    k = np.exp(np.random.default_rng(nT).normal(-2.0, 2.0, (nT, nX, n)))
    left = 1000.0 + per * 0.01 * np.arange(nb)
    spec = dict(kappa=k, wv0=1000.0, dwv=0.01, first=np.arange(nb, dtype=np.int64) * per,
                count=np.full(nb, per + 1, np.int32), wv_left=left, wv_right=left + per * 0.01)
    gq = np.array([0.1, 0.5, 0.9])
    kq, kavg = D.ck_from_lbl(spec, gq, n_pwrk=500)
    for t in range(nT):
        for x in range(nX):
            q1, a1 = D.ck_from_lbl(dict(spec, kappa=k[t:t + 1, x:x + 1]), gq, n_pwrk=500)
            np.testing.assert_array_equal(kq[..., t, x], q1[..., 0, 0])
            np.testing.assert_array_equal(kavg[t, x], a1[0, 0])
    k[-1, -1, -1] = np.nan
    with pytest.raises(RuntimeError, match="finite"):
        D.ck_from_lbl(spec, gq, n_pwrk=500)
