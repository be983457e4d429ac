"""The gas march's walk generator and padded fields, bit for bit against the
host replay, where they can go wrong: periodic axes shorter than a packet or a
slice's crossings, ragged regions, walks of several chunks (thin media), step
caps inside and at the end of a chunk, packets as rows, every table kind."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from dnsmc_gb300 import synth

from test_gpu_parity import assert_bitexact, smooth_field
from test_gpu_cv import assert_bitexact_cv

pytestmark = pytest.mark.gpu

# model, (ni, nj, nk), overrides, region
CASES = [
    ("grey", (6, 1, 1), dict(kappa=0.3), None),
    ("grey", (9, 3, 2), dict(kappa=0.01), None),
    ("grey", (40, 5, 11), dict(kappa=0.02, max_steps=65), None),
    ("grey", (33, 70, 9), dict(kappa=0.5, stretched_x=1, tile_a=32), (3, 30, 7, 70, 1, 9)),
    ("grey", (150, 8, 8), dict(kappa=0.05, max_steps=64), None),
    ("bands", (21, 19, 10), dict(kappa=0.05), None),
    ("bands", (12, 2, 37), dict(kappa=4.0, stretched_x=1), (0, 12, 0, 2, 5, 36)),
    ("T", (37, 9, 8), dict(max_steps=33), None),
    ("T", (17, 33, 3), dict(tile_a=8), (0, 17, 20, 33, 0, 3)),
    ("TX", (70, 6, 9), dict(toll=1e-6), None),
    ("TX", (11, 41, 13), dict(stretched_x=1, n_groups=3, local_sampling=1), (2, 9, 1, 40, 0, 13)),
    ("TXcv", (23, 10, 15), dict(n_groups=2, local_sampling=1, control_variate=1), None),
    ("greycv", (64, 7, 8), dict(kappa=0.1, control_variate=1), None),
]


@pytest.mark.parametrize("model,size,kw,region", CASES)
def test_walks_match_the_replay(model, size, kw, region):
    ni, nj, nk = size
    kind = model.replace("cv", "")
    cfg = dict(model={"grey": D.MODEL_GREY, "bands": D.MODEL_GREY_BANDS}.get(kind, D.MODEL_TABLE), imax=ni, jmax=nj,
               kmax=nk, Lx=1.5, Ly=2.0, Lz=0.7, stretched_x=0, T_west=500.0, T_east=700.0, seed=321,
               sampler=D.SAMPLER_RQMC, nvar=2)
    cfg.update(kw)
    s = D.Solver(D.default_config(**cfg))
    x = None
    T = smooth_field(ni, nj, nk, 600, 1500, 3)
    if kind == "bands":
        s.use_grey_band_tables(40, 12, 15000.0, 500.0)
    elif kind in ("T", "TX"):
        t = synth.ck_table(nbands=6, nq=4, nT=14, nX=4, seed=5)
        if kind == "T":
            s.set_table(t["k"][..., 2] * 0.05, t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"])
        else:
            s.set_table(t["k"] * 0.05, t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
            x = np.full(T.shape, 0.12, np.float32) + 0.05 * np.random.default_rng(1).uniform(-1, 1, T.shape).astype(np.float32)
    s.set_fields(T, x)
    if region:
        s.set_region(*region)
    s.set_rays(14)
    status = s.status
    if "max_steps" in kw:  # the comparison holds for capped rays too; the cap itself is reported
        s.status = lambda: status() & ~D.STATUS_STEP_CAP
    (assert_bitexact_cv if model.endswith("cv") else assert_bitexact)(s, T, x)
    assert status() == (D.STATUS_STEP_CAP if "max_steps" in kw else 0)
    s.close()


def test_traces_of_several_chunks_match_the_replay():
    """Walks beyond one chunk, recorded step by step; the packet shape changed
    by the region after the solve."""
    from oracle import oracle as O
    s = D.Solver(D.default_config(model=D.MODEL_GREY, imax=90, jmax=12, kmax=16, Lx=2.0, Ly=0.8, Lz=0.6, stretched_x=1,
                                  T_west=400, T_east=500, kappa=0.02, seed=8))
    T = smooth_field(90, 12, 16, 600, 1000, 2)
    s.set_fields(T)
    s.set_rays(8)
    s.solve(timeout_s=60)
    for region in (None, (0, 90, 0, 12, 3, 9)):
        if region:
            s.set_region(*region)
        c, keep = O.packet_config(s, T, None)
        longest = 0
        for p, r in [(0, 0), (s.packet_count() - 1, 3), (s.packet_count() // 2, 7), (5, 1)]:
            rec, n, rng = s.trace(0, 0, p, r)
            rec2, n2, rng2 = O.packet_trace(c, 0, 0, p, r)
            assert n == n2
            np.testing.assert_array_equal(rng, rng2)
            np.testing.assert_array_equal(rec, rec2)
            longest = max(longest, n)
        assert longest > 64
    s.close()


@pytest.mark.parametrize("size,groups,rays,sampler", [
    ((5, 9, 8), 1, 37, D.SAMPLER_IID),       # a unit per ray
    ((40, 24, 24), 2, 50, D.SAMPLER_RQMC),   # 720 items: uneven units
    ((64, 64, 40), 1, 26, D.SAMPLER_RQMC),   # 2560 items: units of several rays
    ((96, 72, 64), 8, 2, D.SAMPLER_RQMC),    # 55296 items: a unit per item
])
def test_split_items_match_the_replay(size, groups, rays, sampler):
    """Items of few-item solves are split over queue units by rays: the sums
    are the replay's bit for bit."""
    ni, nj, nk = size
    t = synth.ck_table(nbands=8, nq=4, nT=24, nX=4, seed=9)
    s = D.Solver(D.default_config(model=D.MODEL_TABLE, imax=ni, jmax=nj, kmax=nk, Lx=1.0, Ly=2.0, Lz=2.0, stretched_x=0,
                                  T_west=500.0, T_east=600.0, seed=5, sampler=sampler, nvar=2, n_groups=groups,
                                  local_sampling=1))
    s.set_table(t["k"] * 0.05, t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
    T = smooth_field(ni, nj, nk, 600, 1500, 3)
    x = np.full(T.shape, 0.1, np.float32)
    s.set_fields(T, x)
    s.set_rays(rays)
    assert_bitexact(s, T, x)
    c = s.counters()
    assert c.rays == ni * nj * nk * groups * rays
    s.close()


# kind, (ni, nj, nk), albedo scale of the particles, overrides, region
GEN_CASES = [
    ("grey", (9, 3, 2), 1.0, dict(kappa=0.05, eps_east=0.3), None),
    ("grey", (40, 5, 11), 0.1, dict(kappa=0.02, max_steps=65), None),
    ("grey", (60, 8, 8), 0.0, dict(kappa=0.05, eps_west=0.2, eps_east=0.2), None),       # no scattering: reflections only
    ("T", (17, 33, 9), 5.0, dict(eps_west=0.9, tile_a=16, max_steps=40), (1, 16, 3, 31, 0, 9)),
    ("TX", (70, 6, 9), 0.3, dict(toll=1e-5), None),
    ("TX", (13, 26, 19), 1.0, dict(stretched_x=1, n_groups=2, local_sampling=1, control_variate=1, cv_moments=1), None),
    ("TX", (48, 64, 40), 1.0, dict(n_groups=8, eps_west=0.8), None),                     # a unit per item
]


@pytest.mark.parametrize("kind,size,albedo,kw,region", GEN_CASES)
def test_general_medium_walks_match_the_replay(kind, size, albedo, kw, region):
    """Chunks that end at collisions, walls and caps; restarts from any point of
    a cell; packed fields with the volume fraction; split and whole items."""
    from test_gpu_scatter import check_bitexact, particle_table
    ni, nj, nk = size
    cfg = dict(model=D.MODEL_GREY if kind == "grey" else D.MODEL_TABLE, imax=ni, jmax=nj, kmax=nk, Lx=1.5, Ly=2.0, Lz=0.7,
               stretched_x=0, T_west=500.0, T_east=700.0, seed=77, sampler=D.SAMPLER_RQMC, nvar=2)
    cfg.update(kw)
    s = D.Solver(D.default_config(**cfg))
    T, x, nb = smooth_field(ni, nj, nk, 600, 1500, 3), None, 1
    rng = np.random.default_rng(5)
    if kind != "grey":
        t = synth.ck_table(nbands=8, nq=4, nT=24, nX=4, seed=5)
        nb = 8
        if kind == "T":
            s.set_table(t["k"][..., 2] * 0.05, t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"])
        else:
            s.set_table(t["k"] * 0.05, t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
            x = (0.12 + 0.05 * rng.uniform(-1, 1, T.shape)).astype(np.float32)
    s.set_fields(T, x)
    a, sc = particle_table(nb)
    fv = rng.uniform(0.0, 2e-5, T.shape).astype(np.float32)
    s.set_particles(a, sc * albedo, -0.3)
    s.set_particle_field(fv)
    if region:
        s.set_region(*region)
    s.set_rays(2 if ni * nj * nk > 1e5 else 10)
    status = s.status
    if "max_steps" in kw:
        s.status = lambda: status() & ~D.STATUS_STEP_CAP
    check_bitexact(s, T[None], None if x is None else x[None], fv[None])
    assert status() == (D.STATUS_STEP_CAP if "max_steps" in kw else 0)
    s.close()


@pytest.mark.parametrize("model,size,kw", [
    ("grey", (200, 8, 8), dict(kappa=0.01, max_steps=128)),   # the cap at a chunk's end, and one step on
    ("grey", (200, 8, 8), dict(kappa=0.01, max_steps=129)),
    ("grey", (64, 3, 64), dict(kappa=0.02)),                  # as many planes as a chunk lists crossings
    ("bands", (131, 9, 6), dict(kappa=0.03)),
    ("T", (150, 5, 8), dict(max_steps=129)),
    ("T", (150, 5, 8), dict(max_steps=128)),
    ("grey", (300, 8, 8), dict(kappa=0.005, max_steps=192)),  # (uniform absorption takes longer chunks)
    ("bands", (300, 6, 9), dict(kappa=0.005, max_steps=193)),
])
def test_walks_at_the_edges_of_a_chunk_match_the_replay(model, size, kw):
    test_walks_match_the_replay(model, size, kw, None)


@pytest.mark.parametrize("nT", [2, 3, 4, 55])
def test_band_tables_that_end_below_the_field_match_the_replay(nT):
    """With few temperatures the grey band tables end below the field's
    maximum: cells at the table's end point, and at its first point."""
    s = D.Solver(D.default_config(model=D.MODEL_GREY_BANDS, imax=14, jmax=12, kmax=9, Lx=1.5, Ly=2.0, Lz=0.7, stretched_x=0,
                                  T_west=500.0, T_east=700.0, kappa=0.7, seed=12, sampler=D.SAMPLER_RQMC, nvar=2))
    s.use_grey_band_tables(40, nT, 15000.0, 900.0)
    T = smooth_field(14, 12, 9, 600, 1500, 3)
    s.set_fields(T)
    s.set_rays(14)
    assert_bitexact(s, T)
    assert s.status() == 0
    s.close()
