"""What a solver holds between calls: captured graphs, resident fields and
buffers across changes of the snapshots' number, refused inputs and short device
memory."""
from __future__ import annotations

import numpy as np
import pytest

import dnsmc_gb300 as D
from dnsmc_gb300 import _lib, synth
from oracle import oracle as O

from test_gpu_cv import assert_bitexact_cv
from test_gpu_parity import assert_bitexact, smooth_field
from test_gpu_scatter import check_bitexact, particle_table

pytestmark = pytest.mark.gpu

NI, NJ, NK = 12, 40, 9


def snapshots(n, seed=1):
    T = np.stack([smooth_field(NI, NJ, NK, 450, 1600, seed + f) for f in range(n)])
    rng = np.random.default_rng(seed)
    x = (0.1 + 0.05 * rng.uniform(-1, 1, T.shape)).astype(np.float32)
    fv = (1e-5 * rng.uniform(0.2, 1.0, T.shape)).astype(np.float32)
    fv[:, 0, 0, 0] = 1e-5  # the same largest fraction in every snapshot
    return T, x, fv


def particle_solver(**kw):
    cfg = dict(model=D.MODEL_TABLE, imax=NI, jmax=NJ, kmax=NK, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=0, T_west=400,
               T_east=700, n_groups=2, seed=8, local_sampling=1)
    s = D.Solver(D.default_config(**dict(cfg, **kw)))
    t = synth.ck_table(nbands=8, nq=4, nT=14, nX=4, seed=5)
    s.set_table(t["k"], t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
    s.set_particles(*particle_table(8, 2), 0.4)
    return s


def test_graph_is_captured_again_for_other_field_arrays():
    """Fields of two snapshots take the place of one's arrays; back at one
    snapshot, nothing else that the solve reads has moved."""
    T, x, fv = snapshots(2)
    eager, graph = particle_solver(), particle_solver()
    graph.set_graph(True)
    out = []
    for s in (eager, graph):
        s.set_rays(16)
        s.set_fields(T[0], x[0])
        s.set_particle_field(fv[0])
        first = s.solve(timeout_s=60)
        s.set_fields(T, x)
        s.set_particle_field(fv)
        s.set_fields(T[0], x[0])
        s.set_particle_field(fv[0])
        out.append((first, s.solve(timeout_s=60)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(out[1][0][0], out[1][1][0])
    assert graph.graph_info() == (2, 2)
    eager.close()
    graph.close()


def test_ray_counts_are_read_after_the_kernel_that_sets_them():
    """Adaptive counts, read back at once: the kernel runs on the solver's own
    stream.  (A solve in between must find the same ones.)"""
    n = 64
    T = smooth_field(n, n, n, 450, 1600, 3)
    s = D.Solver(D.default_config(model=D.MODEL_GREY, imax=n, jmax=n, kmax=n, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=0,
                                  T_west=400, T_east=400, kappa=0.5, seed=2))
    s.set_fields(T)
    for per_tau in (40.0, 400.0) * 4:
        s.set_rays_adaptive(per_tau, 8, 4096)
        now = s.rays_per_item()
        s.solve(timeout_s=60)
        np.testing.assert_array_equal(now, s.rays_per_item())
    s.close()


def test_coarse_fields_whatever_follows_the_call():
    """The coarsening's tables are still being copied when set_fields returns:
    solvers of other sizes, whose tables would take freed memory of the same
    kind, must not change them."""
    sizes = ((24, 16, 8), (40, 8, 24), (16, 32, 16))
    cfg = [dict(model=D.MODEL_GREY, imax=a, jmax=b, kmax=c, Lx=2.0 + a, Ly=6.28, Lz=3.14, stretched_x=1, grid_num=3,
                kappa=1.0, T_west=300, T_east=300) for a, b, c in sizes]
    T = [smooth_field(*n, 450, 1300, 9) for n in sizes]
    ref = [[O.coarsen(np.pad(t, 1).ravel(), *n, 2.0 + n[0], 6.28, 3.14, 1, 3, lv)[1:-1, 1:-1, 1:-1] for lv in (1, 2)]
           for n, t in zip(sizes, T)]
    solvers = [D.Solver(D.default_config(**c)) for c in cfg]
    for _ in range(10):
        for s, t in zip(solvers, T):
            s.set_fields(t)
        for s, r in zip(solvers, ref):
            for lv in (1, 2):
                np.testing.assert_array_equal(s.coarse_field(0, lv), r[lv - 1])
    for s in solvers:
        s.close()


def test_sampling_prepared_while_a_solve_is_under_way():
    """The sampling tables rewritten right after solve_async: the solve has its
    own copies of them, and the next one builds them again."""
    T, x, fv = snapshots(1)
    s = particle_solver()
    s.set_rays(64)
    s.set_fields(T, x)
    s.set_particle_field(fv)
    Q, S = s.solve(timeout_s=60)
    for Tmax in (600.0, 1500.0, 900.0):
        s.prepare_sampling(Tmax, 0.05)  # (the solve that follows uploads its tables)
        s.solve_async()
        s.prepare_sampling(Tmax + 50.0, 0.2)
        s.wait(60)
        Q1, S1 = s.results()
        np.testing.assert_array_equal(Q, Q1)
        np.testing.assert_array_equal(S, S1)
    s.close()


def test_coefficients_are_read_back_before_the_first_solve():
    """As many band groups as were set, though no solve has built its sampling
    tables yet."""
    T, x, fv = snapshots(1)
    s = particle_solver(control_variate=1)
    s.set_fields(T, x)
    beta = np.random.default_rng(4).normal(size=(1, 2, NK, NJ, NI, 2)).astype(np.float32)
    s.set_cv_beta(beta)
    np.testing.assert_array_equal(s.cv_beta(), beta)
    s.close()


def test_refused_fractions_of_more_snapshots_leave_the_resident_field():
    """The refused field would need a larger array than the resident one has."""
    T, x, fv = snapshots(3)
    s = particle_solver()
    s.set_rays(16)
    s.set_fields(T[0], x[0])
    s.set_particle_field(fv[0])
    Q, S = s.solve(timeout_s=60)
    s.set_fields(T, x)
    bad = fv.copy()
    bad[2, 3, 5, 7] = -1e-6
    with pytest.raises(RuntimeError, match="volume fractions"):
        s.set_particle_field(bad)
    with pytest.raises(RuntimeError, match="particle field"):
        s.solve(timeout_s=60)  # three snapshots, the resident fractions are one's
    s.set_fields(T[0], x[0])
    Q1, S1 = s.solve(timeout_s=60)
    np.testing.assert_array_equal(Q, Q1)
    np.testing.assert_array_equal(S, S1)
    s.close()


@pytest.mark.parametrize("kind", ["grey walls", "grey particles", "bands", "particles cv", "levels"])
def test_a_closed_solver_leaves_no_device_memory_behind(kind):
    """Ten solvers one after the other: an array left behind by each (a padded
    field of these 64^3 cells is 2 MB and more) would show."""
    torch = pytest.importorskip("torch")
    n = 64
    T = smooth_field(n, n, n, 450, 1300, 2)

    def cycle():
        cfg = dict(imax=n, jmax=n, kmax=n, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=0, T_west=400, T_east=400, kappa=1.0)
        if kind == "particles cv":
            s = particle_solver(**dict(cfg, control_variate=1, model=D.MODEL_TABLE))
            s.set_fields(T, np.full(T.shape, 0.1, np.float32))
            s.set_particle_field(np.full(T.shape, 1e-6, np.float32))
        else:
            s = D.Solver(D.default_config(model=D.MODEL_GREY_BANDS if kind == "bands" else D.MODEL_GREY,
                                          **dict(cfg, eps_west=0.5 if kind == "grey walls" else 1.0,
                                                 grid_num=3 if kind == "levels" else 1)))
            if kind == "bands":
                s.use_grey_band_tables(40, 12, 15000.0, 500.0)
            s.set_fields(T)
            if kind == "grey particles":
                s.set_particles(np.array([0.5e5], np.float32), np.array([1.0e5], np.float32), 0.3)
                s.set_particle_field(np.full(T.shape, 1e-6, np.float32))
        s.set_graph(kind != "levels")
        s.set_rays(2)
        s.solve(timeout_s=60)
        s.close()
        return torch.cuda.mem_get_info()[0]

    cycle()
    first = cycle()
    for _ in range(9):
        last = cycle()
    assert first - last < 10 << 20, (first, last)


def test_only_the_plain_grey_march_has_its_field_prepared():
    """Grey walls and particles march on an array of their own: set_fields
    writes T^4 for black walls and gas alone, and a solve that turns to them
    afterwards writes it then."""
    T, _, fv = snapshots(1)
    T, fv = T[0], fv[0]
    cfg = dict(model=D.MODEL_GREY, imax=NI, jmax=NJ, kmax=NK, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=0, T_west=400,
               T_east=700, kappa=0.8, seed=4)

    def launches(s):
        n0 = _lib.launch_count()
        s.set_fields(T)
        return _lib.launch_count() - n0

    black, grey = D.Solver(D.default_config(**cfg)), D.Solver(D.default_config(eps_west=0.5, **cfg))
    assert launches(black) == 2 and launches(grey) == 1
    black.set_rays(8)
    Q, S = black.solve(timeout_s=60)
    s = D.Solver(D.default_config(**cfg))
    s.set_rays(8)
    s.set_particles(np.array([0.5e5], np.float32), np.array([1.0e5], np.float32), 0.3)
    assert launches(s) == 1
    s.set_particle_field(fv)
    s.solve(timeout_s=60)
    s.set_particles(None, None)
    Q1, S1 = s.solve(timeout_s=60)
    np.testing.assert_array_equal(Q, Q1)
    np.testing.assert_array_equal(S, S1)
    for s in (s, black, grey):
        s.close()


@pytest.mark.parametrize("kw", [dict(), dict(eps_west=0.5), dict(control_variate=1), dict(grid_num=2)],
                         ids=["gas", "walls", "cv", "levels"])
def test_the_longest_grey_band_tables(kw):
    """3489 temperatures: a sample's k and Ib (2 x 3488 pairs) in each of four
    warps, with 64 bytes a thread and 1 KB beside them, are all of the shared
    memory; one temperature more is refused."""
    ni, nj, nk = 8, 16, 8
    T = smooth_field(ni, nj, nk, 600, 1500, 3)
    for nT in (3489, 3490):
        s = D.Solver(D.default_config(model=D.MODEL_GREY_BANDS, imax=ni, jmax=nj, kmax=nk, Lx=1.5, Ly=2.0, Lz=0.7,
                                      stretched_x=0, T_west=500.0, T_east=700.0, kappa=0.7, seed=12, **kw))
        s.use_grey_band_tables(3, nT, 15000.0, 500.0)
        s.set_fields(T)
        s.set_rays(16)
        if nT == 3490:
            with pytest.raises(RuntimeError, match="shared memory"):
                s.solve(timeout_s=60)
        elif "grid_num" in kw or "eps_west" in kw:
            Q, S = s.solve(timeout_s=60)
            assert np.isfinite(Q).all() and s.status() == 0
        else:
            (assert_bitexact_cv if "control_variate" in kw else assert_bitexact)(s, T)
        s.close()


@pytest.mark.parametrize("nX,kw", [
    (14, dict()), (15, dict(control_variate=1, cv_moments=1)),   # two blocks of fewer than 8 warps an SM
    (34, dict()), (34, dict(block_threads=256)),                 # 8 warps no longer fit
    (50, dict(control_variate=1)), (71, dict(block_threads=128)),  # down to 3 warps
])
def test_table_slabs_that_leave_room_for_fewer_warps(nX, kw):
    ni, nj, nk = 9, 17, 10
    s = D.Solver(D.default_config(model=D.MODEL_TABLE, imax=ni, jmax=nj, kmax=nk, Lx=1.5, Ly=2.0, Lz=0.7, stretched_x=0,
                                  T_west=500.0, T_east=700.0, n_groups=2, local_sampling=1, seed=3,
                                  sampler=D.SAMPLER_RQMC, nvar=2, **kw))
    t = synth.ck_table(nbands=4, nq=2, nT=50, nX=nX, seed=5)
    s.set_table(t["k"], t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
    T = smooth_field(ni, nj, nk, 600, 1500, 3)
    x = np.random.default_rng(1).uniform(0.05, 0.2, T.shape).astype(np.float32)
    s.set_fields(T, x)
    s.set_rays(16)
    (assert_bitexact_cv if "control_variate" in kw else assert_bitexact)(s, T, x)
    s.close()


def test_particles_and_a_table_slab_that_leaves_room_for_fewer_warps():
    T, x, fv = snapshots(1)
    s = particle_solver(nvar=1)
    t = synth.ck_table(nbands=8, nq=4, nT=50, nX=33, seed=5)
    s.set_table(t["k"], t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])
    s.set_fields(T, x)
    s.set_particle_field(fv)
    s.set_rays(8)
    check_bitexact(s, T, x, fv)
    s.close()


def test_a_split_solve_runs_where_its_contributions_have_no_room(monkeypatch):
    """32^3 cells, 256 rays: the rays' contributions of the split items are 34
    MB, all other arrays together under 8 MB.  The sums are the same without."""
    n = 32
    T = smooth_field(n, n, n, 450, 1300, 2)

    def solver():
        s = D.Solver(D.default_config(model=D.MODEL_GREY, imax=n, jmax=n, kmax=n, Lx=2.0, Ly=6.28, Lz=3.14,
                                      stretched_x=0, T_west=400, T_east=400, kappa=1.0, seed=6))
        s.set_rays(256)
        return s

    s = solver()
    s.set_fields(T)
    ref = s.solve(timeout_s=60)
    # 16 snapshots: 0.52 M cells of 68 bytes (fields, tallies, results), 36 MB, in
    # part where the last solve's contributions were: they are given up
    monkeypatch.setenv("DNSMC_TEST_DEVICE_BYTES", str(44 << 20))
    many = np.stack([T] * 16)
    s.set_fields(many)
    Q, S = s.solve(timeout_s=60)
    np.testing.assert_array_equal(Q[0], ref[0][0])
    s.close()
    ran = []
    for mb in (1, 2, 4, 8, 16, 24, 32, 40, 64):
        monkeypatch.setenv("DNSMC_TEST_DEVICE_BYTES", str(mb << 20))
        s = solver()
        try:
            s.set_fields(T)
            Q, S = s.solve(timeout_s=60)
            Q2, S2 = s.solve(timeout_s=60)
        except RuntimeError as e:
            assert "cudaMalloc" in str(e)
        else:
            ran.append(mb)
            for a, b in ((Q, ref[0]), (S, ref[1]), (Q2, ref[0]), (S2, ref[1])):
                np.testing.assert_array_equal(a, b)
            assert s.status() == 0
        s.close()
    assert ran == [8, 16, 24, 32, 40, 64] or ran == [4, 8, 16, 24, 32, 40, 64]


def test_results_after_a_solve_that_did_not_fit(monkeypatch):
    """Half a grid solved, then the whole one with too little device memory, a
    little more each time: what is read afterwards are the half's results or an
    error, never the contents of an array that was being replaced."""
    n = 64
    T = smooth_field(n, n, n, 450, 1300, 2)
    s = D.Solver(D.default_config(model=D.MODEL_GREY, imax=n, jmax=n, kmax=n, Lx=2.0, Ly=6.28, Lz=3.14, stretched_x=0,
                                  T_west=400, T_east=400, kappa=1.0, seed=6))
    s.set_fields(T)
    s.set_rays(2)
    half, whole = (0, n, 0, n, 0, n // 2), (0, n, 0, n, 0, n)
    s.set_region(*half)
    ref = s.solve(timeout_s=60)
    steps = s.item_steps()
    seen = []
    for kb in range(1 << 10, 40 << 10, 1 << 10):  # 0.26 M cells of 68 bytes: 18 MB for the whole grid
        monkeypatch.setenv("DNSMC_TEST_DEVICE_BYTES", str(kb << 10))
        s.set_region(*whole)
        try:
            full = s.solve(timeout_s=60)
            break
        except RuntimeError as e:
            assert "cudaMalloc" in str(e)
        s.set_region(*half)
        try:
            Q, S = s.results()
        except RuntimeError as e:
            assert "no solve" in str(e)
            with pytest.raises(RuntimeError, match="no solve"):
                s.item_steps()
            seen.append("error")
            continue
        np.testing.assert_array_equal(Q, ref[0])
        np.testing.assert_array_equal(S, ref[1])
        np.testing.assert_array_equal(s.item_steps(), steps)
        seen.append("results")
    assert "error" in seen
    monkeypatch.delenv("DNSMC_TEST_DEVICE_BYTES")
    other = D.Solver(s.cfg)
    other.set_fields(T)
    other.set_rays(2)
    for a, b in zip(full, other.solve(timeout_s=60)):
        np.testing.assert_array_equal(a, b)
    other.close()
    s.close()
