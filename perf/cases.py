"""What the solver's speed is measured on: the calls a user's program makes.

Every case is one whole call (or the short sequence of calls a program repeats
per snapshot) through the public entry points: fields in, radiative source
out; a training pass; a spectral-table build.  Listed sizes come from the
benchmark's workloads (grey 64^3, correlated-k 128^3, batched and particle
96^3 snapshots), the defaults of the drop-in pair and the tests' small grids;
drawn cases spread over the same ranges.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os

import numpy as np
import torch

import dnsmc_gb300 as D
from dnsmc_gb300 import _lib, cvtrain, synth

NET = os.path.join(os.path.dirname(os.path.abspath(D.__file__)), "nets", "ck128_g8.cvnet")
SIGMA = 5.670373e-08


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a few cells and rays, as a smoke check or a unit
        # test of a coupled code makes; latency and launches count
        dict(name="grey_8x32x4", kind="grey", ni=8, nj=32, nk=4, rays=32, rqmc=False, f32=False),
        # a coarse grey grid that is already resident on the GPU, solved there
        # without allocating (a host code whose pool owns the device memory)
        dict(name="grey_resident_32", kind="noalloc", ni=32, nj=32, nk=32, rays=60),
        # the grey channel at the configuration's 256 rays per cell
        dict(name="grey_64", kind="grey", ni=64, nj=64, nk=64, rays=256, rqmc=True, f32=True),
        # the reference's own call surface: the DNS hands over its Fortran
        # array every few steps and collects Q and sigma (grey band tables)
        dict(name="dropin_bands_64", kind="bands", ni=64, nj=64, nk=64, rays=396, p_row=1),
        # the reference's shipped multigrid (five levels, five steps a level)
        dict(name="multigrid_64", kind="mg", ni=64, nj=64, nk=64, rays=60, levels=5),
        # the flagship: correlated-k channel, learned control variate and ray
        # allocation at the 1 % budget (48 rays a cell and band group)
        dict(name="ck_net_128", kind="net", ni=128, nj=128, nk=128, rays=48),
        # several snapshots at once: one graph-replayed launch, rays by optical
        # thickness with the floor of 64, profile control variate
        dict(name="ck_batch_4x96", kind="batch", ni=96, nj=96, nk=96, fields=4, rays=64, nbands=64, nq=16, nT=50, nX=8),
        # ragged sizes, a small table, FP64 results
        dict(name="ck_ragged_45x60x52", kind="ck", ni=45, nj=60, nk=52, rays=32, nbands=16, nq=8, nT=24, nX=5, groups=4,
             rqmc=True),
        # tables without an x_H2O axis, plain Monte Carlo sampled at Tmax: the
        # reference's own estimator and table sizes (119 bands, 16 g-points)
        dict(name="ck_plain_96x64x64", kind="plain", ni=96, nj=64, nk=64, rays=60, nbands=119, nq=16, nT=52),
        # scattering particles between grey walls
        dict(name="particles_96", kind="particles", ni=96, nj=96, nk=96, rays=8),
        # a training pass of the control-variate network over resident data
        dict(name="net_train_128k", kind="train", ni=64, nj=64, nk=32, batch=4096),
        # a correlated-k table from line-by-line spectra: the reference's 52
        # temperatures and 10000 bins, bands of 25 1/cm at 0.01 1/cm
        dict(name="lbl_table_52x32", kind="lbl", nT=52, nX=1, nbands=32, points=2500, bins=10000),
    ]


def _log(rng, lo, hi, even=False):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    v = min(max(v, lo), hi)
    return v - v % 2 if even else v


def draw(rng):
    kind = rng.choice(["grey", "grey", "noalloc", "bands", "mg", "net", "batch", "ck", "ck", "plain", "particles", "train",
                       "lbl"])
    ni, nj, nk = (_log(rng, 8, 80) for _ in range(3))
    rays = _log(rng, 16, 256, even=True)
    c = dict(kind=kind, ni=ni, nj=nj, nk=nk, rays=rays)
    if kind == "grey":
        c.update(rqmc=rng.random() < 0.5, f32=rng.random() < 0.5)
    elif kind == "noalloc":
        c.update(ni=_log(rng, 8, 64), nj=_log(rng, 8, 64), nk=_log(rng, 3, 64))
    elif kind == "bands":
        c.update(p_row=rng.choice([1, 1, 2]), nj=max(2, nj - nj % 2))
    elif kind == "mg":
        levels = rng.choice([2, 3, 5])
        r = 1 << (levels - 1)
        c.update(ni=max(r, ni - ni % r), nj=max(r, nj - nj % r), nk=max(r, nk - nk % r), levels=levels)
    elif kind == "net":
        c.update(ni=_log(rng, 24, 100), nj=_log(rng, 24, 100), nk=_log(rng, 24, 100), rays=_log(rng, 16, 64, even=True))
    elif kind == "batch":
        c.update(fields=rng.randint(2, 6), ni=_log(rng, 16, 64), nj=_log(rng, 16, 64), nk=_log(rng, 16, 64), rays=64,
                 nbands=rng.choice([16, 32, 64]), nq=rng.choice([8, 16]), nT=rng.randint(20, 60), nX=rng.randint(3, 10))
    elif kind == "ck":
        c.update(rays=_log(rng, 8, 96, even=True), nbands=rng.randint(6, 70), nq=rng.choice([4, 8, 16]), nT=rng.randint(12, 60),
                 nX=rng.randint(2, 10), groups=rng.randint(1, 6), rqmc=rng.random() < 0.6)
    elif kind == "plain":
        c.update(nbands=rng.randint(10, 130), nq=rng.choice([1, 8, 16]), nT=rng.randint(12, 60))
    elif kind == "particles":
        c.update(rays=_log(rng, 4, 32, even=True))
    elif kind == "train":
        c.update(ni=_log(rng, 16, 64), nj=_log(rng, 16, 64), nk=_log(rng, 8, 32), batch=128 * _log(rng, 2, 48))
        del c["rays"]
    else:
        c = dict(kind="lbl", nT=_log(rng, 2, 52), nX=rng.randint(1, 4), nbands=_log(rng, 2, 32), points=_log(rng, 400, 2500),
                 bins=rng.choice([1000, 10000]))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _field(c, seed, T_wall, T_rise):
    """T = (T_wall + T_rise (1 - y^2)) (1 + 5 % Fourier), [nk][nj][ni]."""
    y = synth.cell_centres(c["ni"], synth.LY) - 1.0
    f = synth.fourier_fluct(c["ni"], c["nj"], c["nk"], seed)
    return np.ascontiguousarray((T_wall + T_rise * (1.0 - y * y))[None, None, :] * (1.0 + 0.05 * f), dtype=np.float32)


def _h2o(c, seed):
    return np.ascontiguousarray(0.1 + 0.05 * synth.fourier_fluct(c["ni"], c["nj"], c["nk"], seed + 1000), dtype=np.float32)


@functools.lru_cache(maxsize=4)
def _table(nbands, nq, nT, nX):
    return synth.ck_table(nbands, nq, nT, nX)


def _config(c, model, T_wall, seed, **kw):
    return D.default_config(model=model, imax=c["ni"], jmax=c["nj"], kmax=c["nk"], Lx=synth.LY, Ly=synth.LX, Lz=synth.LZ,
                            stretched_x=0, T_west=T_wall, T_east=T_wall, seed=seed % 65521 + 1, **kw)


def _set_table(s, t):
    s.set_table(t["k"], t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"], X0=t["X0"], dX=t["dX"])


_dropin = None


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(kind=kind, case=c)
    if kind == "grey":
        s = D.Solver(_config(c, D.MODEL_GREY, 300.0, seed, kappa=1.0, nvar=2,
                             sampler=D.SAMPLER_RQMC if c["rqmc"] else D.SAMPLER_IID))
        s.set_rays(c["rays"])
        if c["f32"]:
            s.set_result_type(D.RESULT_F32)
        st.update(s=s, T=_field(c, seed, 300.0, 700.0))
    elif kind == "noalloc":
        cfg = _config(c, D.MODEL_GREY, 300.0, seed, kappa=1.0, nvar=2, photmax=c["rays"] // 2)
        T = torch.from_numpy(_field(c, seed, 300.0, 700.0)).cuda()
        out = torch.zeros((2, c["nk"], c["nj"], c["ni"]), dtype=torch.float64, device="cuda")
        xu = np.linspace(0.0, synth.LY, c["ni"] + 1).astype(np.float32)
        st.update(cfg=cfg, T=T, out=out, xu=xu, status=torch.zeros(1, dtype=torch.int32, device="cuda"))
    elif kind == "bands":
        cfg = _config(c, D.MODEL_GREY_BANDS, 300.0, 0, kappa=1.0, nvar=2, photmax=c["rays"] // 2, sampler=D.SAMPLER_RQMC,
                      p_row=c["p_row"])
        global _dropin
        if _dropin != repr(sorted(c.items())):  # the pair's configuration is the process's: set once
            D.dropin_configure(cfg)
            _dropin = repr(sorted(c.items()))
        T = np.zeros((c["nk"] + 2, c["nj"] + 2, c["ni"] + 2), np.float32)
        T[1:-1, 1:-1, 1:-1] = _field(c, seed, 300.0, 700.0)
        Q = np.zeros((c["nk"] + 2, c["nj"] // c["p_row"] + 2, c["ni"] + 2), np.float32)
        st.update(T=T, Q=Q, V=np.zeros_like(Q))
    elif kind == "mg":
        s = D.Solver(_config(c, D.MODEL_GREY_BANDS, 300.0, seed, kappa=1.0, nvar=3, grid_num=c["levels"]))
        s.use_grey_band_tables()
        s.set_rays(c["rays"])
        s.set_result_type(D.RESULT_F32)
        st.update(s=s, T=_field(c, seed, 300.0, 700.0))
    elif kind in ("net", "batch", "ck", "particles"):
        t = _table(*((c["nbands"], c["nq"], c["nT"], c["nX"]) if "nbands" in c else (64, 16, 50, 8)))
        kw = dict(n_groups=c.get("groups", 8), nvar=2, local_sampling=1, control_variate=1,
                  sampler=D.SAMPLER_RQMC if c.get("rqmc", True) else D.SAMPLER_IID)
        if kind == "net":
            kw["block_threads"] = 128
        if kind == "particles":
            kw.update(block_threads=128, eps_west=0.8, eps_east=0.8)
        s = D.Solver(_config(c, D.MODEL_TABLE, 400.0, seed, **kw))
        _set_table(s, t)
        n = c.get("fields", 1)
        T = np.stack([_field(c, seed * 16 + f, 400.0, 1400.0) for f in range(n)])
        x = np.stack([_h2o(c, seed * 16 + f) for f in range(n)])
        if kind != "ck":
            s.set_result_type(D.RESULT_F32)
        if kind == "batch":
            s.set_graph(True)
        else:
            s.set_rays(c["rays"])
        st.update(s=s, T=T, x=x)
        if kind == "net":
            st["net"] = D.CvNet.load(NET)
        if kind == "particles":
            p = synth.particle_table(t["k"].shape[0])
            s.set_particles(p["absorption"], p["scattering"], p["g"])
            st["fv"] = np.ascontiguousarray(
                1e-5 * (1.0 + 0.5 * synth.fourier_fluct(c["ni"], c["nj"], c["nk"], seed + 2000)), dtype=np.float32)
    elif kind == "plain":
        t = _table(c["nbands"], c["nq"], c["nT"], 8)
        s = D.Solver(_config(c, D.MODEL_TABLE, 400.0, seed, n_groups=1, nvar=3))
        s.set_table(t["k"][..., 3], t["wvc"], t["T0"], t["dT"], dnu=t["dnu"], wq=t["wq"])
        s.set_rays(c["rays"])
        st.update(s=s, T=_field(c, seed, 400.0, 1400.0))
    elif kind == "train":
        t = _table(64, 16, 50, 8)
        s = D.Solver(_config(c, D.MODEL_TABLE, 400.0, seed, n_groups=8, nvar=4, local_sampling=1, control_variate=1,
                             cv_moments=1, sampler=D.SAMPLER_RQMC))
        _set_table(s, t)
        s.set_fields(_field(c, seed, 400.0, 1400.0), _h2o(c, seed))
        s.set_rays(8)
        s.solve()
        net = D.CvNet(cvtrain.feature_config(t, batch=c["batch"], seed=seed % 65521 + 1))
        net.add_training_data(s)
        s.close()
        p, sc = net.params()
        st.update(net=net, p0=p, sc=sc)
    else:
        st.update(spec=_spectra(c, seed), gq=synth.gauss_legendre_half(16)[0])
    return st


def _spectra(c, seed):
    """Line-by-line-like spectra (Lorentz lines of log-normal strength) on a
    0.01 1/cm grid, `points` intervals a band."""
    rng = np.random.default_rng(seed)
    nb, per = c["nbands"], c["points"]
    npts, dwv, wv0 = nb * per + 1, 0.01, 1000.0
    nl = 40 * nb
    pos = wv0 + rng.uniform(0, nb * per * dwv, nl)
    S0 = np.exp(rng.normal(np.log(1e-2), 2.0, nl))
    E, g0 = rng.uniform(0.0, 3000.0, nl), rng.uniform(0.02, 0.1, nl)
    T = np.linspace(300.0, 2500.0, c["nT"])
    X = np.linspace(0.05, 0.3, c["nX"])
    dev = dict(dtype=torch.float64, device="cuda")
    S = S0 * (296.0 / T[:, None]) ** 1.5 * np.exp(-1.4388 * E * (1.0 / T[:, None] - 1.0 / 296.0))
    gam = g0 * (296.0 / T[:, None, None]) ** 0.7 * (1.0 + 4.0 * X[:, None])      # [T][X][line]
    nu = wv0 + dwv * torch.arange(npts, **dev)
    gam, S = torch.tensor(gam, **dev), torch.tensor(S, **dev)
    k = torch.zeros((c["nT"], c["nX"], npts), **dev)
    for q in range(nl):
        g = gam[:, :, q, None]
        k += (S[:, q, None, None] * g / math.pi) / ((nu - pos[q]) ** 2 + g * g)
    k = 100.0 * torch.tensor(X, **dev)[None, :, None] * k + 1e-6
    left = wv0 + per * dwv * np.arange(nb)
    return dict(kappa=k.cpu().numpy(), wv0=wv0, dwv=dwv, first=np.arange(nb, dtype=np.int64) * per,
                count=np.full(nb, per + 1, np.int32), wv_left=left, wv_right=left + per * dwv)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind, c = state["kind"], state["case"]
    if kind == "noalloc":
        lib, T, out, cfg = _lib.load(), state["T"], state["out"], state["cfg"]
        ptr = ctypes.c_void_p
        _lib.check(lib.dnsmc_solve_grey_noalloc(ctypes.byref(cfg), state["xu"].ctypes.data_as(_lib.c_float_p),
                                                ptr(T.data_ptr()), ptr(out[0].data_ptr()), ptr(out[1].data_ptr()),
                                                ptr(state["status"].data_ptr()),
                                                ptr(torch.cuda.current_stream().cuda_stream)))
        return out, state["status"]
    if kind == "bands":
        D.mc_gpu(state["T"], 1)
        D.get_results(state["Q"], state["V"])
        return state["Q"], state["V"]
    if kind == "train":
        net = state["net"]
        net.set_params(state["p0"], state["sc"])
        loss = net.train(1)
        return net.params()[0], np.array(loss)
    if kind == "lbl":
        return D.ck_from_lbl(state["spec"], state["gq"], n_pwrk=c["bins"])
    s = state["s"]
    s.set_fields(state["T"], state.get("x"))
    if kind == "net":
        state["net"].apply(s, mean_rays=c["rays"], min_rays=4, max_rays=4096)
    elif kind == "batch":
        s.set_rays_adaptive(600.0, c["rays"], 4096)
    elif kind == "particles":
        s.set_particle_field(state["fv"])
    return s.solve()


# ---------------------------------------------------------------------------
# the least a pass has to do
# ---------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "lbl":
        pts = c["nT"] * c["nX"] * (c["nbands"] * c["points"] + 1)
        return dict(bytes=8 * pts + c["nT"] * c["nX"] * c["nbands"] * (16 * 4 + 8), flops=60 * pts)
    cells = c["ni"] * c["nj"] * c["nk"]
    if kind == "train":  # forward and backward of 51 k multiply-adds a row; the features and labels read once
        return dict(bytes=cells * (80 * 2 + 8 * 8 * 4), flops=cells * 3 * 2 * 51200)
    cells *= c.get("fields", 1)
    groups = 8 if kind in ("net", "batch", "particles") else c.get("groups", 1)
    # mean ray-voxel steps a ray: its flight to the wall or the 1e-3 cut-off,
    # about the wall-normal cell count times 1.2 for kappa = 1 and 0.4 for the
    # correlated-k mixtures (counted at the listed sizes)
    steps = c["ni"] * (1.2 if kind in ("grey", "noalloc", "bands", "mg") else 0.4)
    fields = 1 + (kind in ("net", "batch", "ck", "particles")) + (kind == "particles")
    if kind == "bands":
        cells //= c["p_row"]
    out = 16 if kind in ("noalloc", "ck", "plain") or c.get("f32") is False else 8  # Q and sigma, FP64 or FP32
    # a step: two interpolations (k, Ib), an exponential, the update: 30 flops
    return dict(bytes=cells * (4 * fields + out), flops=cells * groups * c["rays"] * steps * 30)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Grey solves: the same rays (counter-based words) through the same cells
    in float64.  Spectral tables: the k-distributions in numpy.  None for the
    tabulated Monte Carlo solves and the training pass: their rays, and the
    order of the rows, come out of the library's own sampling tables and
    shuffles."""
    if case["kind"] == "lbl":
        return _exact_lbl(case, seed)
    if case["kind"] not in ("grey", "noalloc"):
        return None
    c = case
    cfg_seed, N = seed % 65521 + 1, c["rays"] - (c["rays"] % 2 if case["kind"] == "noalloc" else 0)
    if c["ni"] * c["nj"] * c["nk"] * N > 1.5e8:
        return None
    rqmc = bool(c.get("rqmc"))
    s1, s2 = _grey64(c, _field(c, seed, 300.0, 700.0), N, rqmc, cfg_seed)
    m = s1 / N
    if rqmc:
        v = torch.clamp(s2 / 2 - m * m, min=0.0)
    else:
        v = torch.clamp(s2 / N - m * m, min=0.0) / (N - 1)
    if case["kind"] == "noalloc":
        return torch.stack([m, v]), None
    return m[None], torch.sqrt(v)[None]


def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 of int64 tensors holding 32-bit words."""
    M = 0xFFFFFFFF
    k0, k1 = key & M, key >> 32

    def mul(a, b):  # (high, low) words of a * b without overflowing 63 bits
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        t = (lo >> 16) + hi
        return (t >> 16) & M, (((t & 0xFFFF) << 16) | (lo & 0xFFFF)) & M

    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
        h0, l0 = mul(c0, 0xD2511F53)
        h1, l1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
    return c0, c1, c2, c3


def _sobol2(n):
    """The first two Sobol' dimensions (polynomials 1 and x + 1), n points."""
    out = np.zeros((n, 2), np.int64)
    m1 = [1]
    for _ in range(31):
        m1.append(m1[-1] ^ (m1[-1] << 1))
    for i in range(n):
        a = b = 0
        for k in range(32):
            if i >> k & 1:
                a ^= 1 << (31 - k)
                b ^= m1[k] << (31 - k)
        out[i] = a, b
    return torch.from_numpy(out).cuda()


def _grey64(c, T, N, rqmc, key):
    """Sums over the rays of (X, X^2) per cell, or of (X, squared means of the
    two replicates): shapes [nk][nj][ni]."""
    ni, nj, nk = c["ni"], c["nj"], c["nk"]
    f64 = dict(dtype=torch.float64, device="cuda")
    T4 = torch.tensor(T.transpose(2, 0, 1).astype(np.float64) ** 4, **f64).contiguous()   # [i][k][j]
    Tw4, toll, W = 300.0 ** 4, float(np.float32(1e-3)), 4.0 * SIGMA
    ta = 8 if nk >= 8 else (16 if nk >= 4 else 32)
    tb = 64 // ta
    npa, npb = -(-nj // ta), -(-nk // tb)
    fw = torch.linspace(0.0, synth.LY, ni + 1, **f64)
    da, db = synth.LX / nj, synth.LZ / nk
    P = ni * npa * npb
    p = torch.arange(P, device="cuda")
    w0, pb, pa = p // (npa * npb), p // npa % npb, p % npa
    l = torch.arange(64, device="cuda")
    a0 = pa[:, None] * ta + l % ta                                                     # [P][64]
    b0 = pb[:, None] * tb + l // ta
    live0 = (a0 < nj) & (b0 < nk)
    a0, b0 = a0 % nj, b0 % nk
    Ti = T4[w0[:, None], b0, a0]
    oW = 0.5 * (fw[w0] + fw[w0 + 1])
    S1, S2, rep = (torch.zeros((P, 64), **f64) for _ in range(3))
    sob = _sobol2(N // 2) if rqmc else None
    z = torch.zeros_like(p)
    flat = T4.reshape(-1)
    chunk = max(1, int(4e7) // (P * 64))
    for r0 in range(0, N, chunk):
        rs = torch.arange(r0, min(N, r0 + chunk), device="cuda")
        R = len(rs)
        cp = p[:, None].expand(P, R)
        if rqmc:
            h = _philox((rs // (N // 2))[None].expand(P, R), cp, z[:, None].expand(P, R),
                        torch.full((P, R), 0x50B01, device="cuda"), key)
            x0, x1 = h[0] ^ sob[rs % (N // 2), 0][None], h[1] ^ sob[rs % (N // 2), 1][None]
        else:
            h = _philox(rs[None].expand(P, R), cp, z[:, None].expand(P, R), z[:, None].expand(P, R), key)
            x0, x1 = h[0], h[1]
        mu = 1.0 - 2.0 * (x1 >> 8).double() / 2 ** 24
        phi = 2.0 * math.pi * (x0 >> 8).double() / 2 ** 24
        st = torch.sqrt(torch.clamp(1.0 - mu * mu, min=0.0))
        sW, sA, sB = mu, st * torch.cos(phi), st * torch.sin(phi)
        dW, dA, dB = (torch.where(s > 0, 1, -1) for s in (sW, sA, sB))
        up = (dW > 0).long()
        cw = w0[:, None].expand(P, R).clone()
        tW = (fw[cw + up] - oW[:, None]) / sW
        dtA, dtB = da / sA.abs(), db / sB.abs()
        nA, nB = torch.zeros((P, R), **f64), torch.zeros((P, R), **f64)
        tA, tB = 0.5 * dtA, 0.5 * dtB
        t = torch.zeros((P, R), **f64)
        tau = live0[:, None, :].expand(P, R, 64).double().clone()
        Dx = torch.zeros((P, R, 64), **f64)
        va = torch.zeros((P, R), dtype=torch.long, device="cuda")
        vb = va.clone()
        on = torch.ones((P, R), dtype=torch.bool, device="cuda")
        while bool(on.any()):
            ax0 = (tW <= tA) & (tW <= tB)
            ax1 = ~ax0 & (tA <= tB)
            ax2 = ~ax0 & ~ax1
            tn = torch.where(ax0, tW, torch.where(ax1, tA, tB))
            ds = torch.where(on, tn - t, 0.0)
            idx = (cw[:, :, None] * nk + (b0[:, None, :] + vb[:, :, None]) % nk) * nj + (a0[:, None, :] + va[:, :, None]) % nj
            g = Ti[:, None, :] - flat[idx]
            # kappa = 1: the same attenuation in every cell of a packet-ray
            al = -torch.expm1(-ds)[:, :, None]
            take = tau * al
            Dx += take * g
            tau -= take
            low = tau < toll
            Dx += torch.where(low, tau * g, 0.0)
            tau = torch.where(low, 0.0, tau)
            nw = cw + dW
            wall = on & ax0 & ((nw < 0) | (nw >= ni))
            Dx += torch.where(wall[:, :, None], tau * (Ti[:, None, :] - Tw4), 0.0)
            on = on & ~wall & (tau > 0).any(2)
            t = tn
            cw = torch.where(on & ax0, nw, cw)
            tW = torch.where(ax0, (fw[(cw + up).clamp(max=ni)] - oW[:, None]) / sW, tW)
            nA, nB = nA + ax1, nB + ax2
            tA, tB = (nA + 0.5) * dtA, (nB + 0.5) * dtB
            va, vb = torch.where(ax1, (va + dA) % nj, va), torch.where(ax2, (vb + dB) % nk, vb)
        X = W * Dx
        S1 += X.sum(1)
        if rqmc:
            for q in range(R):
                rep += X[:, q]
                if (r0 + q + 1) % (N // 2) == 0:
                    S2 += (rep / (N // 2)) ** 2
                    rep.zero_()
        else:
            S2 += (X * X).sum(1)
    out = []
    for v in (S1, S2):
        g = torch.zeros((ni, npb * tb, npa * ta), **f64)
        g[:] = v.reshape(ni, npb, npa, tb, ta).permute(0, 1, 3, 2, 4).reshape(ni, npb * tb, npa * ta)
        out.append(g[:, :nk, :nj].permute(1, 2, 0).contiguous())
    return out


def _exact_lbl(c, seed):
    sp, gq = _spectra(c, seed), synth.gauss_legendre_half(16)[0]
    nT, nX, nb, NB = c["nT"], c["nX"], c["nbands"], c["bins"]
    kq = np.zeros((nb, len(gq), nT, nX))
    kavg = np.zeros((nT, nX, nb))
    for b in range(nb):
        lo = int(sp["first"][b])
        frac = sp["dwv"] / (sp["wv_right"][b] - sp["wv_left"][b])
        for t in range(nT):
            for x in range(nX):
                k = sp["kappa"][t, x, lo:lo + int(sp["count"][b])]
                p0, p1 = k.min() ** 0.1, k.max() ** 0.1
                step = (p1 - p0) / (NB - 1)
                mid = 0.5 * (k[1:] + k[:-1])
                n = np.bincount(np.clip(((mid ** 0.1 - p0) / step + 1.0).astype(np.int64), 0, NB), minlength=NB + 1)
                e = (p0 + np.arange(NB + 1) * step) ** 10
                kb = 0.5 * (e[:-1] + e[1:])                       # bin values h = 0 .. NB-1
                kavg[t, x, b] = (kb[1:] * n[1:NB] * frac).sum()
                # g(h) = 1 - fraction of the bins h+1 .. NB-1
                g = 1.0 - np.append(np.cumsum(n[NB - 1:0:-1])[::-1], 0) * frac
                h = np.clip(np.searchsorted(g, gq, side="left") - 1, 0, NB - 2)
                d = g[h + 1] - g[h]
                kq[b, :, t, x] = np.where(d == 0, kb[h + 1], kb[h] + (kb[h + 1] - kb[h]) * (gq - g[h]) / np.where(d == 0, 1, d))
    return kq, kavg
