"""The workloads that a user of this framework has it do, with their inputs.

Every case goes through the framework's public entry points: MPMSolver and
the C ABI's record and state calls, Adjoint, and the sensitivity surrogate
(window_stats, features, Ensemble, MLP).

  listed()          the cases
  draw(rng)         one more case of the same ranges
  prepare(c, seed)  inputs on the GPU and the handles a program keeps
  run(state)        one pass
  work(c)           bytes and operations a pass cannot do without
  exact(c, seed)    the outputs in 64 bits by plain torch, where they have
                    such a value

Scenes hold one box (or the four boxes of the mixed scene) of particles in
mid-motion: a linear velocity field with its C, and a smooth deformation, so
that no field is trivially zero.
"""
import ctypes as C
import math

import numpy as np
import torch

from autoquantizer_b200 import _lib, scenes
from autoquantizer_b200 import surrogate as SG
from autoquantizer_b200.adjoint import Adjoint, ek_seed
from autoquantizer_b200.mpm_config import MPMConfig
from autoquantizer_b200.mpm_solver import MPMSolver


def listed():
    return [
        # inference of the sensitivity surrogate for one scene (derive_scheme):
        # the smallest call there is
        {"name": "mlp_forward_1", "kind": "mlp_forward", "batch": 1},
        # one training batch of the surrogate (MLP.fit's default batch)
        {"name": "mlp_grad_128", "kind": "mlp_grad", "batch": 128},
        # a frame of the smallest experiment scene (elastic_block_2d, plain
        # FP32 state): launch latency
        {"name": "step_2d_elastic_8k", "kind": "step", "dim": 2, "n": 8192, "grid": 128, "mat": "elastic",
         "rec": "f32", "substeps": 32, "sparse": False},
        # a frame of the 2D fluid on quantized, dithered records (dam_break_2d)
        {"name": "step_2d_fluid_64k", "kind": "step", "dim": 2, "n": 65536, "grid": 256, "mat": "fluid",
         "rec": "quant", "substeps": 32, "sparse": False},
        # a frame of the 3D elastic block, FP32 state (falling_block_3d)
        {"name": "step_3d_elastic_262k", "kind": "step", "dim": 3, "n": 262144, "grid": 64, "mat": "elastic",
         "rec": "f32", "substeps": 32, "sparse": False},
        # a frame of the 3D throughput scene on quantized records
        # (mixed_boxes_3d): the largest
        {"name": "step_3d_mixed_2m", "kind": "step", "dim": 3, "n": 2097152, "grid": 128, "mat": "mixed",
         "rec": "quant", "substeps": 32, "sparse": False},
        # a frame on a sparse grid, whose dense one would be 512^3
        {"name": "step_3d_sparse_300k", "kind": "step", "dim": 3, "n": 300001, "grid": 512, "mat": "elastic",
         "rec": "f32", "substeps": 16, "sparse": True},
        # initial values stored, the records and the decoded state read back
        # (emission, checkpoints, dumps) at the throughput scene's size
        {"name": "records_3d_2m", "kind": "records", "dim": 3, "n": 2097152, "grid": 128, "mat": "mixed",
         "rec": "quant"},
        # per-field statistics of a state and its error against a reference
        # state (the surrogate's features, the error report)
        {"name": "stats_3d_1m", "kind": "stats", "dim": 3, "n": 1000003, "grid": 128, "mat": "elastic",
         "rec": "quant"},
        # sensitivities of the 2D experiment: forward and backward, segment
        # checkpoints
        {"name": "adjoint_2d_8k", "kind": "adjoint", "dim": 2, "n": 8192, "grid": 128, "mat": "elastic",
         "prec": "f32", "T": 32, "every": 16},
        # sensitivities of the 3D falling block
        {"name": "adjoint_3d_262k", "kind": "adjoint", "dim": 3, "n": 262144, "grid": 64, "mat": "elastic",
         "prec": "f32", "T": 32, "every": 16},
        # a scheme's features and predicted sensitivities for a new scene:
        # simulator set-up, 16-substep window, statistics, inference
        {"name": "derive_3d_255k", "kind": "derive", "dim": 3, "n": 255001, "grid": 64, "mat": "elastic"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene_draw(rng, n_min, n_max, mats=("elastic", "fluid")):
    dim = rng.choice((2, 3))
    n = _log_int(rng, n_min, n_max)
    mat = rng.choice(mats if dim == 3 else mats[:2])
    grids = (64, 128, 256, 512) if dim == 2 else (32, 64, 128)
    # the coarsest grid on which the particles take at most 0.55 of the domain's edge
    grid = next((g for g in grids if (n / 8.0) ** (1.0 / dim) <= 0.55 * g), grids[-1])
    return {"dim": dim, "n": n, "grid": grid, "mat": mat}


def draw(rng):
    """One more case: every kind, sizes spread over their range's logarithm."""
    kind = rng.choice(("step", "step", "step", "step", "step", "records", "records", "stats", "stats", "adjoint",
                       "adjoint", "adjoint", "derive", "mlp"))
    if kind == "step":
        rec = rng.choice(("f32", "quant", "quant", "f64"))
        c = _scene_draw(rng, 5_000, 200_000 if rec == "f64" else 1_500_000, ("elastic", "fluid", "mixed"))
        sparse = c["n"] <= 400_000 and rng.random() < 0.25
        if sparse:  # unquantized: the scenes' widths do not resolve so fine a grid's cells
            c["grid"] = 512 if c["dim"] == 3 else 2048
            rec = "f32" if rec == "quant" else rec
        return {"kind": kind, **c, "rec": rec, "substeps": rng.choice((1, 5, 16, 31)), "sparse": sparse}
    if kind in ("records", "stats"):
        c = _scene_draw(rng, 10_000, 2_000_000, ("elastic", "fluid", "mixed"))
        return {"kind": kind, **c, "rec": rng.choice(("f32", "quant", "quant"))}
    if kind == "adjoint":
        prec = rng.choice(("f32", "f32", "f64"))
        c = _scene_draw(rng, 5_000, 60_000 if prec == "f64" else 200_000)
        T = rng.choice((9, 16, 24))
        return {"kind": kind, **c, "prec": prec, "T": T, "every": rng.choice((0, 4, 16))}
    if kind == "derive":
        return {"kind": kind, **_scene_draw(rng, 10_000, 500_000)}
    return {"kind": rng.choice(("mlp_forward", "mlp_grad")), "batch": _log_int(rng, 2, 2048)}


# ------------------------------------------------------------------ scenes


def _config(c, seed):
    """MPMConfig of a case: random_scene's materials and time step, the
    scenes' record layouts."""
    dim, grid = c["dim"], c["grid"]
    g = np.random.default_rng([seed, 1])
    m = MPMConfig()
    m.dim, m.n_grid, m.grid_res, m.n_particles = dim, grid, [grid] * dim, c["n"]
    m.size, m.bound, m.use_friction, m.use_bls = 1.0, [3] * dim, False, True
    m.precision = "f64" if "f64" in (c.get("rec"), c.get("prec")) else "f32"
    m.compute_fp = m.precision
    m.p_rho = 1.0
    dx = 1.0 / grid
    m.p_vol = (dx * 0.5) ** dim
    m.use_fluid = c["mat"] == "fluid"
    # quantized scenes are soft enough for their widths (the noise of a
    # 16-bit F times a stiffness of 1e5 outweighs the motion)
    e_max = 4 if c.get("rec") == "quant" else 5
    m.E, m.nu = float(10 ** g.uniform(3, e_max)), float(g.uniform(0.2, 0.4))
    m.la = float(10 ** g.uniform(2.5, e_max - 1))
    E = m.E
    if c["mat"] == "mixed":
        E = 1e4 if e_max == 4 else 1e5
        m.materials = [(_lib.AQ_MAT_COROTATED, m.E, m.nu, 0.0),
                       (_lib.AQ_MAT_COROTATED, float(10 ** g.uniform(3, e_max)), 0.3, 0.0),
                       (_lib.AQ_MAT_FLUID, 0.0, 0.0, 1e3), (_lib.AQ_MAT_FLUID, 0.0, 0.0, 1e3)]
    mu, la0 = E / (2 * (1 + m.nu)), E * m.nu / ((1 + m.nu) * (1 - 2 * m.nu))
    m.dt = float(min(2e-4, 0.2 * dx / math.sqrt(m.la if m.use_fluid else la0 + 2 * mu)))
    m.n_timesteps = c.get("T", 64) + 1
    m.use_dithering = False
    m.sparse_grid = bool(c.get("sparse", False))
    if c.get("rec") == "quant":
        m.use_quantaichi = m.use_bitpack = m.use_dithering = True
        m.v_exp_bits = 6
        fj = "J" if m.use_fluid else "F"
        m.quantized_properties = {"x": 1, "v": 1, "C": 1, fj: 1}
        nf = 1 if m.use_fluid else dim * dim
        x, v = (20, 13) if dim == 2 else (21, 12)
        m.quant_bits = np.array([x] * dim + [v] * dim + [16] * (dim * dim + nf))
        m.quant_ranges = np.array([1.0] * 2 * dim + [64.0] * (dim * dim) + [0.5 if m.use_fluid else 2.0] * nf)
    return m


def _slots(c):
    d = c["dim"]
    nf = 1 if c["mat"] == "fluid" else d * d
    return 2 * d + d * d, nf, 2 * d + d * d + nf + (1 if c["mat"] == "mixed" else 0)


def _values(c, seed):
    """Initial particle values (CUDA, n x n_slots, float64 holding float32 values)."""
    d, n = c["dim"], c["n"]
    dev = "cuda"
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 13)
    g = np.random.default_rng([seed, 2])
    f0, nf, ns = _slots(c)
    vals = torch.zeros((n, ns), dtype=torch.float64, device=dev)
    domain = c["grid"] if not c.get("sparse") else 128 if d == 3 else 512  # cells the scene is laid out in
    u = torch.rand((n, d), generator=gen, device=dev, dtype=torch.float64)
    if c["mat"] == "mixed":  # the four boxes of mixed_boxes_3d
        sizes = g.uniform(0.25, 0.4, (4, d))
        lows = np.array([g.uniform(0.08, 0.92 - s) for s in sizes.ravel()]).reshape(4, d)
        cnt = np.floor(n * sizes.prod(1) / sizes.prod(1).sum()).astype(np.int64)
        cnt[-1] = n - cnt[:-1].sum()
        mat = torch.repeat_interleave(torch.arange(4, device=dev), torch.from_numpy(cnt).to(dev))
        x = torch.from_numpy(lows).to(dev)[mat] + u * torch.from_numpy(sizes).to(dev)[mat]
        vals[:, -1] = mat.double()
    else:
        side = min(0.7, (n / (8.0 if d == 3 else 6.0)) ** (1.0 / d) / domain)
        asp = g.uniform(0.85, 1.15, d)
        x = 0.5 + (u - 0.5) * torch.from_numpy(side * asp).to(dev)
        if c.get("sparse"):  # the same cells in a larger index space
            x = 0.5 + (x - 0.5) * (domain / c["grid"])
    W = torch.from_numpy(g.normal(0, 5.0, (d, d))).to(dev)
    c0 = torch.from_numpy(g.uniform(0.4, 0.6, d)).to(dev)
    push = torch.from_numpy(g.uniform(-0.5, 0.5, d)).to(dev)
    vals[:, :d] = x
    vals[:, d:2 * d] = push + (x - c0) @ W.T
    vals[:, 2 * d:f0] = W.reshape(-1)
    ph = torch.from_numpy(g.uniform(0, 6.28, nf)).to(dev)
    wave = torch.sin(6.0 * (x - c0).sum(1, keepdim=True) + ph)
    if nf == 1:
        vals[:, f0:f0 + 1] = 1.0 + 0.01 * wave
    else:
        vals[:, f0:f0 + nf] = torch.eye(d, dtype=torch.float64, device=dev).reshape(-1) + 0.01 * wave
    return vals.float().double()


# ------------------------------------------------------------------- cases


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("mlp_forward", "mlp_grad"):
        m = SG.MLP(seed=seed)
        g = np.random.default_rng([seed, 3])
        x = torch.from_numpy(g.normal(size=(c["batch"], SG.N_IN)).astype(np.float32)).cuda()
        dy = torch.from_numpy(g.normal(size=(c["batch"], SG.N_OUT)).astype(np.float32)).cuda()
        return {"kind": kind, "mlp": m, "x": x, "dy": dy}
    cfg = _config(c, seed)
    vals = _values(c, seed)
    st = {"kind": kind, "case": c, "cfg": cfg}
    if kind == "derive":
        g = np.random.default_rng([seed, 4])
        ens = SG.Ensemble(4, seed=seed)
        X, Y = g.normal(size=(64, SG.N_IN)), g.normal(size=(64, SG.N_OUT))
        ens.fit(X, Y, np.ones_like(Y), steps=0)  # the training data's normalization
        st.update(s0=vals.float(), ens=ens)
        return st
    if kind == "adjoint":
        s = MPMSolver(cfg)
        dt = torch.float64 if c["prec"] == "f64" else torch.float32
        s.set_particles(vals.to(dt))
        st.update(adj=Adjoint(s._params()), s0=vals.to(dt), solver=s)
        return st
    f64 = c["rec"] == "f64"
    vals = vals if f64 else vals.float()
    s = MPMSolver(cfg)
    s.set_particles(vals)
    s._ensure_sim()
    st.update(solver=s, f64=f64)
    if kind == "step":
        st["words"] = torch.from_numpy(s.words().view(np.int64)).cuda()
    elif kind == "records":
        st["values"] = vals
        st["words_out"] = torch.empty((c["n"], s.layout().n_words), dtype=torch.int64, device="cuda")
    else:
        ref = _values(c, seed + 1)
        st["ref"] = ref.float()
        st["state"] = s.state_tensor(True)
        st["ref64"] = ref
    return st


def run(st):
    kind = st["kind"]
    if kind == "mlp_forward":
        return st["mlp"].forward_raw(st["x"])
    if kind == "mlp_grad":
        return st["mlp"].grad_raw(st["x"], st["dy"])
    L = _lib.lib()
    if kind == "derive":
        # derive_scheme's way from a new scene to the members' predictions
        s0, cfg = st["s0"], st["cfg"]
        stats = SG.window_stats(cfg, s0)
        f = SG.features(cfg, stats, s0.shape[0])
        y = st["ens"].predict_members(f[None])
        # as float32: they come from a float32 state
        return {"stats": stats.astype(np.float32), "features": f.astype(np.float32), "y": y.astype(np.float32)}
    if kind == "adjoint":
        c, s = st["case"], st["solver"]
        sT = st["adj"].forward(st["s0"], c["T"], c["every"])
        g0, sens = st["adj"].backward(ek_seed(sT, c["dim"], s.p_mass, s.g))
        # sums of squares of the gradients, in the gradients' own precision
        return {"sT": sT, "g0": g0, "sens": sens.astype(np.float64 if c["prec"] == "f64" else np.float32)}
    s = st["solver"]
    if kind == "step":
        c = st["case"]
        # from a checkpoint's records (aq_sim_set_words, as a program that
        # resumes or that moves its own records does), a frame, the state
        _lib.check(L.aq_sim_set_words(s._sim, _ptr(st["words"]), _lib.stream_ptr()), "aq_sim_set_words")
        s.set_step_count(0)
        s.substeps(c["substeps"])
        v = s.state_tensor(st["f64"])
        d, (f0, nf, _) = c["dim"], _slots(c)
        return {"x": v[:, :d], "v": v[:, d:2 * d], "C": v[:, 2 * d:f0], "F": v[:, f0:f0 + nf]}
    if kind == "records":
        _lib.check(L.aq_sim_set_state(s._sim, _ptr(st["values"]), 0, _lib.stream_ptr()), "aq_sim_set_state")
        w = st["words_out"]
        _lib.check(L.aq_sim_get_words(s._sim, _ptr(w), _lib.stream_ptr()), "aq_sim_get_words")
        return {"words": w, "state": s.state_tensor(False)}
    ref, state, ref64 = st["ref"], st["state"], st["ref64"]
    n, ns = state.shape
    sq, mx = (C.c_double * ns)(), (C.c_double * ns)()
    stats = s.field_stats(reference=ref)
    _lib.check(L.aq_state_error(_ptr(state), 1, _ptr(ref64), 1, n, ns, sq, mx, _lib.stream_ptr()), "aq_state_error")
    return {"stats": stats, "sq": np.array(sq[:]), "max": np.array(mx[:])}


def _record_words(c):
    d = c["dim"]
    _, nf, ns = _slots(c)
    mat = 2 if c["mat"] == "mixed" else 0
    if c["rec"] == "f64":
        return ns - (mat > 0) + (1 if mat else 0)
    if c["rec"] == "f32":
        return (32 * (ns - (mat > 0)) + mat + 63) // 64
    x, v = (20, 13) if d == 2 else (21, 12)
    return (d * (x + v) + 6 + 16 * (d * d + nf) + mat + 63) // 64


def work(c):
    kind = c["kind"]
    if kind in ("mlp_forward", "mlp_grad"):
        a, h, o = SG.N_IN, SG.N_H, SG.N_OUT
        p, b = a * h + h + h * h + h + o * h + o, c["batch"]
        if kind == "mlp_forward":
            return {"bytes": 2 * p + 4 * b * (a + o), "flops": 2 * p * b}
        return {"bytes": 2 * p + 4 * p + 4 * b * (a + o), "flops": 6 * p * b}
    d, n = c["dim"], c["n"]
    _, _, ns = _slots(c)
    # a substep's operations per particle: gather and scatter over 3^d nodes
    per = (1700 if d == 3 else 400)
    if kind == "adjoint":
        e = 8 if c["prec"] == "f64" else 4
        T = c["T"]
        return {"bytes": n * ns * e * (2 * T + 4 * T), "flops": n * per * (T + 3 * T)}
    if kind == "derive":
        return {"bytes": n * (4 * ns * 3 + 16 * 2 * 4 * ns), "flops": n * per * 16}
    W = 8 * _record_words(c)
    if kind == "records":
        return {"bytes": n * (4 * ns * 2 + W), "flops": n * ns * 8}
    if kind == "stats":
        return {"bytes": n * (W + 4 * ns + 16 * ns), "flops": n * ns * 14}
    out = (8 if c["rec"] == "f64" else 4) * ns
    return {"bytes": n * (2 * W * c["substeps"] + out), "flops": n * per * c["substeps"]}


# ------------------------------------------------------------ 64-bit values
# The substep in plain torch, float64, one node offset at a time.


def _det_cof(F):
    d = F.shape[-1]
    if d == 2:
        return F[:, 0, 0] * F[:, 1, 1] - F[:, 0, 1] * F[:, 1, 0]
    return (F[:, 0, 0] * (F[:, 1, 1] * F[:, 2, 2] - F[:, 1, 2] * F[:, 2, 1])
            - F[:, 0, 1] * (F[:, 1, 0] * F[:, 2, 2] - F[:, 1, 2] * F[:, 2, 0])
            + F[:, 0, 2] * (F[:, 1, 0] * F[:, 2, 1] - F[:, 1, 1] * F[:, 2, 0]))


def _inv_t(F):
    c = torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                     torch.linalg.cross(F[:, 0], F[:, 1])], 1)
    return c / _det_cof(F)[:, None, None]


def _rotation(F):
    if F.shape[-1] == 2:
        a, b = F[:, 0, 0] + F[:, 1, 1], F[:, 1, 0] - F[:, 0, 1]
        r = torch.sqrt(a * a + b * b)
        return torch.stack([torch.stack([a / r, -b / r], 1), torch.stack([b / r, a / r], 1)], 1)
    X = F
    for _ in range(8):  # Newton's iteration: quadratic, from F near a rotation
        X = 0.5 * (X + _inv_t(X))
    return X


def _stress(F, mu, lam, law):
    """Cauchy stress by material law ("fluid": F is J or a matrix)."""
    if F.dim() == 1:
        raise ValueError
    d = F.shape[-1]
    eye = torch.eye(d, dtype=F.dtype, device=F.device)
    J = _det_cof(F)
    if law == "fluid":
        return lam[:, None, None] * (J - 1)[:, None, None] * eye
    if law == "corotated" or d == 2:
        return 2 * mu[:, None, None] * (F - _rotation(F)) @ F.transpose(1, 2) + (lam * J * (J - 1))[:, None, None] * eye
    return mu[:, None, None] * (F @ F.transpose(1, 2) - eye) + (lam * torch.log(J))[:, None, None]


def _substep(s, P):
    d, nf, g = P["d"], P["nf"], P["grid"]
    dx, dt = 1.0 / g, P["dt"]
    x, v, Cm = s[:, :d], s[:, d:2 * d], s[:, 2 * d:2 * d + d * d].reshape(-1, d, d)
    f0 = 2 * d + d * d
    n = x.shape[0]
    eye = torch.eye(d, dtype=x.dtype, device=x.device)
    one = torch.ones(n, dtype=x.dtype, device=x.device)
    if nf == 1:
        J = s[:, f0]
        sig = (P["la"] * (J - 1))[:, None, None] * eye
    else:
        F = s[:, f0:f0 + nf].reshape(-1, d, d)
        if "mats" in P:
            cid = P["mat"]
            mu, lam = P["mats"][0][cid], P["mats"][1][cid]
            fluid = (cid >= 2)[:, None, None]
            sig = torch.where(fluid, _stress(F, mu, lam, "fluid"), _stress(F, mu, lam, "corotated"))
        else:
            sig = _stress(F, P["mu"] * one, P["lam"] * one, "elastic")
    A = -dt * P["vol"] * 4 / dx / dx * sig + P["vol"] * Cm  # p_rho = 1: mass = volume
    t = x / dx
    base = torch.floor(t.detach() - 0.5)
    fx = t - base
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], 0)
    base = base.long()
    # nodes in the particles' bounding box only (a sparse case's index space is large)
    lo, hi = base.min(0).values, base.max(0).values + 3
    ext = (hi - lo).tolist()
    offs = torch.cartesian_prod(*[torch.arange(3, device=x.device)] * d).reshape(-1, d)
    ncell = int(np.prod(ext))
    idx = []
    m = torch.zeros((ncell, d + 1), dtype=x.dtype, device=x.device)
    for o in offs.tolist():
        wt = w[o[0], :, 0]
        for k in range(1, d):
            wt = wt * w[o[k], :, k]
        I = base - lo + torch.tensor(o, device=x.device)
        i = I[:, 0]
        for k in range(1, d):
            i = i * ext[k] + I[:, k]
        dpos = (torch.tensor(o, dtype=x.dtype, device=x.device) - fx) * dx
        mom = P["vol"] * v + (A @ dpos[:, :, None])[:, :, 0]
        m = m.index_add(0, i, wt[:, None] * torch.cat([P["vol"] * one[:, None], mom], 1))
        idx.append((i, wt, dpos))
    gv = m[:, 1:] / (m[:, :1] + 1e-10)
    grav = torch.zeros(d, dtype=x.dtype, device=x.device)
    grav[1] = dt * 9.8
    gv = gv - grav
    node = torch.arange(ncell, device=x.device)
    I = []
    for k in reversed(range(d)):
        I.append(node % ext[k] + lo[k])
        node = torch.div(node, ext[k], rounding_mode="floor")
    I = torch.stack(I[::-1], 1)
    gv = torch.where(((I < 3) & (gv < 0)) | ((I > g - 3) & (gv > 0)), torch.zeros_like(gv), gv)
    nv, nC = torch.zeros_like(x), torch.zeros((n, d, d), dtype=x.dtype, device=x.device)
    for i, wt, dpos in idx:
        q = wt[:, None] * gv[i]
        nv = nv + q
        nC = nC + 4 / dx / dx * q[:, :, None] * dpos[:, None, :]
    parts = [x + dt * nv, nv, nC.reshape(n, -1)]
    if nf == 1:
        parts.append(((1 + dt * nC.diagonal(dim1=1, dim2=2).sum(1)) * J)[:, None])
    else:
        nF = (eye + dt * nC) @ F
        if "mats" in P:
            Jn = _det_cof(nF)
            iso = (Jn.abs() ** (1.0 / d) * torch.sign(Jn))[:, None, None] * eye
            nF = torch.where(fluid, iso, nF)
        parts.append(nF.reshape(n, -1))
    return torch.cat(parts, 1)


def _physics(c, cfg, vals):
    f0, nf, _ = _slots(c)
    mu = cfg.E / (2 * (1 + cfg.nu))
    lam = cfg.E * cfg.nu / ((1 + cfg.nu) * (1 - 2 * cfg.nu))
    P = {"d": c["dim"], "nf": nf, "grid": c["grid"], "dt": cfg.dt, "vol": cfg.p_vol, "mu": mu, "lam": lam,
         "la": cfg.la}
    if c["mat"] == "mixed":
        mus, lams = [], []
        for kind, E, nu, la in cfg.materials:
            fluid = kind == _lib.AQ_MAT_FLUID
            mus.append(0.0 if fluid else E / (2 * (1 + nu)))
            lams.append(la if fluid else E * nu / ((1 + nu) * (1 - 2 * nu)))
        P["mats"] = [torch.tensor(t, dtype=torch.float64, device="cuda") for t in (mus, lams)]
        P["mat"] = vals[:, -1].long()
    return P


def _bf(t):
    return t.to(torch.float32).to(torch.bfloat16).double()


def _mlp_exact(case, seed):
    """The network in float64; operands of a product rounded to bf16, which
    is what the layers are defined on."""
    st = prepare(case, seed)
    a, h, o = SG.N_IN, SG.N_H, SG.N_OUT
    p, at, W = st["mlp"].p.double(), 0, []
    for i, j in ((a, h), (h, h), (h, o)):
        W.append((_bf(p[at:at + i * j].reshape(j, i)), p[at + i * j:at + i * j + j]))
        at += i * j + j
    gelu = lambda z: 0.5 * z * (1 + torch.erf(z / math.sqrt(2.0)))  # noqa: E731
    gelu_d = lambda z: 0.5 * (1 + torch.erf(z / math.sqrt(2.0))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi)  # noqa: E731
    x = st["x"].double()
    z1 = _bf(x) @ W[0][0].T + W[0][1]
    a1 = gelu(z1)
    z2 = _bf(a1) @ W[1][0].T + W[1][1]
    a2 = gelu(z2)
    if case["kind"] == "mlp_forward":
        return _bf(a2) @ W[2][0].T + W[2][1]
    dy = st["dy"].double()
    g3 = _bf(dy).T @ _bf(a2)
    dz2 = (_bf(dy) @ W[2][0]) * gelu_d(z2)
    g2 = _bf(dz2).T @ _bf(a1)
    dz1 = (_bf(dz2) @ W[1][0]) * gelu_d(z1)
    g1 = _bf(dz1).T @ _bf(x)
    return torch.cat([t.reshape(-1) for t in (g1, dz1.sum(0), g2, dz2.sum(0), g3, dy.sum(0))])


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind in ("mlp_forward", "mlp_grad"):
        return _mlp_exact(c, seed)
    cfg = _config(c, seed)
    vals = _values(c, seed)
    d = c["dim"]
    f0, nf, ns = _slots(c)
    if kind in ("records", "stats") and c["rec"] != "f32":
        return None  # the codes' own values: whole numbers and their multiples
    if kind == "records":
        return {"words": None, "state": vals}
    if kind == "stats":
        e = (vals - _values(c, seed + 1)).abs()
        stats = torch.stack([vals.abs().sum(0), vals.sum(0), (vals * vals).sum(0), vals.abs().max(0).values, e.sum(0)], 1)
        return {"stats": stats, "sq": (e * e).sum(0), "max": e.max(0).values}
    P = _physics(c, cfg, vals)
    s = vals[:, :f0 + nf]
    if kind == "step":
        with torch.no_grad():
            for _ in range(c["substeps"]):
                s = _substep(s, P)
        # quantized: C's own step is of the size of its values
        q = c["rec"] == "quant"
        return {"x": s[:, :d], "v": s[:, d:2 * d], "C": None if q else s[:, 2 * d:f0], "F": s[:, f0:]}
    if kind == "derive":
        s0 = s
        with torch.no_grad():
            for _ in range(SG.WINDOW):
                s = _substep(s, P)
        st = torch.stack([s.abs().sum(0), s.sum(0), (s * s).sum(0), s.abs().max(0).values, (s - s0).abs().sum(0)], 1)
        return {"stats": st, "features": None, "y": None}
    states = [s]
    with torch.no_grad():
        for _ in range(c["T"]):
            states.append(_substep(states[-1], P))
    sT = states[-1]
    v = sT[:, d:2 * d]
    g = torch.zeros_like(sT)
    if d == 3:
        g[:, d:2 * d] = cfg.p_vol * v
        g[:, 1] = cfg.g * cfg.p_vol
    else:
        g[:, d:2 * d] = 2 * v
    sens = torch.zeros(sT.shape[1], dtype=torch.float64, device="cuda")
    for t in reversed(range(c["T"])):
        s = states[t].detach().requires_grad_(True)
        (g,) = torch.autograd.grad(_substep(s, P), s, g)
        if t >= 1:
            sens += (g * g).sum(0)
    return {"sT": sT, "g0": g, "sens": sens}
