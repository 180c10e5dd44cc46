"""Performance cases: what a user of bfe_gb300 has it do, through its public entry points.

A case is a dict of plain values with a "kind":

  call     one load step through the drop-in fn_explicit_dynamic_solver_gb300
           (matrices in, histories and frames out; a plan is made and dropped)
  run      one load step on a plan that the program keeps (Plan.run)
  batch    many sources, or many sources over several joined models, as one
           march of a kept plan (Plan.run_batched)
  v5       one load step of the v5 scheme with prescribed displacements
  entry    the whole fn_BristolFE_v2_gb300 call: assembly, plan, march, and
           kinetic-energy frames
  adjoint  misfit and its gradient with respect to the elements
  fmc      full-matrix-capture time data from the monitored histories

The models are the repository's own families (bfe_gb300.model): a steel
plate, water over steel with an array in the water, steel sub-domains with a
void, a 3D steel block, and the plate of the adjoint. The seed sets the
stiffness (a factor of 0.94 to 1 on Young's modulus), the centre frequency,
the amplitudes and which sources and monitors are used. The mesh and the
matrices of the last model are kept between preparations, as a program that
runs many load steps over one model keeps them.

FP32 plans store FP32 histories in FP64 arrays: their outputs are returned as
FP32, which loses nothing of a history.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bristolfe-v2_gb300"))
import bfe_gb300  # noqa: E402
from bfe_gb300 import model  # noqa: E402
from bfe_gb300.entry import fn_BristolFE_v2_gb300  # noqa: E402

E0, NU, RHO = model.STEEL["E"], model.STEEL["nu"], model.STEEL["rho"]


def listed():
    return [
        # a first try on a small model: what one call costs when there is next to nothing to march
        dict(name="call_plate_small_f64", kind="call", model="plate", W=3e-3, H=1.5e-3, h=0.1e-3, prec="double",
             n_t=400, n_mon=16, every=0),
        # the plain 2D workload: 40,602 DOF, 2,000 samples, 16 monitors, 4 snapshots, through the drop-in call
        dict(name="call_plate_f64", kind="call", model="plate", W=20e-3, H=10e-3, h=0.1e-3, prec="double",
             n_t=2000, n_mon=16, every=500),
        # post-processing of a 64-element capture: 64 x 64 A-scans from the monitored histories
        dict(name="fmc_64x64", kind="fmc", n_el=64, per_el=1, n_t=2000, n_sig=180),
        # one source over the coupled water/steel model, in the reference's arithmetic and in FP32
        dict(name="run_coupled_f64", kind="run", model="coupled", W=60e-3, H=30e-3, h=0.05e-3, prec="double",
             n_t=2000, n_mon=64, every=0),
        dict(name="run_coupled_f32", kind="run", model="coupled", W=60e-3, H=30e-3, h=0.05e-3, prec="single",
             n_t=2000, n_mon=64, every=0),
        # full-matrix capture: 64 sources over the same model, the largest case
        dict(name="batch_coupled_f32_r64", kind="batch", model="coupled", W=60e-3, H=30e-3, h=0.05e-3,
             prec="single", n_t=1000, n_mon=64, R=64, n_models=1),
        # the same capture in the reference's arithmetic, on the coarser mesh that FP64 runs are made on
        dict(name="batch_coupled_f64_r64", kind="batch", model="coupled", W=60e-3, H=30e-3, h=0.1e-3,
             prec="double", n_t=600, n_mon=64, R=64, n_models=1),
        # uneven scatterer sub-domains joined in one plan, with a rank's share of 64 sources over three ranks
        dict(name="batch_subdomains_f32_r21", kind="batch", model="subdomains", W=10e-3, H=10e-3, h=0.05e-3,
             prec="single", n_t=800, n_mon=64, R=21, n_models=4),
        # one source in 3D
        dict(name="run_brick_f32", kind="run", model="brick", W=10e-3, H=5e-3, h=0.2e-3, prec="single",
             n_t=800, n_mon=64, every=0),
        # one gradient of an inversion: 16 sources x 16 receivers
        dict(name="adjoint_f32_16x16", kind="adjoint", W=30e-3, H=15e-3, h=0.1e-3, prec="single", n_t=1000, R=16,
             n_rec=16),
        # prescribed displacements along a line, the older solver's scheme
        dict(name="v5_plate_f64", kind="v5", W=20e-3, H=10e-3, h=0.1e-3, prec="double", n_t=1500, n_dsp=21, n_mon=16),
        # the reference's whole entry function, with an animation's frames
        dict(name="entry_plate_f64", kind="entry", W=20e-3, H=10e-3, h=0.1e-3, prec="double", n_t=1200, n_mon=16,
             n_src=1, every=60),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """Another case of the same ranges: sizes by their logarithm, odd ones among them."""
    kind = rng.choice(["call", "call", "run", "run", "run", "batch", "batch", "batch", "adjoint", "v5", "entry", "fmc"])
    prec = rng.choice(["double", "single"])
    if kind == "fmc":
        n_el = int(_log(rng, 8, 64))
        return dict(kind=kind, n_el=n_el, per_el=rng.randint(1, 3), n_t=int(_log(rng, 300, 3000)),
                    n_sig=int(_log(rng, 60, 240)))
    if kind in ("v5", "entry"):
        W = _log(rng, 3e-3, 20e-3)
        c = dict(kind=kind, W=W, H=W * rng.uniform(0.3, 0.7), h=0.1e-3, n_t=int(_log(rng, 200, 2000)),
                 n_mon=rng.randint(1, 32))
        if kind == "v5":
            return dict(c, prec=prec, n_dsp=rng.randint(1, 40))
        return dict(c, prec=prec, n_src=rng.randint(1, 5), every=rng.choice([0, 25, 60, 117]))
    if kind == "adjoint":
        W = _log(rng, 8e-3, 30e-3)
        return dict(kind=kind, W=W, H=W * rng.uniform(0.4, 0.6), h=0.1e-3, prec=prec, n_t=int(_log(rng, 200, 1000)),
                    R=rng.randint(2, 16), n_rec=rng.randint(2, 24))
    if kind == "batch":
        what = rng.choice(["plate", "coupled", "subdomains", "brick"])
        R = int(_log(rng, 2, 96))
        W = _log(rng, 4e-3, 8e-3) if what == "brick" else _log(rng, 8e-3, 30e-3) if what != "subdomains" else \
            _log(rng, 5e-3, 9e-3)
        h = rng.choice([0.2e-3, 0.25e-3]) if what == "brick" else 0.1e-3 if what != "subdomains" else 0.05e-3
        n_t = int(_log(rng, 200, 300 if what == "brick" else 1000))
        return dict(kind=kind, model=what, W=W, H=W * (0.5 if what != "subdomains" else 1.0), h=h, prec=prec, n_t=n_t,
                    n_mon=rng.choice([1, 16, 49, 64]), R=R, n_models=rng.randint(2, 5) if what == "subdomains" else 1)
    what = rng.choice(["plate", "coupled"] if kind == "call" else ["plate", "coupled", "coupled", "brick"])
    W = _log(rng, 4e-3, 10e-3) if what == "brick" else _log(rng, 2.5e-3, 20e-3) if kind == "call" else \
        _log(rng, 8e-3, 60e-3)
    return dict(kind=kind, model=what, W=W, H=W * rng.uniform(0.45, 0.55), h=0.2e-3 if what == "brick" else 0.1e-3,
                prec=prec, n_t=int(_log(rng, 300, 2000)), n_mon=rng.choice([1, 16, 33, 64]),
                every=rng.choice([0, 0, 100, 251]))


# ---------------------------------------------------------------------------
# Models

@functools.lru_cache(maxsize=1)
def _model(kind, W, H, h, n_mon, R, n_models):
    if kind == "plate":
        m = model.steel_plate(W, H, h, n_mon)
        top = np.nonzero(np.isclose(m["nds"][:, 1], m["nds"][:, 1].max()))[0] + 1
        src = [[int(n)] for n in top[np.linspace(0, top.size - 1, max(R, 1)).astype(int)]]
        return [dict(m, src=src, src_dof=2)]
    if kind == "coupled":
        wave = model.coupled_water_steel(W, 2 * H / 3, H / 3, h, abs_wavelengths=min(3.0, W / 8e-3),
                                         blob_radius=min(1.5e-3, H / 16), array_elements=max(R, n_mon),
                                         array_pitch=0.6 * W / max(R, n_mon))
        src = [[int(x) for x in np.ravel(s)] or [int(c)] for s, c in zip(wave["src_nodes"], wave["mon_nodes"])]
        return [dict(wave, src=src)]
    if kind == "subdomains":
        sides = np.linspace(0.55, 1.0, n_models) * W          # 50,000 DOF and up, uneven
        out = []
        for k, side in enumerate(sides):
            m = model.steel_subdomain(float(side), h, seed=k, n_src=max(R, 2), n_mon=max(n_mon, 2))
            out.append(dict(m, src=[list(s) for s in m["src_nodes"]][:R], mon_nodes=m["mon_nodes"][:n_mon]))
        dt = min(m["dt"] for m in out)
        return [dict(m, dt=dt) for m in out]
    if kind == "brick":
        m = model.steel_block_3d(W, W, H, h, n_mon=n_mon)
        top = np.nonzero(np.isclose(m["nds"][:, 2], m["nds"][:, 2].max()))[0] + 1
        src = [[int(n)] for n in top[np.linspace(0, top.size - 1, R + 2).astype(int)[1:-1]]] if R > 1 else \
            [[int(np.ravel(m["src_nodes"])[0])]]
        return [dict(m, src=src)]
    m = model.steel_plate_adjoint(W, H, h, n_src=R, n_rec=n_mon, abs_wavelengths=1.0)
    return [dict(m, src=m["src_nodes"], src_dof=2, mon_nodes=m["rec_nodes"], mon_dof=2)]


def _models(c):
    kind = c.get("model", "adjoint" if c["kind"] == "adjoint" else "plate")
    n_mon, R = c.get("n_rec", c.get("n_mon", 16)), c.get("R", c.get("n_src", 1))
    if kind == "coupled":                # one array serves as sources and monitors
        n = max(n_mon, R)
        m = _model(kind, c["W"], c["H"], c["h"], n, n, 1)[0]
        return [dict(m, src=m["src"][:R] if c["kind"] == "batch" else m["src"], mon_nodes=m["mon_nodes"][:n_mon])]
    return _model(kind, c["W"], c["H"], c["h"], n_mon, R, c.get("n_models", 1))


def _burst(t, fc, start=0.0, cycles=5):
    """A Gaussian-windowed burst that begins at 1 % of its envelope."""
    T = cycles / (2 * fc * math.sqrt(math.log(100.0)))
    x = t - start - T * math.sqrt(math.log(100.0))
    s = np.exp(-(x / T) ** 2) * np.sin(2 * np.pi * fc * x)
    s[t < start] = 0.0
    return s


def _gi(m, nodes, dof):
    return model.global_indices(m["gl"], np.ravel(nodes), dof)


def _inputs(c, seed):
    """What the march is given: scaled matrices, signals, forced and monitored DOFs."""
    rng = np.random.default_rng(seed)
    ms = _models(c)
    scale = rng.uniform(0.94, 1.0)
    t = np.arange(c["n_t"]) * ms[0]["dt"]
    fc = rng.uniform(4e6, 5e6) if ms[0]["nds"].shape[1] == 2 else rng.uniform(2e6, 3e6)
    d = dict(ms=ms, t=t, dt=t[1] - t[0], rng=rng, fc=fc, scale=scale, K=[m["K"] * scale for m in ms],
             C=[m["C"] for m in ms], M=[m["M"] for m in ms], gl=[m["gl"] for m in ms])
    n_src = len(ms[0]["src"])
    if c["kind"] in ("call", "run"):
        pick = int(rng.integers(n_src))
        d["fi"] = _gi(ms[0], ms[0]["src"][pick], ms[0]["src_dof"])
        d["F"] = rng.uniform(0.5, 2.0) * _burst(t, fc)[None, :]
    elif c["kind"] in ("batch", "adjoint"):
        offs = np.concatenate([[0], np.cumsum([m["K"].shape[0] for m in ms])])
        d["offs"] = offs
        d["fi"] = [np.concatenate([_gi(m, m["src"][r], m["src_dof"]) + o for m, o in zip(ms, offs)])
                   for r in range(n_src)]
        amp = rng.uniform(0.5, 2.0, n_src)
        d["F"] = np.asfortranarray(_burst(t, fc)[None, :, None] * amp[None, None, :])
    else:
        return d
    if c["kind"] in ("batch", "adjoint"):
        d["hi"] = np.concatenate([_gi(m, m["mon_nodes"], m["mon_dof"]) + o for m, o in zip(ms, d["offs"])])
    else:
        d["hi"] = _gi(ms[0], ms[0]["mon_nodes"], ms[0]["mon_dof"])
    return d


def _line(c, m):
    """Nodes along the left edge whose vertical displacement is prescribed."""
    left = np.nonzero(np.isclose(m["nds"][:, 0], 0.0))[0]
    return left[np.linspace(0, left.size - 1, min(c["n_dsp"], left.size)).astype(int)] + 1


# ---------------------------------------------------------------------------
# State and pass

def prepare(case, seed):
    c = case
    if c["kind"] == "fmc":
        return _fmc_state(c, seed)
    d = _inputs(c, seed)
    m, s = d["ms"][0], dict(case=c, d=d)
    inf = float("inf")
    s["every"] = c["every"] if c.get("every") else inf
    if c["kind"] == "run":
        s["plan"] = bfe_gb300.Plan(d["K"][0], d["C"][0], d["M"][0], d["dt"], bfe_gb300.VEL_CURRENT, c["prec"],
                                   d["gl"][0], one_source=True)
    elif c["kind"] == "batch" and c["n_models"] > 1:
        s["plan"], _ = bfe_gb300.Plan.multi(list(zip(d["K"], d["C"], d["M"], d["gl"])), d["dt"],
                                            bfe_gb300.VEL_CURRENT, c["prec"])
    elif c["kind"] in ("batch", "adjoint"):
        s["plan"] = bfe_gb300.Plan(d["K"][0], d["C"][0], d["M"][0], d["dt"], bfe_gb300.VEL_CURRENT, c["prec"],
                                   d["gl"][0])
    elif c["kind"] == "v5":
        s["plan"] = bfe_gb300.Plan(d["K"][0], d["C"][0], d["M"][0], d["dt"], bfe_gb300.V5, c["prec"], d["gl"][0],
                                   one_source=True)
    if c["kind"] == "adjoint":
        ke, mh, ch, dof = m["element_data"]
        s["elements"] = (ke * d["scale"], mh, ch, dof)
        # observed A-scans: bursts at surface-wave arrival times, of the size of the plate's response
        x = m["nds"][np.asarray(m["rec_nodes"]) - 1, 0]
        xs = m["nds"][[n[0] - 1 for n in m["src"]], 0]
        size = 1.0 / (E0 / (2 * (1 + NU)))
        s["obs"] = np.asfortranarray(np.stack([np.stack([
            size * d["rng"].uniform(0.2, 1.0) * _burst(d["t"], d["fc"], abs(a - b) / 2900.0) for a in x])
            for b in xs], axis=2))
    elif c["kind"] == "v5":
        rng, t = d["rng"], d["t"]
        line = _line(c, m)
        s["di"] = _gi(m, line, 2)
        s["D"] = 1e-9 * rng.uniform(0.5, 1.0, (s["di"].size, 1)) * _burst(t, d["fc"])[None, :]
        s["fi"] = _gi(m, m["src"][0], 2)
        s["F"] = rng.uniform(0.5, 2.0) * _burst(t, d["fc"], 0.1 * t[-1])[None, :]
        s["hi"] = _gi(m, m["mon_nodes"], 2)
    elif c["kind"] == "entry":
        rng, t = d["rng"], d["t"]
        s["mod"] = dict(nds=m["nds"], els=m["els"], el_mat_i=np.ones(m["els"].shape[0], np.int64),
                        el_abs_i=np.zeros(m["els"].shape[0]))
        s["matls"] = [dict(rho=RHO, D=model.isotropic_stiffness(E0 * d["scale"], NU), el_typ="CPE3")]
        s["steps"] = [dict(load=dict(time=t, frc_nds=np.asarray(src), frc_dfs=np.full(len(src), 2),
                                     frcs=rng.uniform(0.5, 2.0) * _burst(t, d["fc"])[None, :]),
                           mon=dict(nds=np.asarray(m["mon_nodes"]), dfs=np.full(len(m["mon_nodes"]), 2)))
                      for src in m["src"]]
        s["opt"] = dict(dof_to_use=[1, 2], solver_precision=c["prec"], field_output_every_n_frames=s["every"],
                        field_output_type="KE")
    return s


def _cast(c, *arrays):
    """Outputs of an FP32 march as FP32 (None where there is none)."""
    return [a if a is None or c["prec"] == "double" else a.astype(np.float32) for a in arrays]


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "fmc":
        return bfe_gb300.fn_parse_to_fmc_gb300(s["tx"], s["rx"], s["mon"], s["hist"], s["nds"], s["wts"], s["sig"])
    d = s["d"]
    if c["kind"] == "call":
        h, f, _, _ = bfe_gb300.fn_explicit_dynamic_solver_gb300(
            d["K"][0], d["C"][0], d["M"][0], d["t"], d["fi"], d["F"], [], [], d["hi"], s["every"], 1, "raw(u)",
            bfe_gb300.VEL_CURRENT, c["prec"], gl_lookup=d["gl"][0])
        return _cast(c, h, f)
    if c["kind"] == "run":
        h, f, _ = s["plan"].run(d["t"], d["fi"], d["F"], d["hi"], s["every"], False)
        return _cast(c, h, f)
    if c["kind"] == "batch":
        return _cast(c, s["plan"].run_batched(d["t"], d["fi"], d["F"], d["hi"]))
    if c["kind"] == "v5":
        h, _, f, _ = s["plan"].run_v5(d["t"], s["fi"], s["F"], s["di"], s["D"], s["hi"])
        return _cast(c, h, f)
    if c["kind"] == "adjoint":
        J, gs, gr, h = s["plan"].adjoint_gradient(s["elements"], d["t"], d["fi"], d["F"], d["hi"], s["obs"],
                                                  return_history=True)
        return _cast(c, np.array([J]), gs, gr, h)
    res, _ = fn_BristolFE_v2_gb300(s["mod"], s["matls"], s["steps"], s["opt"])
    return [_cast(c, r["dsps"], r["fld"]) for r in res]


# ---------------------------------------------------------------------------
# Work of a pass: inputs read once, outputs written once; the arithmetic of every step

def work(case):
    c = case
    if c["kind"] == "fmc":
        n_pairs, q = c["n_el"] ** 2, c["n_el"] * c["per_el"]
        # the convolution by FFTs of 2 n_t points, one each way
        L = 2 * c["n_t"]
        return dict(bytes=8.0 * c["n_t"] * (q * c["n_el"] + n_pairs), flops=2 * 2.5 * L * math.log2(L) * n_pairs)
    ms = _models(c)
    n = sum(m["K"].shape[0] for m in ms)
    nnz = sum(m["K"].nnz for m in ms)
    R, b = c.get("R", c.get("n_src", 1)), 8 if c["prec"] == "double" else 4
    q = c.get("n_rec", c.get("n_mon", 16)) * len(ms)
    T, n_el = c["n_t"], ms[0]["els"].shape[0]
    frames = -(-T // c["every"]) if c.get("every") else 0
    byt = nnz * (b + 4.0) + 2.0 * n * b + 8.0 * R * T * (1 + q)
    flops = T * R * (2.0 * nnz + 4.0 * n)
    if c["kind"] in ("call", "run"):
        byt += 8.0 * n * frames
    elif c["kind"] == "entry":
        byt += 8.0 * n_el * frames * R
    elif c["kind"] == "v5":
        byt += 16.0 * T * c["n_dsp"]
    elif c["kind"] == "adjoint":
        byt += n_el * (36 + 12) * 8.0 + 16.0 * n_el + 8.0 * R * T * q
        flops = 2 * flops + T * R * n_el * (2.0 * 36 + 12 + 36)
    return dict(bytes=byt, flops=flops)


# ---------------------------------------------------------------------------
# The same in 64 bits, by plain torch

def _csr(A):
    A = A.tocsr()
    return torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)),
                                   torch.from_numpy(A.indices.astype(np.int64)),
                                   torch.from_numpy(A.data.astype(np.float64)), size=A.shape,
                                   check_invariants=False).cuda()


def _blocks(parts):
    """Block-diagonal (rows, columns, values) of CSR matrices."""
    r, c, v, o = [], [], [], 0
    for A in parts:
        A = A.tocsr()
        r.append(np.repeat(np.arange(A.shape[0]), np.diff(A.indptr)) + o)
        c.append(A.indices.astype(np.int64) + o)
        v.append(A.data.astype(np.float64))
        o += A.shape[0]
    return np.concatenate(r), np.concatenate(c), np.concatenate(v), o


class _Operators:
    """P u+ = dt^2 M^-1 (f - K u) + 2 u - (I - G) u-, with G = dt/2 M^-1 C and P = I + G."""

    def __init__(self, K, C, M, dt):
        r, c, v, n = _blocks(K)
        coo = torch.sparse_coo_tensor(torch.from_numpy(np.stack([r, c])), torch.from_numpy(v), (n, n)).cuda()
        self.n, self.dt, self.K = n, dt, coo.coalesce().to_sparse_csr()
        mr, mc, mv, _ = _blocks(M)
        self.m = torch.from_numpy(np.bincount(mc, mv, n)).cuda()[:, None]
        cr, cc, cv, _ = _blocks(C)
        dg = cr == cc
        g = dt / 2 * np.bincount(cr[dg], cv[dg], n) / self.m[:, 0].cpu().numpy()
        self.g = torch.from_numpy(g).cuda()[:, None]
        off = ~dg
        self.ix = None
        if off.any():
            ix = np.unique(np.concatenate([cr[off], cc[off]]))
            loc = np.zeros(n, np.int64)
            loc[ix] = np.arange(ix.size)
            G = torch.zeros((ix.size, ix.size), dtype=torch.float64, device="cuda")
            mo = self.m[:, 0].cpu().numpy()
            G.index_put_((torch.from_numpy(loc[cr[off]]).cuda(), torch.from_numpy(loc[cc[off]]).cuda()),
                         torch.from_numpy(dt / 2 * cv[off] / mo[cr[off]]).cuda(), accumulate=True)
            self.ix, self.Go = torch.from_numpy(ix).cuda(), G
            self.Pi = torch.linalg.inv(torch.eye(ix.size, dtype=torch.float64, device="cuda") + G +
                                       torch.diag(self.g[self.ix, 0]))

    def step(self, un, up, f_idx=None, f_val=None):
        b = 2 * un - (1 - self.g) * up - (self.dt ** 2 / self.m) * (self.K @ un)
        if f_idx is not None:
            b.index_put_(f_idx, (self.dt ** 2 / self.m)[f_idx[0], 0] * f_val, accumulate=True)
        if self.ix is not None:
            b[self.ix] = b[self.ix] + self.Go @ up[self.ix]
        out = b / (1 + self.g)
        if self.ix is not None:
            out[self.ix] = self.Pi @ b[self.ix]
        return out


def _forced(fi, F):
    """Index pairs (row, source) and their signals [n_t][entries] (one signal row per source)."""
    rows = np.concatenate([np.unique(np.asarray(x)) - 1 for x in fi])
    src = np.concatenate([np.full(np.unique(np.asarray(x)).size, r) for r, x in enumerate(fi)])
    sig = torch.from_numpy(np.ascontiguousarray(F[0][:, src])).cuda()
    return (torch.from_numpy(rows).cuda(), torch.from_numpy(src).cuda()), sig


def _march(op, fi, F, hi, every=0, keep=False):
    """Histories (q, n_t, R), frames [(n, R)] and, with keep, every state."""
    R, n_t = len(fi), F.shape[1]
    idx, sig = _forced(fi, F)
    mon = torch.from_numpy(np.asarray(hi) - 1).cuda()
    up = torch.zeros((op.n, R), dtype=torch.float64, device="cuda")
    un, hist, frames, states = torch.zeros_like(up), [], [], []
    start = int(np.argmax(np.abs(F).max(axis=(0, 2)) > 0))
    for k in range(n_t):
        if k >= start:
            un, up = op.step(un, up, idx, sig[k]), un
        hist.append(un[mon])
        if every and k % every == 0:
            frames.append(un)
        if keep:
            states.append(un)
    return torch.stack(hist, 1), frames, states


def exact(case, seed):
    c = case
    if c["kind"] == "fmc":
        return _fmc_exact(c, seed)
    d = _inputs(c, seed)
    if c["kind"] == "entry":
        return _entry_exact(c, seed, d)
    if c["kind"] == "v5":
        return _v5_exact(c, seed, d)
    if c["kind"] == "batch" and c["n_t"] * c["R"] * sum(K.nnz for K in d["K"]) > 6e11:
        return None                                     # over 20 seconds
    op = _Operators(d["K"], d["C"], d["M"], d["dt"])
    if c["kind"] == "adjoint":
        return _adjoint_exact(c, seed, d, op)
    if c["kind"] == "batch":
        return [_march(op, d["fi"], d["F"], d["hi"])[0].cpu().numpy()]
    h, frames, _ = _march(op, [d["fi"]], d["F"][:, :, None], d["hi"], c["every"])
    return [h[:, :, 0].cpu().numpy(), torch.cat(frames, 1).cpu().numpy() if frames else None]


def _v5_exact(c, seed, d):
    s = prepare(case=c, seed=seed)
    s["plan"].close()
    K, dt = _csr(d["K"][0]), d["dt"]
    n = K.shape[0]
    m = torch.from_numpy(np.asarray(d["M"][0].sum(0)).ravel()).cuda()
    di, fi, hi = (torch.from_numpy(np.asarray(x) - 1).cuda() for x in (s["di"], s["fi"], s["hi"]))
    D, F = torch.from_numpy(s["D"]).cuda(), torch.from_numpy(s["F"]).cuda()
    pad = torch.cat([torch.zeros((D.shape[0], 2), dtype=D.dtype, device="cuda"), D], 1)
    acc = (pad[:, 2:] - 2 * pad[:, 1:-1] + pad[:, :-2]) / dt ** 2
    u, v = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    hist, frc = [], []
    start = int(np.argmax((np.abs(s["D"]).max(0) > 0) | (np.abs(s["F"]).max(0) > 0)))
    for k in range(c["n_t"]):                            # the plate has no damping
        if k < start:
            hist.append(torch.zeros_like(u[hi]))
            frc.append(torch.zeros_like(acc[:, k]))
            continue
        ku = K @ u
        a = -ku
        a[fi] += F[0, k]
        v = v + dt * a / m
        u = u + dt * v
        u[di] = D[:, k]
        hist.append(u[hi])
        frc.append(m[di] * acc[:, k] + ku[di])
    return [torch.stack(hist, 1).cpu().numpy(), torch.stack(frc, 1).cpu().numpy()]


def _entry_exact(c, seed, d):
    """The plate assembled here (two displacement DOFs per node), marched, frames as sqrt of kinetic energy."""
    s = prepare(case=c, seed=seed)
    nds, els = s["mod"]["nds"], s["mod"]["els"][:, :3] - 1
    x, y = nds[els, 0], nds[els, 1]
    J = (x[:, 0] - x[:, 2]) * (y[:, 1] - y[:, 2]) - (x[:, 1] - x[:, 2]) * (y[:, 0] - y[:, 2])
    gx = np.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], 1) / J[:, None]
    gy = np.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], 1) / J[:, None]
    B = np.zeros((els.shape[0], 3, 6))
    B[:, 0, 0::2], B[:, 1, 1::2], B[:, 2, 0::2], B[:, 2, 1::2] = gx, gy, gy, gx
    D = np.asarray(s["matls"][0]["D"])[np.ix_([0, 1, 5], [0, 1, 5])]
    ke = B.transpose(0, 2, 1) @ D @ B * (0.5 * J)[:, None, None]
    dof = (2 * els[:, :, None] + np.arange(2)).reshape(-1, 6)
    n = 2 * nds.shape[0]
    op = _Operators.__new__(_Operators)
    ind = np.stack([np.repeat(dof, 6, 1).ravel(), np.tile(dof, (1, 6)).ravel()])
    op.n, op.dt, op.ix = n, d["dt"], None
    op.K = torch.sparse_coo_tensor(torch.from_numpy(ind), torch.from_numpy(ke.ravel()), (n, n)).cuda().coalesce()
    op.K = op.K.to_sparse_csr()
    mass = np.bincount(dof.ravel(), np.repeat(RHO * J / 6.0, 6), n)
    op.m, op.g = torch.from_numpy(mass).cuda()[:, None], torch.zeros((n, 1), dtype=torch.float64, device="cuda")
    out, e = [], torch.from_numpy(els).cuda()
    for st in s["steps"]:
        fi = [2 * (np.asarray(st["load"]["frc_nds"]) - 1) + 2]
        hi = 2 * (np.asarray(st["mon"]["nds"]) - 1) + 2
        every = c["every"] or 0
        h, _, states = _march(op, fi, np.asarray(st["load"]["frcs"])[:, :, None], hi, 0, keep=bool(every))
        fld = None
        if every:
            cols = []
            for k in range(0, c["n_t"], every):
                v = (states[k] - (states[k - 1] if k else 0 * states[k]))[:, 0] / op.dt
                if k < int(np.argmax(np.abs(st["load"]["frcs"][0]) > 0)):
                    v = 0 * v
                ke_n = (op.m[:, 0] * v * v).reshape(-1, 2).sum(1)
                cols.append(torch.sqrt(0.5 * ke_n[e].mean(1)))
            fld = torch.stack(cols, 1).cpu().numpy()
        out.append([h[:, :, 0].cpu().numpy(), fld])
    return out


def _adjoint_exact(c, seed, d, op):
    s = prepare(case=c, seed=seed)
    s["plan"].close()
    ke, mh, ch, dof = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in s["elements"])
    h, _, u = _march(op, d["fi"], d["F"], d["hi"], keep=True)
    res = h - torch.from_numpy(s["obs"]).cuda()
    start = int(np.argmax(np.abs(d["F"]).max(axis=(0, 2)) > 0))
    J = 0.5 * (res[:, start:] ** 2).sum()
    mon, R, dt = torch.from_numpy(np.asarray(d["hi"]) - 1).cuda(), res.shape[2], op.dt
    l1 = torch.zeros((op.n, R), dtype=torch.float64, device="cuda")
    l2, gs, gr = torch.zeros_like(l1), torch.zeros(dof.shape[0], dtype=torch.float64, device="cuda"), None
    gr, zero = torch.zeros_like(gs), torch.zeros_like(l1)
    for k in range(c["n_t"] - 1, start - 1, -1):
        # (M + dt/2 C) lam = r + (2 M - dt^2 K) lam+ - (M - dt/2 C) lam++
        b = 2 * l1 - (1 - op.g) * l2 - (dt ** 2 / op.m) * (op.K @ l1)
        b.index_add_(0, mon, res[:, k] / op.m[mon])
        lam, l2 = b / (1 + op.g), l1
        l1 = lam
        u0, u1, u2 = u[k], u[k - 1] if k >= 1 else zero, u[k - 2] if k >= 2 else zero
        le, ue = lam[dof], u1[dof]                                   # (n_el, 6, R)
        gs -= dt ** 2 * (le * torch.bmm(ke, ue)).sum((1, 2))
        w, v = lam * (u0 - 2 * u1 + u2), lam * (u0 - u2)
        gr -= (mh * w.sum(1)[dof] + 0.5 * dt * ch * v.sum(1)[dof]).sum(1)
    return [J.reshape(1).cpu().numpy(), gs.cpu().numpy(), gr.cpu().numpy(), h.cpu().numpy()]


# ---------------------------------------------------------------------------
# Full-matrix capture from histories

def _fmc_state(c, seed):
    """Histories of every element's nodes for each transmitter, as a batched run leaves them."""
    rng = np.random.default_rng(seed)
    n, per, n_t = c["n_el"], c["per_el"], c["n_t"]
    t = np.arange(n_t) * 6.3e-9
    nds = [np.arange(1 + per * k, 1 + per * (k + 1)) for k in range(n)]
    delay = rng.uniform(0, 0.6 * t[-1], (n * per, n))
    centre = t[None, :, None] - delay[:, None, :]
    hist = 1e-11 * np.exp(-(centre / 1.5e-7) ** 2) * np.sin(2 * np.pi * 5e6 * centre)
    tx, rx = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    sig = _burst(np.arange(c["n_sig"]) * 6.3e-9, 5e6, 0.0, 4)
    return dict(case=c, tx=tx.ravel(), rx=rx.ravel(), mon=[np.concatenate(nds)] * n, hist=np.asfortranarray(hist),
                nds=nds, wts=[rng.uniform(0.5, 1.0, per) for _ in range(n)], sig=sig)


def _fmc_exact(c, seed):
    s = _fmc_state(c, seed)
    h = torch.from_numpy(s["hist"]).cuda()
    n, per, n_t = c["n_el"], c["per_el"], c["n_t"]
    w = torch.from_numpy(np.stack(s["wts"])).cuda()
    raw = (h.reshape(n, per, n_t, n) * w[:, :, None, None]).sum(1)             # (rx, n_t, tx)
    raw = raw.permute(1, 2, 0).reshape(n_t, n * n)                            # pair = tx * n + rx
    g = torch.fft.rfft(torch.from_numpy(s["sig"]).cuda(), 2 * n_t)
    return torch.fft.irfft(torch.fft.rfft(raw, 2 * n_t, dim=0) * g[:, None], 2 * n_t, dim=0)[:n_t].cpu().numpy()
