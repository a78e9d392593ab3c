"""Work that users of this framework run, as cases that can be prepared, run and checked.

The kinds of a case are the entry points that programs call:

pipeline   S, positions and wavelength per time step, on the GPU -> level images
           (Pipeline.process_device / images_device), one whole imaging call
staged     the same from pinned host buffers, images back on the host
           (Pipeline.stage_host_ptr / process_staged / images)
levels     batched eigenvalues that the energy levels are calibrated from
           (eigh_gram_batched, complex64 host arrays)
eigen      one time step's eigenpairs and the virtual visibilities of its levels
           (eigh_gram, virtual_vis), with or without beamforming, single or double precision
synthesis  level images of a dataset of eigenpairs (image_synthesis)
direct     the direct sum over baselines at given directions (nuft_sum)

Observations are seeded synthetic ones of bipp_b200.simulate; `ha` moves a block of time
steps away from transit, in steps, which sets the w extent of its baselines.
"""
import dataclasses
import math

import numpy as np
import torch

import bipp_b200 as bipp
from bipp_b200 import simulate as sim

_context = None


def context():
    """The program's one context."""
    global _context
    if _context is None:
        _context = bipp.Context("GPU", device=0)
    return _context


def listed():
    return [
        # one integration of a small array as it arrives: launches and latency
        {"name": "pipeline-60x1", "kind": "pipeline", "n": 60, "steps": 1, "ha": 0, "channels": 1, "keep": 1.0,
         "levels": 2, "filter": "lsq", "image": 256, "fov": 10.0, "eps": 1e-5, "wl": 2.0, "sources": 20},
        # a short block of a medium array off transit
        {"name": "pipeline-256x64", "kind": "pipeline", "n": 256, "steps": 64, "ha": -512, "channels": 1, "keep": 1.0,
         "levels": 4, "filter": "lsq", "image": 512, "fov": 16.0, "eps": 1e-5, "wl": 2.0, "sources": 100},
        # odd sizes, flagged antennas, another filter, a loose tolerance
        {"name": "pipeline-333x37", "kind": "pipeline", "n": 333, "steps": 37, "ha": 101, "channels": 1, "keep": 0.75,
         "levels": 5, "filter": "sqrt", "image": 701, "fov": 12.0, "eps": 1e-4, "wl": 1.7, "sources": 77},
        # a whole observation: the benchmark's batch
        {"name": "pipeline-512x2048", "kind": "pipeline", "n": 512, "steps": 2048, "ha": 0, "channels": 1,
         "keep": 0.74, "levels": 4, "filter": "lsq", "image": 1024, "fov": 16.0, "eps": 1e-5, "wl": 2.0,
         "sources": 200},
        # the largest array, several frequency channels, a quarter of the antennas flagged
        {"name": "pipeline-1024x64", "kind": "pipeline", "n": 1024, "steps": 8, "ha": 0, "channels": 8, "keep": 0.75,
         "levels": 8, "filter": "lsq", "image": 2048, "fov": 16.0, "eps": 1e-5, "wl": 2.0, "sources": 500},
        # one snapshot on a large image at a tight tolerance
        {"name": "pipeline-550x1-4096px", "kind": "pipeline", "n": 550, "steps": 1, "ha": 0, "channels": 1,
         "keep": 1.0, "levels": 8, "filter": "lsq", "image": 4096, "fov": 4.0, "eps": 1e-6, "wl": 0.21,
         "sources": 1000},
        # host data streamed through the staging slots, images read back every batch
        {"name": "staged-512x128", "kind": "staged", "n": 512, "steps": 128, "ha": 256, "channels": 1, "keep": 0.74,
         "levels": 4, "filter": "lsq", "image": 1024, "fov": 16.0, "eps": 1e-5, "wl": 2.0, "sources": 200},
        # energy-level calibration of a run from its first steps
        {"name": "levels-256x64", "kind": "levels", "n": 256, "steps": 64, "sources": 200},
        # one beamformed step of a station array through the reference's call
        {"name": "eigen-55-beams", "kind": "eigen", "n": 55, "beams": 55, "identity": False, "double": False,
         "levels": 4, "sources": 30},
        # a large step in double precision
        {"name": "eigen-512-double", "kind": "eigen", "n": 512, "beams": 512, "identity": True, "double": True,
         "levels": 2, "sources": 200},
        # level images of a dataset of precomputed eigenpairs
        {"name": "synthesis-512x16", "kind": "synthesis", "n": 512, "samples": 16, "levels": 4, "image": 1024,
         "fov": 16.0, "eps": 1e-5, "sources": 200},
        # direct evaluation of one step's baselines at chosen directions
        {"name": "direct-256", "kind": "direct", "n": 256, "pixels": 16384, "double": False, "sources": 100},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))


def draw(rng):
    kind = rng.choice(["pipeline"] * 6 + ["staged", "levels", "eigen", "eigen", "synthesis", "direct"])
    if kind in ("pipeline", "staged"):
        n = _logint(rng, 40, 900)
        channels = rng.choice([1, 1, 1, 4])
        steps = max(1, _logint(rng, 1, min(1024, 1.5e10 / n ** 3)) // channels)
        image = _logint(rng, 200, 2048)
        return {"kind": kind, "n": n, "steps": steps, "ha": rng.choice([0, 50, -400, 700]) if image <= 1024 else 0,
                "channels": channels, "keep": rng.choice([1.0, 0.9, 0.75]), "levels": rng.randint(1, 8 if image <= 1024 else 4),
                "filter": rng.choice(["lsq", "lsq", "lsq", "sqrt"]), "image": image, "fov": rng.choice([8.0, 12.0, 16.0]),
                "eps": rng.choice([1e-4, 1e-5, 1e-5, 1e-6]), "wl": rng.choice([1.5, 2.0, 3.0]),
                "sources": _logint(rng, 10, 500)}
    if kind == "levels":
        n = _logint(rng, 40, 600)
        return {"kind": kind, "n": n, "steps": _logint(rng, 4, min(256, 1.5e9 / n ** 3 + 4)), "sources": _logint(rng, 10, 300)}
    if kind == "eigen":
        double = rng.random() < 0.5
        n = _logint(rng, 30, 400 if double else 700)
        identity = rng.random() < 0.6
        return {"kind": kind, "n": n, "beams": n if identity else max(4, int(n * rng.uniform(0.4, 1.0))),
                "identity": identity, "double": double, "levels": rng.randint(1, 6), "sources": _logint(rng, 10, 200)}
    if kind == "synthesis":
        return {"kind": kind, "n": _logint(rng, 40, 512), "samples": _logint(rng, 1, 16), "levels": rng.randint(1, 6),
                "image": _logint(rng, 200, 1024), "fov": rng.choice([8.0, 16.0]), "eps": rng.choice([1e-3, 1e-4, 1e-5]),
                "sources": _logint(rng, 10, 200)}
    return {"kind": kind, "n": _logint(rng, 30, 400), "pixels": _logint(rng, 64, 16384), "double": rng.random() < 0.5,
            "sources": _logint(rng, 10, 100)}


# --- inputs ---------------------------------------------------------------------------

def _observation(case, seed, steps, ha=0, image=8, fov=16.0, wl=2.0):
    n = case["n"]
    cfg = sim.config_c2(n_antenna=n, n_steps=steps, n_src=case["sources"], image_size=image, fov_deg=fov, wl=wl,
                        seed=1000 + 7919 * int(seed), keep=None)
    cfg = dataclasses.replace(cfg, layout="logradial" if n >= 200 else "disc",
                              extent_m=(35000.0 if n >= 200 else 4000.0) * (1.0 if wl > 1.0 else 1.8),
                              src_radius_deg=min(8.0, 0.45 * fov))
    obs = sim.observation(cfg)
    obs.times = obs.times + ha * cfg.dt_s
    return cfg, obs


def _visibilities(case, seed):
    """S [T, N, N] (logical), positions [T, N, 3] and wavelengths [T] of a case's entries, on the GPU."""
    T, C, n = case["steps"], case["channels"], case["n"]
    cfg, obs = _observation(case, seed, T, case["ha"], case["image"], case["fov"], case["wl"])
    masks = None
    if case["keep"] < 1.0:
        rng = np.random.default_rng(cfg.seed + 2000)
        low = max(2, int(case["keep"] * n))
        masks = np.zeros((T, n), dtype=bool)
        for t in range(T):
            masks[t, rng.permutation(n)[:int(rng.integers(low, n + 1))]] = True
    wls = np.linspace(0.75 * case["wl"], 1.5 * case["wl"], C) if C > 1 else [case["wl"]]
    S = torch.empty((T * C, n, n), dtype=torch.complex64, device="cuda")
    xyz = torch.empty((T * C, n, 3), dtype=torch.float64, device="cuda")
    wl = torch.empty((T * C,), dtype=torch.float64, device="cuda")
    chunk = max(1, min(64, 2 ** 24 // n ** 2))
    for s0 in range(0, T, chunk):
        steps = list(range(s0, min(T, s0 + chunk)))
        for c, w in enumerate(wls):
            s, x = sim.visibilities(obs, steps, device="cuda", dtype=torch.complex64, masks=masks, wl=float(w), noise_key=c)
            at = slice(s0 * C + c, (s0 + len(steps)) * C, C)
            S[at], xyz[at], wl[at] = s, x, float(w)
    return obs, S, xyz, wl


def _sinc_gram(xyz, wl):
    x = 2.0 * torch.cdist(xyz, xyz, compute_mode="donot_use_mm_for_euclid_dist") / wl
    return torch.special.sinc(x)


def _solve(S, xyz, wl, W=None, vectors=True):
    """Generalised eigenpairs of one step in 64 bits: eigenvalues, antenna-space eigenvectors (or
    None), kept rows. S is the logical matrix; zero rows and columns are flagged ones."""
    S = S.to(torch.complex128)
    S = torch.tril(S) + torch.tril(S, -1).mH
    keep = torch.nonzero((S.abs() > 0).any(0)).flatten()
    S = S[keep][:, keep]
    if W is None:
        G = _sinc_gram(xyz[keep], wl).to(torch.complex128)
    else:
        Wk = W[:, keep].to(torch.complex128)
        G = Wk.mH @ _sinc_gram(xyz, wl).to(torch.complex128) @ Wk
        G = 0.5 * (G + G.mH)
    L = torch.linalg.cholesky(G)
    A = torch.linalg.solve_triangular(L, S, upper=False)
    A = torch.linalg.solve_triangular(L, A.mH.contiguous(), upper=False)
    A = 0.5 * (A + A.mH)
    if not vectors:
        return torch.linalg.eigvalsh(A), None, keep
    d, y = torch.linalg.eigh(A)
    x = torch.linalg.solve_triangular(L.mH.contiguous(), y, upper=True)
    return d, x if W is None else Wk @ x, keep


def _intervals(d, levels):
    """Energy levels over the eigenvalues d: equal counts of those above a thousandth of the largest,
    each border in the widest of the gaps beside its place; the lowest level reaches down to zero."""
    d = np.sort(np.asarray(d, dtype=np.float64))
    d = d[d > 1e-3 * d[-1]]
    borders = []
    for k in range(1, levels):
        at = range(max(0, k * len(d) // levels - 3), min(len(d) - 1, k * len(d) // levels + 4))
        best = max(at, key=lambda i: d[i + 1] / d[i], default=None)
        borders.append(math.sqrt(d[best] * d[best + 1]) if best is not None else d[-1] * (1 + k))
    borders = np.array([0.0] + borders + [np.inf])
    return np.stack([borders[:-1], borders[1:]], axis=1)


def _calibrate(case, S, xyz, wl):
    m = min(S.shape[0], 1 if case["n"] > 256 else 4)
    at = np.linspace(0, S.shape[0] - 1, m).astype(int)
    d = [_solve(S[k], xyz[k], wl[k], vectors=False)[0].cpu().numpy() for k in at]
    return _intervals(np.concatenate(d), case["levels"])


def _pipeline(case, obs, intervals, entries):
    n = case["image"]
    lm = obs.lmn[:, :2].reshape(n, n, 2)
    (l0, m0), (la, ma), (lb, mb) = lm[0, 0], lm[1, 0] - lm[0, 0], lm[0, 1] - lm[0, 0]
    return bipp.Pipeline(context(), case["n"], intervals, (n, n, l0, m0, la, lb, ma, mb), obs.lmn[:, 2], obs.basis,
                         tolerance=case["eps"], filter=case["filter"], chunk_steps=min(entries, 512), max_steps=entries)


def _step(case, seed, steps):
    """Host arrays of `steps` steps through the simulator: S, positions, wavelength."""
    cfg, obs = _observation(case, seed, steps)
    s, x = sim.visibilities(obs, list(range(steps)), device="cuda", dtype=torch.complex128)
    return obs, s, x, cfg.wl


def _eigen_inputs(case, seed):
    obs, s, x, wl = _step(case, seed, 1)
    s, x = s[0], x[0]
    W = None
    if not case["identity"]:
        rng = np.random.default_rng(5000 + int(seed))
        W = rng.standard_normal((case["n"], case["beams"])) + 1j * rng.standard_normal((case["n"], case["beams"]))
        W = torch.from_numpy(np.linalg.qr(W)[0]).cuda()   # orthonormal beams
        s = W.mH @ s @ W
    if not case["double"]:
        s, x = s.to(torch.complex64).to(torch.complex128), x.float().double()
        W = W if W is None else W.to(torch.complex64).to(torch.complex128)
    d, v, _ = _solve(s, x, wl, W)
    return s, x, wl, W, d, v, _intervals(d.cpu().numpy(), case["levels"])


def _synthesis_inputs(case, seed):
    obs, s, x, wl = _step({**case}, seed, case["samples"])
    lmn = sim.make_lmn_grid(case["image"], math.radians(case["fov"])).astype(np.float32)
    d, v = torch.linalg.eigh(s.to(torch.complex64))
    d, v, x = d.cpu().numpy(), v.cpu().numpy(), x.cpu().numpy()
    uvw = [sim.baseline_uvw(obs, xk) for xk in x]
    return obs, wl, d, v, uvw, lmn, _intervals(d[0], case["levels"])


def _direct_inputs(case, seed):
    obs, s, x, wl = _step(case, seed, 1)
    ct, rt = (np.complex128, np.float64) if case["double"] else (np.complex64, np.float32)
    uvw = (sim.baseline_uvw(obs, x[0].cpu().numpy()).astype(np.float64) * (2.0 * math.pi / wl)).astype(rt)
    rng = np.random.default_rng(6000 + int(seed))
    lm = rng.uniform(-0.14, 0.14, (2, case["pixels"]))
    lmn = np.stack([lm[0], lm[1], np.sqrt(1.0 - lm[0] ** 2 - lm[1] ** 2)]).astype(rt)
    values = s[0].cpu().numpy().reshape(-1, order="F").astype(ct)
    return values, np.ascontiguousarray(uvw.T), lmn


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind}
    if kind in ("pipeline", "staged"):
        obs, S, xyz, wl = _visibilities(case, seed)
        intervals = _calibrate(case, S, xyz, wl)
        T = S.shape[0]
        S = S.transpose_(1, 2)   # each step's matrix in column-major order
        S = S if S.is_contiguous() else S.contiguous()
        state.update(entries=T, pipe=_pipeline(case, obs, intervals, T), S=S, xyz=xyz, wl=wl)
        if kind == "staged":
            state.update(S=S.cpu().pin_memory(), xyz=xyz.cpu().pin_memory(), wl=wl.cpu().pin_memory())
        else:
            state["images"] = torch.zeros((case["levels"], case["image"] ** 2), dtype=torch.float32, device="cuda")
    elif kind == "levels":
        _, s, x, wl = _step(case, seed, case["steps"])
        state.update(s=s.to(torch.complex64).cpu().numpy(), xyz=x.cpu().numpy(),
                     wl=np.full(case["steps"], wl, dtype=np.float32))
    elif kind == "eigen":
        s, x, wl, W, _, _, intervals = _eigen_inputs(case, seed)
        ct, rt = (np.complex128, np.float64) if case["double"] else (np.complex64, np.float32)
        W = np.eye(case["n"]) if W is None else W.cpu().numpy()
        state.update(s=np.asfortranarray(s.cpu().numpy(), dtype=ct), xyz=np.asfortranarray(x.cpu().numpy(), dtype=rt),
                     wl=rt(wl), w=np.asfortranarray(W, dtype=ct), intervals=intervals)
    elif kind == "synthesis":
        _, wl, d, v, uvw, lmn, intervals = _synthesis_inputs(case, seed)
        ds = bipp.InMemoryDataset(case["n"], case["n"])
        for k in range(case["samples"]):
            ds.write(k, wl, 1.0 / case["n"] ** 2, v[k], d[k], uvw[k])
        selection = {"level%d" % i: {k: d[k] * ((d[k] >= lo) & (d[k] <= hi)) for k in range(case["samples"])}
                     for i, (lo, hi) in enumerate(intervals)}
        state.update(ds=ds, selection=selection, lmn=lmn, options=bipp.NufftSynthesisOptions().set_tolerance(case["eps"]))
    else:
        values, uvw, lmn = _direct_inputs(case, seed)
        state.update(values=values, uvw=uvw, lmn=lmn)
    context()
    torch.cuda.synchronize()   # the library works on its own stream
    return state


# --- one pass -------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "pipeline":
        p = state["pipe"]
        p.reset()
        p.process_device(state["entries"], state["S"].data_ptr(), state["xyz"].data_ptr(), state["wl"].data_ptr())
        p.images_device(state["images"].data_ptr())
        return state["images"]
    if kind == "staged":
        p = state["pipe"]
        p.reset()
        p.stage_host_ptr(state["entries"], state["S"].data_ptr(), state["xyz"].data_ptr(), state["wl"].data_ptr())
        p.process_staged()
        return p.images()
    if kind == "levels":
        _, d, nred, scale = bipp.eigh_gram_batched(state["wl"], state["s"], state["xyz"], ctx=context())
        return d, nred, scale
    if kind == "eigen":
        v, d, scale = bipp.eigh_gram(state["wl"], state["s"], state["w"], state["xyz"], ctx=context())
        vv = [bipp.virtual_vis(scale, np.where((d >= lo) & (d <= hi), d, 0), v, ctx=context())
              for lo, hi in state["intervals"]]
        return d, scale, vv
    if kind == "synthesis":
        return bipp.image_synthesis(context(), state["options"], state["ds"], state["selection"], state["lmn"])
    u, x = state["uvw"], state["lmn"]
    return bipp.nuft_sum(1.0, state["values"], u[0], u[1], u[2], x[0], x[1], x[2], ctx=context())


# --- the same in 64 bits --------------------------------------------------------------

def _direct_sum(values, uvw, lmn):
    """Re sum_k values[c, k] exp(i uvw[k] . lmn[p]) for every c and p, in 64 bits."""
    out = torch.zeros((values.shape[0], lmn.shape[0]), dtype=torch.float64, device="cuda")
    chunk = max(1, 2 ** 27 // max(1, uvw.shape[0]))
    for p0 in range(0, lmn.shape[0], chunk):
        phase = uvw @ lmn[p0:p0 + chunk].T
        out[:, p0:p0 + chunk] = values.real @ torch.cos(phase) - values.imag @ torch.sin(phase)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pipeline", "staged"):
        T, P, n = case["steps"] * case["channels"], case["image"] ** 2, case["n"]
        if T * P * n * n / 2 > 6e10 or T * n ** 3 > 1e9:
            return None
        obs, S, xyz, wl = _visibilities(case, seed)
        intervals = _calibrate(case, S, xyz, wl)
        lmn = torch.from_numpy(obs.lmn).cuda()
        basis = torch.from_numpy(obs.basis).cuda()
        out = torch.zeros((case["levels"], P), dtype=torch.float64, device="cuda")
        for k in range(T):
            d, x, keep = _solve(S[k], xyz[k], wl[k])
            seen = torch.tril(S[k]).to(torch.complex128)
            eps = float(np.finfo(np.float32).eps)
            full = (seen + torch.tril(seen, -1).mH).abs() ** 2 > eps
            scale = 1.0 / float(full.sum())
            f = torch.sqrt(d.clamp(min=0)) if case["filter"] == "sqrt" else d
            au = (xyz[k][keep] @ basis) * (2.0 * math.pi / float(wl[k]))
            i, j = torch.tril_indices(len(keep), len(keep), -1, device="cuda")
            vv = []
            for lo, hi in intervals:
                g = torch.where((d >= lo) & (d <= hi), f, torch.zeros_like(f)) * scale
                vv.append((x * g) @ x.mH)
            vv = torch.stack(vv)
            out += 2.0 * _direct_sum(vv[:, i, j], au[i] - au[j], lmn)
            out += torch.diagonal(vv.real, dim1=1, dim2=2).sum(1)[:, None]
        return out / T
    if kind == "levels":
        if case["steps"] * case["n"] ** 3 > 4e9:
            return None
        _, s, x, wl = _step(case, seed, case["steps"])
        s, x = s.to(torch.complex64), x.float().double()
        d = torch.stack([_solve(s[k], x[k], wl, vectors=False)[0] for k in range(case["steps"])])
        return d, None, None
    if kind == "eigen":
        s, x, wl, W, d, v, intervals = _eigen_inputs(case, seed)
        eps = float(np.finfo(np.float64 if case["double"] else np.float32).eps)
        scale = 1.0 / float((s.abs() ** 2 > eps).sum())
        vv = [(v * torch.where((d >= lo) & (d <= hi), d, torch.zeros_like(d)) * scale) @ v.mH for lo, hi in intervals]
        return d, scale, [w.cpu().numpy() for w in vv]
    if kind == "synthesis":
        if case["samples"] * case["image"] ** 2 * case["n"] ** 2 > 6e10:
            return None
        _, wl, d, v, uvw, lmn, intervals = _synthesis_inputs(case, seed)
        lmn = torch.from_numpy(lmn.astype(np.float64)).cuda()
        out = torch.zeros((case["levels"], lmn.shape[0]), dtype=torch.float64, device="cuda")
        for k in range(case["samples"]):
            vk = torch.from_numpy(v[k]).cuda().to(torch.complex128)
            dk = torch.from_numpy(d[k].astype(np.float64)).cuda()
            vv = torch.stack([((vk * torch.where((dk >= lo) & (dk <= hi), dk, torch.zeros_like(dk))) @ vk.mH).mT.reshape(-1)
                              for lo, hi in intervals]) / case["n"] ** 2
            out += _direct_sum(vv, torch.from_numpy(uvw[k].astype(np.float64) * (2.0 * math.pi / wl)).cuda(), lmn)
        return {"level%d" % i: out[i] / case["samples"] for i in range(case["levels"])}
    values, uvw, lmn = _direct_inputs(case, seed)
    to = [torch.from_numpy(a).cuda() for a in (values.astype(np.complex128)[None], uvw.T.astype(np.float64).copy(),
                                               lmn.T.astype(np.float64).copy())]
    return _direct_sum(*to)[0]


# --- what a pass cannot do without ----------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; arithmetic of the eigensolves (real operations of
    the dense algorithm), of the kernel sums over the points' supports and of the FFT of the image's cells."""
    kind, n = case["kind"], case["n"]
    solve = (1.0 / 3 + 3.0 + 16.0 / 3 + 4.0) * n ** 3
    if kind in ("pipeline", "staged"):
        T, L, P = case["steps"] * case["channels"], case["levels"], case["image"] ** 2
        W = math.ceil(-math.log(case["eps"]) / (math.pi * math.sqrt(1.0 - 1.0 / 1.75)))
        nk = n * (0.5 + 0.5 * case["keep"])
        points = T * nk * nk / 2
        return {"bytes": T * (4.0 * nk * nk + 24.0 * n) + 4.0 * L * P,
                "flops": T * solve * (nk / n) ** 3 + points * L * 4.0 * W ** 3 + 15.0 * L * P * math.log2(P)}
    if kind == "levels":
        return {"bytes": case["steps"] * 12.0 * n * n, "flops": case["steps"] * solve}
    if kind == "eigen":
        m, size = case["beams"], 16.0 if case["double"] else 8.0
        beam = 0.0 if case["identity"] else 4.0 * n * n * m + 8.0 * n * m * m
        return {"bytes": size * (0.5 * m * m + (0 if case["identity"] else n * m) + case["levels"] * n * n),
                "flops": (solve / n ** 3) * m ** 3 + beam + 8.0 * n * n * m}
    if kind == "synthesis":
        k, L, P = case["samples"], case["levels"], case["image"] ** 2
        W = math.ceil(-math.log(case["eps"]) / (math.pi * math.sqrt(1.0 - 1.0 / 1.75)))
        return {"bytes": k * (8.0 + 12.0) * n * n + 12.0 * P + 4.0 * L * P,
                "flops": k * (8.0 * n ** 3 + n * n / 2 * L * 4.0 * W ** 3) + 15.0 * L * P * math.log2(P)}
    size = 8.0 if case["double"] else 4.0
    return {"bytes": size * (5.0 * n * n + 4.0 * case["pixels"]), "flops": 20.0 * n * n * case["pixels"]}
