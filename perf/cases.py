"""The workloads this framework is timed on.

Three families, each through the package's public entry points:

* the reconstruction chain (PixelChain): single events through run_event, as the plain per-event
  chain and a trigger-like consumer use it, and streamed batches through the input slots, the
  captured graph and the batched export, as the benchmark streams them;
* local reconstruction alone (digis, clusters and rechits of one event, hits copied out), the
  producer boundary that stops before the tracking;
* the stand-alone track fits on device tensors: broken line, Riemann and the adjoint of the
  broken line (chi2 and its gradients for the alignment).

Events and tracks come from the package's seeded generator.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "cms-julia_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

B_FIELD = 0.0114256972711507  # 1 / (pT R) at 3.8 T, GeV^-1 cm^-1

# hit-count mix of the generator's fit tracks (3, 4, 5, then 6, 7 and 8 hits equally)
MEAN_HITS = 0.3 * 3 + 0.4 * 4 + 0.2 * 5 + 0.1 * 7


def listed():
    return [
        # one clean event of 100 tracks: the smallest call, where latency and launches count
        {"name": "event_100_tracks", "kind": "event", "mode": "single", "size": 100, "precision": 0},
        # one pileup-50 event: the plain per-event chain of the benchmark
        {"name": "event_pu50", "kind": "event", "mode": "pu", "size": 50, "precision": 0},
        # one dense event under the extended capacities, fits in mixed precision
        {"name": "event_pu170_mixed", "kind": "event", "mode": "pu", "size": 170, "precision": 1},
        # rechits of one pileup-140 event for a consumer that brings its own tracking
        {"name": "hits_pu140", "kind": "hits", "mode": "pu", "size": 140},
        # the throughput path: a streamed batch of pileup-50 events, launch shapes from the autotuner
        {"name": "batch_512_pu50", "kind": "batch", "mode": "pu", "size": 50, "events": 512, "precision": 0,
         "tuned": True},
        # uneven events (pileup 0 to 200), extended capacities, an odd count, default launch shapes
        {"name": "batch_111_uneven", "kind": "batch", "mode": "uniform", "size": 200, "events": 111, "precision": 0,
         "tuned": False},
        # the fit workload of the benchmark: mixed precision, 2^20 tracks
        {"name": "bl_mixed_1048576", "kind": "bl", "tracks": 1 << 20, "precision": 1},
        # FP64 fits as the reference computes them, a ragged count
        {"name": "bl_fp64_99991", "kind": "bl", "tracks": 99991, "precision": 0},
        # the tracks of one small event, where launches count
        {"name": "bl_mixed_1237", "kind": "bl", "tracks": 1237, "precision": 1},
        # Riemann fits, the alternative helix fit
        {"name": "riemann_fp64_262144", "kind": "rm", "tracks": 1 << 18, "precision": 0},
        # one alignment iteration: gradients with respect to hits and the module alignment
        {"name": "adjoint_align_524288", "kind": "adjoint", "tracks": 1 << 19, "align": True},
        # gradients of a small sample with respect to its hits alone
        {"name": "adjoint_5003", "kind": "adjoint", "tracks": 5003, "align": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["event", "event", "batch", "hits", "bl", "bl", "rm", "adjoint"])
    if kind == "event":
        if rng.random() < 0.3:
            return {"kind": kind, "mode": "single", "size": _log(rng, 10, 1000), "precision": rng.randrange(2)}
        return {"kind": kind, "mode": "pu", "size": rng.randint(5, 170), "precision": rng.randrange(2)}
    if kind == "hits":
        return {"kind": kind, "mode": "pu", "size": rng.randint(5, 140)}
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": kind, "mode": "pu", "size": rng.randint(30, 50), "events": _log(rng, 3, 480),
                    "precision": rng.randrange(2), "tuned": rng.random() < 0.5}
        return {"kind": kind, "mode": "uniform", "size": rng.randint(60, 200), "events": _log(rng, 3, 110),
                "precision": rng.randrange(2), "tuned": rng.random() < 0.5}
    if kind == "adjoint":
        return {"kind": kind, "tracks": _log(rng, 300, 1 << 19), "align": rng.random() < 0.5}
    return {"kind": kind, "tracks": _log(rng, 300, 1 << (20 if kind == "bl" else 18)), "precision": rng.randrange(2)}


# ------------------------------------------------------------------------------- inputs
def _events(case, seed, n):
    from pixeltrack import gen
    mode = {"single": gen.MODE_SINGLE, "pu": gen.MODE_PU, "uniform": gen.MODE_UNIFORM}[case["mode"]]
    return gen.events(n, mode, pu=float(case["size"]), ntracks=int(case["size"]), seed=seed)


def _tracks(case, seed):
    """Tracks of the generator in its order, each hit count at its exact share of the mix."""
    from pixeltrack import gen
    n = case["tracks"]
    w = gen.fit_tracks(int(1.1 * n) + 600, seed=seed)
    count = np.diff(w["offsets"])
    want = {k: int(n * share) for k, share in zip(range(4, 9), (0.4, 0.2, 0.1 / 3, 0.1 / 3, 0.1 / 3))}
    want[3] = n - sum(want.values())
    keep = np.sort(np.concatenate([np.nonzero(count == k)[0][:m] for k, m in want.items()]))
    offs = np.concatenate([[0], np.cumsum(count[keep])]).astype(np.int32)
    at = np.repeat(w["offsets"][keep] - offs[:-1], count[keep]) + np.arange(offs[-1])
    return {"hits": w["hits"][at], "ge": w["ge"][at], "module": w["module"][at], "offsets": offs}


def _alignment(seed):
    """Module centres and a misalignment: translations ~ N(0, 50 um), rotations ~ N(0, 0.1 mrad)."""
    from pixeltrack import gen
    pos = gen.module_positions()
    rng = np.random.default_rng(seed)
    align = np.zeros((pos.shape[0], 6), np.float32)
    align[:, :3] = rng.normal(0, 50e-4, (pos.shape[0], 3))
    align[:, 3:] = rng.normal(0, 1e-4, (pos.shape[0], 3))
    return pos, align


def prepare(case, seed):
    from pixeltrack import PRODUCTS, PixelChain, TrackExport, batch_params, extended_params, gen
    kind = case["kind"]
    if kind in ("event", "hits"):
        blob, offs = _events(case, seed, 1)
        dense = case["size"] > 60 and case["mode"] == "pu"
        params = extended_params(max_hits=65536, max_doublets=2_000_000, max_tuples=180_000,
                                 fit_precision=case.get("precision", 0)) if dense else \
            batch_params(1, words_per_event=300_000, hits_per_event_avg=49_152, doublets_per_event_avg=458_752,
                         tuples_per_event_avg=32_768, fit_precision=case.get("precision", 0))
        st = {"kind": kind, "chain": PixelChain(gen.conditions(), params), "event": blob}
        if kind == "event":
            st["out"] = TrackExport(1, 32768, 1024, cov=True)
            for t in st["out"].arrays.values():
                t.zero_()
        else:  # the consumer's hit collection
            st["hits"] = {k: np.zeros(65536, PRODUCTS[k][1]) for k in _HITS}
        return st
    if kind == "batch":
        n = case["events"]
        blob, offs = _events(case, seed, n)
        dense = case["mode"] == "uniform"
        words = int(np.diff(offs).max() // 4)
        params = batch_params(n, words_per_event=words, fit_precision=case["precision"], extended=dense,
                              **(dict(hits_per_event_avg=26_000, doublets_per_event_avg=420_000,
                                      tuples_per_event_avg=42_000) if dense else {}))
        chain = PixelChain(gen.conditions(), params)
        pinned = torch.from_numpy(blob).pin_memory()
        # room for the loose tracks: about 27 per unit of pileup
        out = TrackExport(n, n * 3600 + 6000 if dense else n * 1800 + 1000, n * 120 + 400, cov=True)
        for t in out.arrays.values():
            t.zero_()
        st = {"kind": kind, "chain": chain, "pinned": pinned, "blob": pinned.numpy(), "offs": offs, "out": out,
              "copy": torch.cuda.Stream(), "compute": torch.cuda.Stream(), "back": torch.cuda.Stream()}
        chain.stage_batch(st["blob"], offs)
        chain.sync()
        if case["tuned"]:
            chain.autotune()
        chain.capture_graph()
        return st
    w = _tracks(case, seed)
    dev = torch.device("cuda")
    st = {"kind": kind, "precision": case.get("precision", 0), "hits": torch.as_tensor(w["hits"]).to(dev),
          "ge": torch.as_tensor(w["ge"]).to(dev), "offsets": torch.as_tensor(w["offsets"]).to(dev)}
    if kind == "adjoint":
        if case["align"]:
            pos, align = _alignment(seed)
            st.update(module=torch.as_tensor(w["module"]).to(dev), pos=torch.as_tensor(pos).to(dev),
                      align=torch.as_tensor(align).to(dev))
    else:
        from pixeltrack.fits import workspace
        st["ws"] = workspace(case["tracks"], dev)
    return st


# ------------------------------------------------------------------------------- one pass
_HITS = ("xl", "yl", "xerr", "yerr", "xg", "yg", "zg", "iphi", "charge", "xsize", "ysize", "det_ind")


def run(state):
    kind = state["kind"]
    if kind == "event":
        chain, out = state["chain"], state["out"]
        chain.run_event(state["event"])
        chain.export_async(out)
        chain.sync()
        return out.arrays
    if kind == "hits":
        from pixeltrack import STAGE_DIGIS, STAGE_HITS
        chain = state["chain"]
        chain.run_event(state["event"], STAGE_DIGIS | STAGE_HITS)
        for k, mine in state["hits"].items():
            got = chain.product(k)
            mine[:len(got)] = got
        return state["hits"]
    if kind == "batch":
        chain, out = state["chain"], state["out"]
        s = state["compute"].cuda_stream
        chain.stage_slot(0, state["blob"], state["offs"], state["copy"].cuda_stream)
        chain.launch_slot(0, s)
        chain.export_async(out, s, state["back"].cuda_stream)
        return out.arrays
    from pixeltrack.fits import bl_fit, bl_fit_adjoint, riemann_fit
    args = state["hits"], state["ge"], state["offsets"], B_FIELD
    if kind == "bl":
        return bl_fit(*args, precision=state["precision"], ws=state["ws"])
    if kind == "rm":
        return riemann_fit(*args, precision=state["precision"], ws=state["ws"])
    if "align" in state:
        return bl_fit_adjoint(*args, state["module"], state["pos"], state["align"], True)
    return bl_fit_adjoint(*args)


def work(case):
    kind = case["kind"]
    if kind in ("event", "hits", "batch"):
        n = case.get("events", 1)
        pu = 0.5 * case["size"] if case["mode"] == "uniform" else case["size"]
        # about 19 digis per track, 30 tracks per vertex; 1e-4 noise of 123.5 M pixels
        tracks = case["size"] if case["mode"] == "single" else 30 * pu
        digis = 19 * tracks + (0 if case["mode"] == "single" else 12_350)
        if kind == "hits":
            return {"bytes": 4 * digis + 40 * digis / 3.9, "flops": 60 * digis}
        # loose tracks with covariance, state and vertex out
        return {"bytes": n * (4 * digis + 0.8 * tracks * 99), "flops": n * (60 * digis + 3000 * tracks)}
    n = case["tracks"]
    hits = n * MEAN_HITS
    into = 48 * hits + 4 * n
    # operations of one track's fit, estimated from the formulas: per hit the geometry, weights, scattering
    # and band elimination of the two systems, per track the covariance transport
    if kind == "bl":
        return {"bytes": into + (5 + 15 + 4) * 4 * n, "flops": 350 * hits + 500 * n}
    if kind == "rm":
        return {"bytes": into + (5 + 2 + 2) * 4 * n, "flops": 600 * hits + 800 * n}
    extra = 2 * hits + 1856 * (24 + 24 + 72) if case["align"] else 0
    return {"bytes": into + 12 * hits + 4 * n + extra, "flops": 700 * hits + 300 * n}


# ------------------------------------------------------------------------------- the fits in 64 bits
# Dense, batched restatements of the published algorithms (broken-line helix fit; Riemann-Chernov
# circle and line fit), one batch per hit count.
def _atan2p(y, x):
    """atan2 on the branch (-pi/2, 3 pi/2) that the reference uses."""
    a = torch.atan2(y, x)
    return torch.where(a <= -math.pi / 2, a + 2 * math.pi, a)


def _scatter(length, radius, slope):
    pt2 = torch.clamp(B_FIELD * radius, max=20.0) ** 2
    x = length.abs() * (0.06 / 16.0)
    return 0.7 * 0.0136 ** 2 / (pt2 * (1 + slope * slope)) * x * (1 + 0.038 * torch.log(x)) ** 2


def _drop_tiny(v):
    return torch.where(v.abs() < 1e-12, torch.zeros_like(v), v)


class _BrokenLine:
    """The two systems of the broken-line fit of (n, N, 3) hits with (n, N, 6) covariances, in 64 bits."""

    def __init__(self, h, ge):
        n, N = h.shape[:2]
        x, y, z = (h[:, :, k] - h[:, :1, k] for k in range(3))
        m = N // 2
        a1, a2, c1, c2 = x[:, m], y[:, m], -x[:, -1], -y[:, -1]
        half = 0.5 / (c1 * a2 - c2 * a1)
        nc, na = c1 * c1 + c2 * c2, a1 * a1 + a2 * a2
        cx, cy = -(a2 * nc + c2 * na) * half, (a1 * nc + c1 * na) * half
        R = torch.sqrt(cx * cx + cy * cy)
        turn = _atan2p(-cx * y[:, -1] + cy * x[:, -1], cx * cx + cy * cy - cx * x[:, -1] - cy * y[:, -1])
        bend = x[:, 1] * (y[:, -1] - y[:, -2]) - y[:, 1] * (x[:, -1] - x[:, -2])
        self.q = q = torch.where(bend > 0, -1.0, 1.0).to(h)
        self.slope = t = -q / (R * turn / z[:, -1])
        ux, uy = -cx[:, None], -cy[:, None]
        uu = ux * ux + uy * uy
        qR = (q * R)[:, None]
        self.s = s = -qR * _atan2p(ux * y - uy * x, uu + ux * x + uy * y)
        h0x, h0y = h[:, :1, 0], h[:, :1, 1]
        self.s0 = (qR * _atan2p(-(ux * h0y - uy * h0x), uu - (ux * h0x + uy * h0y)))[:, 0]
        self.a = a = 1 / torch.sqrt(1 + t * t)
        self.b = b = t * a
        self.S, self.Z = a[:, None] * s + b[:, None] * z, -b[:, None] * s + a[:, None] * z
        ms = _scatter(self.S[:, 1:] - self.S[:, :-1], R[:, None], t[:, None])
        self.ms0 = ms[:, 0]
        self.VB = ms[:, 1:] + ms[:, :-1]
        rx, ry = x - cx[:, None], y - cy[:, None]
        self.rn = rn = torch.sqrt(rx * rx + ry * ry)
        self.rx, self.ry, self.R = rx / rn, ry / rn, R
        self.x, self.y, self.z, self.h = x, y, z, h
        # line weights: variance across the line in the rotated (s, z) plane
        vxx, vxy, vyy, vxz, vyz, vzz = (ge[:, :, k] for k in range(6))
        vxy, vxz, vyz = _drop_tiny(vxy), _drop_tiny(vxz), _drop_tiny(vyz)
        j = (-b[:, None] * self.ry, b[:, None] * self.rx, a[:, None].expand_as(rx))
        var = j[0] * j[0] * vxx + j[1] * j[1] * vyy + j[2] * j[2] * vzz + \
            2 * (j[0] * j[1] * vxy + j[0] * j[2] * vxz + j[1] * j[2] * vyz)
        self.wl = 1 / var
        # circle weights and radial residuals
        vxx, vyy = _drop_tiny(vxx), _drop_tiny(vyy)
        self.wc = 1 / (self.rx ** 2 * vxx + 2 * self.rx * self.ry * vxy + self.ry ** 2 * vyy)
        self.Zc = (2 * (ux * x + uy * y) + x * x + y * y) / (rn + R[:, None])
        self.VBc = self.VB * (1 + t * t)[:, None]

    @staticmethod
    def kinks(s, border):
        """Rows of the kink operator: angle at each inner hit as a linear form of the corrections."""
        n, N = s.shape
        K = s.new_zeros(n, N - 2, N + int(border))
        d = s[:, 1:] - s[:, :-1]
        for i in range(1, N - 1):
            K[:, i - 1, i - 1] = 1 / d[:, i - 1]
            K[:, i - 1, i] = -(d[:, i] + d[:, i - 1]) / (d[:, i] * d[:, i - 1])
            K[:, i - 1, i + 1] = 1 / d[:, i]
            if border:
                K[:, i - 1, N] = (s[:, i + 1] - s[:, i - 1]) / 2
        return K

    def solve(self, border):
        """Solution, inverse and chi2 of the line (border False) or circle (True) system."""
        s, Z, w, VB = (self.s, self.Zc, self.wc, self.VBc) if border else (self.S, self.Z, self.wl, self.VB)
        n, N = s.shape
        with torch.no_grad():
            K = self.kinks(s, border)
            C = K.transpose(1, 2) @ (K / VB[:, :, None])
            C[:, range(N), range(N)] += w
            r = torch.zeros_like(C[:, 0])
            r[:, :N] = w * Z
            # one unit for all corrections, so that the inverse keeps its digits
            k = 1 / torch.sqrt(torch.diagonal(C, dim1=1, dim2=2))
            I = torch.linalg.inv(C * k[:, :, None] * k[:, None, :]) * k[:, :, None] * k[:, None, :]
            u = (I @ r[:, :, None])[:, :, 0]
            u = u + (I @ (r - (C @ u[:, :, None])[:, :, 0])[:, :, None])[:, :, 0]
        kink = (self.kinks(s, border) @ u[:, :, None])[:, :, 0]
        chi2 = (w * (Z - u[:, :N]) ** 2).sum(1) + (kink ** 2 / VB).sum(1)
        return u, I, chi2


def _sandwich(J, C):
    return J @ C @ J.transpose(1, 2)


def _mat(rows, like):
    one = torch.ones_like(like)
    return torch.stack([torch.stack([e if torch.is_tensor(e) else e * one for e in r], -1) for r in rows], -2)


def _move(par, cov, x0, y0):
    """Karimaki parameters and covariance moved to the point (x0, y0)."""
    phi, d, rho = par
    sn, cs = torch.sin(phi), torch.cos(phi)
    dp, do = x0 * cs + y0 * sn, x0 * sn - y0 * cs + d
    uu = 1 + rho * d
    C, BB = -rho * y0 + uu * cs, rho * x0 + uu * sn
    A = 2 * do + rho * (do * do + dp * dp)
    U = torch.sqrt(1 + rho * A)
    xi, v = 1 / (BB * BB + C * C), 1 + rho * do
    lam = 0.5 * A / (U * (1 + U) ** 2)
    mu = 1 / (U * (1 + U)) + rho * lam
    J = _mat([[xi * uu * v, -xi * rho * rho * dp, xi * dp],
              [2 * mu * uu * dp, 2 * mu * v, mu * (do * do + dp * dp) - lam * A], [0., 0., 1.]], phi)
    return (_atan2p(BB, C), A / (1 + U), rho), _sandwich(J, cov)


def _bl_group(h, ge):
    f = _BrokenLine(h, ge)
    N = h.shape[1]
    # line
    u, I, chi2l = f.solve(False)
    Sc, Zc = f.a * f.s0 + f.b * h[:, 0, 2], -f.b * f.s0 + f.a * h[:, 0, 2]
    d = f.S[:, 1] - f.S[:, 0]
    p0 = (u[:, 1] - u[:, 0]) / d
    p1 = u[:, 0] + Zc - p0 * (f.S[:, 0] + Sc)
    off = (I[:, 0, 1] - I[:, 0, 0]) / d
    cov = _mat([[(I[:, 0, 0] - 2 * I[:, 0, 1] + I[:, 1, 1]) / d ** 2 + f.ms0, off], [off, I[:, 0, 0]]], d)
    cov = _sandwich(_mat([[1., 0.], [-(f.S[:, 0] + Sc), 1.]], d), cov)
    j = 1 / (f.a - p0 * f.b)
    cov = _sandwich(_mat([[j * j, 0.], [p1 * f.b * j * j, j]], d), cov)
    line, lcov = ((f.b + p0 * f.a) * j, p1 * j), cov
    # circle
    u, I, chi2c = f.solve(True)
    I = I[:, [0, 1, N]][:, :, [0, 1, N]]
    t1, t2 = u[:, 0] - f.Zc[:, 0], u[:, 1] - f.Zc[:, 1]
    dx, dy = t1 * f.rx[:, 0], t1 * f.ry[:, 0]
    ex, ey = f.x[:, 1] + t2 * f.rx[:, 1] - dx, f.y[:, 1] + t2 * f.ry[:, 1] - dy
    c2 = ex * ex + ey * ey
    par = (_atan2p(ey, ex), -f.q * 0.25 * c2 / (f.R + torch.sqrt(f.R ** 2 - 0.25 * c2)), f.q * (1 / f.R + u[:, N]))
    fl = torch.floor(f.q / 2)
    den = torch.sqrt(4 * f.R ** 2 - c2)
    J = _mat([[(f.ry[:, 0] * ex - ey * f.rx[:, 0]) / c2, (f.ry[:, 1] * ex - ey * f.rx[:, 1]) / c2, 0.],
              [fl * (ex * f.rx[:, 0] + ey * f.ry[:, 0]) / den, fl * (ex * f.rx[:, 1] + ey * f.ry[:, 1]) / den, 0.],
              [0., 0., f.q]], d)
    par, cov = _move(par, _sandwich(J, I), 0.5 * ex, 0.5 * ey)
    cov = cov.clone()
    cov[:, 0, 0] += (1 + f.slope ** 2) * f.ms0
    (phi, tip, rho), cov = _move(par, cov, h[:, 0, 0] + dx, h[:, 0, 1] + dy)
    ib, o = 1 / B_FIELD, torch.zeros_like(d)
    return {"state": torch.stack([phi, tip, rho * ib, line[0], line[1]], 1),
            "cov": torch.stack([cov[:, 0, 0], cov[:, 0, 1], ib * cov[:, 0, 2], o, o, cov[:, 1, 1], ib * cov[:, 1, 2],
                                o, o, ib * ib * cov[:, 2, 2], o, o, lcov[:, 0, 0], lcov[:, 0, 1], lcov[:, 1, 1]], 1),
            "chi2": (chi2l + chi2c) / (2 * N - 5), "pt": B_FIELD / rho.abs(), "eta": torch.asinh(line[0])}


def _rm_group(h, ge):
    n, N = h.shape[:2]
    x, y, z = (h[:, :, k] - h[:, :1, k] for k in range(3))
    X, Y, Zg = h[:, :, 0], h[:, :, 1], h[:, :, 2]
    m = N // 2
    # circle through the first, middle and last hits
    b0, b1, c0, c1 = x[:, m], y[:, m], x[:, -1], y[:, -1]
    b2, c2 = b0 * b0 + b1 * b1, c0 * c0 + c1 * c1
    div = 2 * (b0 * c1 - b1 * c0)
    fx, fy = (c1 * b2 - b1 * c2) / div, (b0 * c2 - c0 * b2) / div
    fR = torch.sqrt(fx * fx + fy * fy)
    ftan = fR * _atan2p(fy * c0 - fx * c1, fx * fx + fy * fy - fx * c0 - fy * c1) / z[:, -1]
    rad = torch.sqrt(X * X + Y * Y)
    gx, gy = X[:, :1] + fx[:, None], Y[:, :1] + fy[:, None]
    pt = torch.clamp(fR * B_FIELD, max=20.0)
    p2 = pt * pt * (1 + 1 / ftan ** 2)
    arc = (_atan2p(gy * (X - gx) - gx * (Y - gy), -gx * (X - gx) - gy * (Y - gy)) * fR[:, None]).abs()
    grow = torch.sqrt(1 + 1 / ftan ** 2)[:, None]
    sin2 = torch.sin(torch.atan(ftan))[:, None] ** 2

    def layers(path):  # traversed radiation lengths, segment by segment
        rl = torch.cat([path[:, :1], (path[:, 1:] - path[:, :-1]).abs()], 1) * (0.06 / 16.0)
        return torch.where(rl > 0, (1 + 0.038 * torch.log(rl.clamp(min=1e-300))) ** 2 * rl, torch.zeros_like(rl))

    before = torch.tril(torch.ones(N, N, dtype=h.dtype, device=h.device))  # layers a hit has behind it
    lever = (rad[:, :, None] - rad[:, None, :]) * before
    C = (lever * (layers(arc * grow) * 0.000225 / (p2[:, None] * sin2))[:, None, :]) @ lever.transpose(1, 2)
    bx, by = X - gx, Y - gy
    tc = -(X * by - Y * bx) / (X * bx + Y * by)
    var = (ge[:, :, 0] + ge[:, :, 2] * tc * tc + 2 * ge[:, :, 1] * tc) / (1 + tc * tc)
    C[:, range(N), range(N)] += torch.where(rad < 1e-4, ge[:, :, 0], var)
    G = torch.linalg.inv(C)
    G = 0.5 * (G + G.transpose(1, 2))
    norm = G.sum((1, 2))
    wgt = G.sum(1) / norm[:, None]
    mx, my = x.mean(1, keepdim=True), y.mean(1, keepdim=True)
    s = torch.sqrt(N / ((x - mx) ** 2 + (y - my) ** 2).sum(1))
    p = torch.stack([(x - mx) * s[:, None], (y - my) * s[:, None]], 1)
    p = torch.cat([p, (p * p).sum(1, keepdim=True)], 1)
    r0 = (p * wgt[:, None, :]).sum(2)
    P = p - r0[:, :, None]
    A = (P @ G @ P.transpose(1, 2)) / norm[:, None, None]
    lam, vec = (r.to(h) for r in torch.linalg.eigh((0.5 * (A + A.transpose(1, 2))).cpu()))
    v, lam = vec[:, :, 0], lam[:, 0]
    v = v * torch.where(v[:, 2:] > 0, 1.0, -1.0).to(h)
    c = -(v * r0).sum(1)
    uvr2 = torch.sqrt(1 - v[:, 2] ** 2 - 4 * c * v[:, 2]) / (2 * v[:, 2])
    cx, cy = -v[:, 0] / (2 * v[:, 2]) / s + mx[:, 0], -v[:, 1] / (2 * v[:, 2]) / s + my[:, 0]
    R = uvr2 / s
    q = torch.where(x[:, 1] * cy - y[:, 1] * cx > 0, -1.0, 1.0).to(h)
    chi2c = lam.abs() * norm / (2 * v[:, 2] * uvr2 * s) ** 2
    # line in the (s, z) plane, rotated by the fast-fit angle
    th = -q * torch.atan(ftan)
    th = torch.where(th < 0, th + math.pi, th)
    sn, cs = torch.sin(th)[:, None], torch.cos(th)[:, None]
    gx, gy = X[:, :1] + cx[:, None], Y[:, :1] + cy[:, None]
    qx, qy = X - gx, Y - gy
    cr, dt = gy * qx - gx * qy, -gx * qx - gy * qy
    qR = (q * R)[:, None]
    sa = -qR * _atan2p(cr, dt)
    k = -qR / (dt * dt + cr * cr)
    dx, dy = k * (gy * dt + gx * cr), k * (-gx * dt + gy * cr)
    t00 = dx * (ge[:, :, 0] * dx + ge[:, :, 1] * dy) + dy * (ge[:, :, 1] * dx + ge[:, :, 2] * dy)
    t01 = dx * ge[:, :, 3] + dy * ge[:, :, 4]
    S3 = torch.sqrt(sa * sa + Zg * Zg)
    path = (S3[:, :, None] - S3[:, None, :]).abs() * before
    Cz = (path * (layers(S3) * 0.000225 / p2[:, None])[:, None, :]) @ path.transpose(1, 2)
    Cz[:, range(N), range(N)] += cs * cs * t00 - 2 * cs * sn * t01 + sn * sn * ge[:, :, 5]
    V = torch.linalg.inv(Cz)
    xr, yr = sn * sa + cs * Zg, -cs * sa + sn * Zg
    w, wx = V.sum(2), (V @ xr[:, :, None])[:, :, 0]
    M00, M01, M11 = w.sum(1), wx.sum(1), (xr * wx).sum(1)
    r0l, r1l = (w * yr).sum(1), (wx * yr).sum(1)
    det = M00 * M11 - M01 * M01
    s0, s1 = (M11 * r0l - M01 * r1l) / det, (M00 * r1l - M01 * r0l) / det
    cf = 1 / (sn[:, 0] - s1 * cs[:, 0])
    res = yr - s0[:, None] - s1[:, None] * xr
    pT = R * B_FIELD
    state = torch.stack([torch.atan2(q * gx[:, 0], -q * gy[:, 0]), q * (torch.hypot(gx, gy)[:, 0] - R), q / pT,
                         cf * (s1 * sn[:, 0] + cs[:, 0]), cf * s0], 1)
    return {"state": state, "chi2": torch.stack([chi2c, (res * (V @ res[:, :, None])[:, :, 0]).sum(1)], 1), "pt": pT}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("event", "hits", "batch"):  # decisions, list orders and 32-bit arithmetic that the outputs hang on
        return None
    w = _tracks(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    hits, ge = torch.as_tensor(w["hits"]).to(dev), torch.as_tensor(w["ge"]).to(dev).double()
    offs = torch.as_tensor(w["offsets"]).to(dev).long()
    n = case["tracks"]
    moved = hits
    if kind == "adjoint" and case["align"]:
        pos, align = (torch.as_tensor(a).to(dev).double() for a in _alignment(seed))
        mod = torch.as_tensor(w["module"]).to(dev).long()
        on = mod >= 0
        arm = hits[on] - pos[mod[on]]
        moved = hits.clone()
        moved[on] += align[mod[on], :3] + torch.linalg.cross(align[mod[on], 3:], arm)
    out = None
    count = offs[1:] - offs[:-1]
    for N in range(3, 9):
        t = torch.nonzero(count == N)[:, 0]
        for t in torch.split(t, 1 << 17):
            if not len(t):
                continue
            at = offs[t][:, None] + torch.arange(N, device=dev)
            if kind == "adjoint":
                h = moved[at].requires_grad_(True)
                f = _BrokenLine(h, ge[at])
                chi2 = f.solve(False)[2] + f.solve(True)[2]
                got = {"chi2": chi2.detach(), "grad_hits": torch.autograd.grad(chi2.sum(), h)[0]}
            else:
                got = (_bl_group if kind == "bl" else _rm_group)(moved[at], ge[at])
            if out is None:
                out = {k: torch.zeros((len(hits) if k == "grad_hits" else n,) + v.shape[(2 if k == "grad_hits" else 1):],
                                      dtype=torch.float64, device=dev) for k, v in got.items()}
            for k, v in got.items():
                out[k][at if k == "grad_hits" else t] = v
    if kind != "adjoint":
        out["status"] = None
    elif case["align"]:
        g = out["grad_hits"][on]
        acc = torch.zeros_like(align)
        acc.index_add_(0, mod[on], torch.cat([g, torch.linalg.cross(arm, g)], 1))
        out["grad_align"], out["grad_align64"] = acc, acc
    return out
