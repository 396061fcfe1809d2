"""The framework's performance cases: analyses a BsaLib user runs, through the public binding.

A pass is the whole call sequence of the reference's driver on host arrays (bsa_Init, the
setters, the evaluation, bsa_Finalise), as app/bsa.F90:72-117 makes it once per structure and
wind case; inputs are seeded structures of the sizes of this repository's configurations, tests
and benchmark.  FP64 is the library's default precision, the split precision (BF16 triples on
the tensor cores) is asked for by the session's argument.

`exact` restates the mathematics in 64-bit torch: nodal spectra, A(f) = S(f) L, the products
E(x, y)[a, b, j] = sum_k Q_ka A(x)_kb A(y)_kj, the FRF product and the integration weights.
"""
import dataclasses
import math
import weakref

import numpy as np
import torch

from bsalib_gb300 import api
from bsalib_gb300.problem import bridge_deck, cantilever_tower, random_structure, tall_building

TWO_PI = 2.0 * math.pi


def listed():
    return [
        # The 30-node cantilever tower of the reference's kind of example: the smallest analysis a
        # user runs, where set-up and launches count.  Default precision, and split.
        {"name": "tower_fp64", "kind": "classic", "model": "tower", "nodes": 30, "modes": 4, "nf": 129, "split": False},
        {"name": "tower_split", "kind": "classic", "model": "tower", "nodes": 30, "modes": 4, "nf": 129, "split": True},
        # A mast of odd sizes on a medium grid, one wind component, default precision.
        {"name": "cantilever_fp64", "kind": "classic", "model": "cantilever", "nodes": 173, "modes": 11, "nf": 193,
         "split": False},
        # The 400-node, 24-mode building with two wind components: default precision on the coarse
        # grid of a first look, split precision on the full 1025 x 1025 grid (the benchmark's step).
        {"name": "building_fp64", "kind": "classic", "model": "building", "nodes": 400, "modes": 24, "nf": 129,
         "split": False},
        {"name": "building_split", "kind": "classic", "model": "building", "nodes": 400, "modes": 24, "nf": 1025,
         "split": True},
        # Same-mode spectra only (the reference's onlyd setting): a design check on a fine grid.
        {"name": "building_diag", "kind": "classic", "model": "building", "nodes": 400, "modes": 24, "nf": 513,
         "split": False, "diag": True},
        # Force and response bispectra at every grid point, brought to the host for plots.
        {"name": "bispectra_fp64", "kind": "bispectra", "model": "cantilever", "nodes": 60, "modes": 6, "nf": 65},
        # Bispectra at a list of frequency pairs (the Mesher's plugin functions, batched).
        {"name": "points_fp64", "kind": "points", "model": "cantilever", "nodes": 150, "modes": 12, "points": 1111},
        # Third moments over the caller's own zones, default precision.
        {"name": "zones_fp64", "kind": "zones", "model": "building", "nodes": 200, "modes": 16, "cells": 8,
         "split": False},
        # The Mesher analysis of the long-span bridge deck (1200 nodes, 60 modes), split precision:
        # layout and zone integration in one bsa_Run, with the driver's controls.
        {"name": "bridge_mesher_split", "kind": "mesher", "nodes": 1200, "modes": 60},
        # A parametric study: structures of uneven size under several wind speeds in one batch.
        {"name": "sweep_split", "kind": "sweep", "structures": 8, "winds": 2, "nodes": 300, "modes": 24, "nf": 257},
        # The zone-refinement proposer: one gradient over a batch of records, refinement probabilities of many zones.
        {"name": "proposer", "kind": "proposer", "records": 4096, "zones": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    cap = {k: work(c)["flops"] for k, c in ((c["name"], c) for c in listed())}
    while True:
        kind = rng.choice(["classic", "classic", "classic", "bispectra", "points", "zones", "mesher", "sweep", "proposer"])
        model = rng.choice(["cantilever", "building"])
        if kind == "classic":
            split = rng.random() < 0.4
            c = {"kind": kind, "model": model, "nodes": _log(rng, 20, 400), "modes": rng.randint(3, 24),
                 "nf": 2 * _log(rng, 24, 512 if split else 128) + 1, "split": split}
            if not split and rng.random() < 0.2:
                c["diag"] = True
            elif not split and rng.random() < 0.3:
                c["analytic"] = True
            limit = cap["building_split"] if split else cap["building_diag"] if c.get("diag") else cap["building_fp64"]
        elif kind == "bispectra":
            c = {"kind": kind, "model": model, "nodes": _log(rng, 20, 120), "modes": rng.randint(2, 8),
                 "nf": 2 * rng.randint(16, 48) + 1}
            limit = 4 * cap["bispectra_fp64"]
        elif kind == "points":
            c = {"kind": kind, "model": model, "nodes": _log(rng, 20, 200), "modes": rng.randint(3, 16),
                 "points": _log(rng, 50, 2000)}
            limit = 4 * cap["points_fp64"]
        elif kind == "zones":
            c = {"kind": kind, "model": model, "nodes": _log(rng, 30, 300), "modes": rng.randint(3, 20),
                 "cells": rng.randint(3, 10), "split": rng.random() < 0.4}
            limit = 4 * cap["zones_fp64"]
        elif kind == "mesher":
            c = {"kind": kind, "nodes": _log(rng, 100, 1200), "modes": rng.randint(6, 60)}
            limit = cap["bridge_mesher_split"]
        elif kind == "sweep":
            c = {"kind": kind, "structures": rng.randint(2, 8), "winds": rng.randint(1, 4), "nodes": _log(rng, 60, 400),
                 "modes": rng.randint(6, 24), "nf": 2 * rng.randint(70, 160) + 1}
            limit = 2 * cap["sweep_split"]
        else:
            c = {"kind": kind, "records": _log(rng, 200, 6000), "zones": _log(rng, 300, 30000)}
            limit = 2 * cap["proposer"]
        if work(c)["flops"] <= limit:
            return c


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------

def _structure(case, seed, rng):
    """The case's structure under a seeded wind case: mean speeds, turbulence, force
    coefficients and damping vary around the model's."""
    model, nodes, modes = case["model"], case["nodes"], case["modes"]
    nf = case.get("nf", 65)
    h = (nf - 1) // 2
    if model == "tower":
        p = cantilever_tower(nfreqs=h + 1, df=2.0 / h, nodes=nodes)
    elif model == "building":
        p = tall_building(nodes=nodes, modes=modes, nfreqs=h + 1, df=4.0 / h, seed=seed)
    else:
        p = random_structure(seed, nodes=(nodes, nodes), modes=(modes, modes), nfreq_grid=(nf, nf))
    return _wind_case(p, rng)


def _wind_case(p, rng):
    xsi = p.xsi * rng.uniform(0.8, 1.25)
    return dataclasses.replace(
        p, u_node=p.u_node * rng.uniform(0.9, 1.1), sigma=p.sigma * rng.uniform(0.85, 1.15),
        wfc=np.asfortranarray(p.wfc * rng.uniform(0.8, 1.2)), xsi=xsi,
        Cg=np.asfortranarray(np.diag(2.0 * xsi * TWO_PI * p.natf)))


def _zones(p, cells, rng):
    """Rectangular zones tiling the half plane f1 >= 0 up to 1.25 times the largest natural
    frequency: lattices of 2-5 points per side, the BRM lattice finer where the zone holds a
    resonance ridge."""
    F = 1.25 * float(p.natf.max())
    h = F / cells
    out = []
    for i in range(cells):
        for j in range(2 * cells):
            x, y = i * h, -F + j * h
            ni, nj = int(rng.integers(2, 6)), int(rng.integers(2, 6))
            ridge = any(lo <= s * f <= hi for lo, hi in ((x, x + h), (y, y + h), (x + y, x + y + 2 * h))
                        for f in p.natf for s in (1.0, -1.0))
            fi, fj = (int(rng.integers(2, 5)), int(rng.integers(2, 5))) if ridge else (1, int(rng.integers(1, 3)))
            out.append(api.Zone(x, y, h / (ni - 1), 0.0, 0.0, h / (nj - 1), ni, nj, fi, fj, 2.0, 0))
    return out


def _sweep_sizes(case):
    """(nodes, modes, grid) of the sweep's structures, uneven up to the case's largest."""
    r = np.random.default_rng(case["structures"])
    return [(int(r.integers(max(20, case["nodes"] // 10), case["nodes"] + 1)), int(r.integers(4, case["modes"] + 1)),
             2 * int(r.integers(64, case["nf"] // 2 + 1)) + 1) for _ in range(case["structures"])]


class _State(dict):
    pass


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = _State(case=case)
    kind = case["kind"]
    if kind == "proposer":
        net = api.Mlp(13, 128, seed + 1)
        weakref.finalize(st, net.close)  # the library holds few networks at a time
        n, z = case["records"], case["zones"]
        x = rng.standard_normal((n + z, 13)).astype(np.float32)
        y = (1.0 / (1.0 + np.exp(-2.0 * x[:n, 0] - x[:n, 5]))).astype(np.float32)
        w = np.where(rng.random(n) < 0.1, 20.0, 1.0).astype(np.float32)
        st.update(net=net, x=x[:n].copy(), y=y, w=w, z=x[n:].copy())
    elif kind == "sweep":
        us = np.linspace(15.0, 50.0, case["winds"]) if case["winds"] > 1 else np.array([30.0])
        st["probs"] = [_wind_case(random_structure(seed * 64 + c, nodes=(nodes, nodes), modes=(modes, modes),
                                                   nfreq_grid=(nf, nf), U_mean=float(u)), rng)
                       for c, (nodes, modes, nf) in enumerate(_sweep_sizes(case)) for u in us]
    elif kind == "mesher":
        st["prob"] = _wind_case(bridge_deck(nodes=case["nodes"], modes=case["modes"], seed=77 + seed), rng)
    else:
        p = _structure(case, seed, rng)
        if case.get("diag"):
            p.settings.onlyd = 1
        st["prob"] = p
        if kind == "points":
            F = 1.25 * float(p.natf.max())
            st["f1"] = rng.uniform(-F, F, case["points"])
            st["f2"] = rng.uniform(-F, F, case["points"])
        elif kind == "zones":
            st["zones"] = _zones(p, case["cells"], rng)
    return st


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------

def _session(st):
    case = st["case"]
    split = case.get("split", case["kind"] == "mesher")
    return api.BsaSession(st["prob"], precision=api.PREC_BF16X3 if split else api.PREC_FP64,
                          classic_truncation=not case.get("analytic", False))


def run(st):
    kind = st["case"]["kind"]
    if kind == "proposer":
        loss, grad = st["net"].gradients(st["x"], st["y"], st["w"])
        return {"loss": np.float32(loss), "grad": grad, "prob": st["net"].forward(st["z"])}
    if kind == "sweep":
        sw = api.Sweep()
        for p in st["probs"]:
            sw.add(p)
        res, _ = sw.run()
        sw.clear()
        return {k: np.concatenate([r[k] for r in res]) for k in ("m3mf", "m3mr", "m2mr")}
    s = _session(st)
    try:
        if kind == "classic":
            out = s.run()
            return {k: out[k] for k in ("m2mf_cls", "m2mr_cls", "m2o2mr_cls", "m3mf_cls", "m3mr_cls")}
        if kind == "mesher":
            s.use_driver_controls()
            out = s.run()
            return {k: out[k] for k in ("m3mf_msh", "m3mr_msh")}
        if kind == "bispectra":
            f, bf, br = s.classic_bispectra()
            return {"f": f, "bf": bf, "br": br}
        if kind == "points":
            bf, br = s.msh_bispectra(st["f1"], st["f2"])
            return {"bf": bf, "br": br}
        mf, mr, cnt = s.msh_zones(st["zones"])
        return {"m3mf": mf, "m3mr": mr, "points": cnt}
    finally:
        s.close()


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------

def _classic_work(nodes, modes, nf, ntc, diag=False, analytic=False):
    k, n3, half = ntc * nodes, modes ** 3, (nf + 1) // 2
    rows = 2 * half if analytic else half  # distinct |f|: every quantity is even in f
    if diag:
        return {"bytes": 8.0 * (5 * modes + 4 * k + 2 * k * modes), "flops": half * nf * (2.0 * k * modes + 20.0 * modes)}
    pairs = half * (half + 1) / 2 + (half * half if analytic else 0)
    return {"bytes": 8.0 * (ntc * nodes * (nodes + 1) / 2 + 2 * k * modes + 3 * modes ** 2 + 2 * n3),
            "flops": rows * ntc * 2.0 * nodes ** 2 * modes + pairs * 2.0 * k * n3 + half * nf * 6.0 * n3}


def _point_work(nodes, modes, ntc, pts, out):
    k, n3 = ntc * nodes, modes ** 3
    return {"bytes": 8.0 * (ntc * nodes * (nodes + 1) / 2 + 2 * k * modes + out),
            "flops": pts * (3.0 * ntc * 2 * nodes ** 2 * modes + 4.0 * k * n3 + 6.0 * n3)}


def work(case):
    kind = case["kind"]
    ntc = 2 if case.get("model") == "building" or kind == "mesher" else 1
    if kind == "classic":
        return _classic_work(case["nodes"], case["modes"], case["nf"], ntc, case.get("diag"), case.get("analytic"))
    if kind == "bispectra":
        w = _classic_work(case["nodes"], case["modes"], case["nf"], ntc)
        w["bytes"] += 16.0 * case["nf"] ** 2 * case["modes"] ** 3
        return w
    if kind == "points":
        return _point_work(case["nodes"], case["modes"], ntc, case["points"], 2 * case["points"] * case["modes"] ** 3)
    if kind == "zones":
        pts = 2 * case["cells"] ** 2 * 12.25  # 3.5 x 3.5 lattice points a zone on average
        return _point_work(case["nodes"], case["modes"], ntc, pts, 2 * case["modes"] ** 3)
    if kind == "mesher":
        pts = 11917.0 * case["modes"] / 60  # the layout's lattice points grow with the modes
        n, m = case["nodes"], case["modes"]
        # lattice frequencies are shared along the zones' lines: about a third of the points'
        return {"bytes": 8.0 * (2 * n * (n + 1) / 2 + 4 * n * m + 2 * m ** 3),
                "flops": pts * (2.0 * 2 * n ** 2 * m / 3 + 12.0 * n * m ** 3) + 8.0 * pts * 6.0 * m ** 3}
    if kind == "sweep":
        each = [_classic_work(nodes, modes, nf, 1) for nodes, modes, nf in _sweep_sizes(case)]
        return {k: case["winds"] * sum(w[k] for w in each) for k in ("bytes", "flops")}
    p = 128 * 13 + 2 * 128 * 128 + 4 * 128 + 1
    n, z = case["records"], case["zones"]
    return {"bytes": 4.0 * ((n + z) * 13 + 2 * n + z + p) + 2.0 * p, "flops": 2.0 * p * (3 * n + z)}


# ---------------------------------------------------------------------------------------------
# The same in 64-bit torch
# ---------------------------------------------------------------------------------------------

class _Model:
    """Nodal tables of a structure as 64-bit tensors: q, l [K, nm], log-coherence, FRF parameters."""

    def __init__(self, p, dev):
        self.p, self.dev = p, dev
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        nn = p.nn
        self.nm = int(p.nm)
        self.tc = list(p.settings.tc)
        phi = t(p.phi)
        lin = [t(p.wfc[0, c - 1, :])[:, None] * phi for c in self.tc]
        quad = [t(p.wfc[0, c + 2, :])[:, None] * phi for c in self.tc]
        self.l, self.q = torch.cat(lin), torch.cat(quad)
        iu = torch.triu_indices(nn, nn)
        self.coh = []
        for c in self.tc:
            m = torch.zeros(nn, nn, dtype=torch.float64, device=dev)
            v = torch.log(t(p.nod_corr[:, c - 1]))
            m[iu[0], iu[1]] = v
            m[iu[1], iu[0]] = v
            self.coh.append(m)
        self.M, self.K, self.C = t(p.Mg), t(p.Kg), t(np.diag(p.Cg))
        self.U = t(p.u_node)
        self.wz = torch.as_tensor(p.wz_node - 1, dtype=torch.long, device=dev)
        self.sig = [t(p.sigma[c - 1])[self.wz] for c in self.tc]
        self.len = [t(p.L[c - 1, 0])[self.wz] for c in self.tc]

    def psd(self, f):
        """S[f, component, node] of the von Karman (1) and Davenport (5) models."""
        out = []
        f = f[:, None]
        for c, sig, ls in zip(self.tc, self.sig, self.len):
            r = ls / self.U
            if self.p.psd_type == 1 and c == 1:
                s = 4.0 * r * sig ** 2 / (1.0 + 70.7 * (f * r) ** 2) ** (5.0 / 6.0)
            elif self.p.psd_type == 1:
                d = 4.0 * (f * r) ** 2
                s = 4.0 * r * sig ** 2 * (1.0 + 188.4 * d) / (1.0 + 70.7 * d) ** (11.0 / 6.0)
            else:
                x = f.abs() * r
                s = (2.0 / 3.0) * x * r * sig ** 2 / (1.0 + x * x) ** (4.0 / 3.0)
            out.append(s / (4.0 * math.pi if self.p.settings.defsc == 1 else 1.0))
        return torch.stack(out, 1)

    def atable(self, f):
        """A[f, k, m] = sqrt(S_i) sum_j c_ij^|f| sqrt(S_j) L_jm."""
        s = self.psd(f).sqrt()
        n = self.p.nn
        out = torch.empty(len(f), self.l.shape[0], self.nm, dtype=torch.float64, device=self.dev)
        for x in range(len(f)):
            for c, lc in enumerate(self.coh):
                g = torch.exp(f[x].abs() * lc)
                out[x, c * n:(c + 1) * n] = s[x, c][:, None] * (g @ (s[x, c][:, None] * self.l[c * n:(c + 1) * n]))
        return out

    def frf(self, f):
        w = TWO_PI * f[:, None]
        return 1.0 / torch.complex(self.K - w * w * self.M, w * self.C)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _classic_exact(p, diag, analytic, dev):
    m = _Model(p, dev)
    nm, df = m.nm, float(p.settings.df)
    N = p.settings.nfreqs - 1
    nf = 2 * N + 1
    idx = torch.arange(-N, N + 1, device=dev)
    f = idx.double() * df
    delta = TWO_PI * df
    H, HS = m.frf(f), m.frf(torch.arange(-2 * N, 2 * N + 1, device=dev).double() * df)
    wf = torch.full((nf,), delta, dtype=torch.float64, device=dev)
    wf[0] = wf[-1] = delta / 2
    edge = torch.ones(nf, dtype=torch.float64, device=dev)
    edge[0] = edge[-1] = 0.5
    hi = 2 * N if analytic else N
    rows = torch.arange(0, hi + 1, device=dev).double() * df

    def wline(i):  # weights along the line of grid index i: edges half, the vertices -1/2
        w = delta * delta * edge * edge[i]
        if i in (0, nf - 1):
            w[0], w[-1] = -0.5 * delta * delta, -0.5 * delta * delta
        return w

    if diag:
        S = m.psd(rows).reshape(hi + 1, -1)
        W3, W2 = m.q * m.l ** 2, m.l ** 2
        psd = (S @ W2)[idx.abs()]
        h2 = (H.conj() * H).real
        out = [(wf[:, None] * psd).sum(0), (wf[:, None] * psd * h2).sum(0),
               (wf[:, None] * psd * h2 * (TWO_PI * f[:, None]) ** 2).sum(0)]
        mf = torch.zeros(nm, dtype=torch.float64, device=dev)
        mr = torch.zeros_like(mf)
        for i in range(nf):
            s = idx + idx[i]
            s12 = torch.where((s.abs() <= hi)[:, None], S[s.abs().clamp(max=hi)], 0.0)
            s1, s2 = S[idx[i].abs()], S[idx.abs()]
            b = 2.0 * (s1 * s2 + s12 * s2 + s1 * s12) @ W3
            g = (H[i] * H * HS[s + 2 * N].conj()).real
            w = wline(i)[:, None]
            mf += (w * b).sum(0)
            mr += (w * b * g).sum(0)
        return out + [mf, mr]
    A = m.atable(rows)
    psd = torch.einsum("ko,fkn->fon", m.l, A)[idx.abs()]
    h2 = (H[:, :, None] * H[:, None, :].conj()).real  # [f, o, n]
    w1 = wf[:, None, None]
    out = [(w1 * psd).sum(0).reshape(-1), (w1 * psd * h2).sum(0).reshape(-1),
           (w1 * psd * h2 * (TWO_PI * f[:, None, None]) ** 2).sum(0).reshape(-1)]
    mf = torch.zeros(nm, nm, nm, dtype=torch.float64, device=dev)
    mr = torch.zeros_like(mf)
    flat = A.permute(1, 0, 2).reshape(A.shape[1], -1)  # [K, rows nm]
    for i in range(N + 1):  # the grid is centrally symmetric: lines -N .. 0, the others by their mirrors
        r = abs(int(idx[i]))
        s = idx + idx[i]
        ok = (s.abs() <= hi).double()
        z = s.abs().clamp(max=hi)
        w = wline(i) * (1.0 if i == N else 2.0) * 2.0
        U = (m.q[:, :, None] * A[r][:, None, :]).reshape(A.shape[1], -1)
        E = (U.T @ flat).reshape(nm, nm, hi + 1, nm).permute(2, 0, 1, 3)  # [row, a, b, j]
        Hs = HS[s + 2 * N].conj()
        # T1 at (i, c): m n o = a b j;  H_a(i) H_b(c) conj H_j(i + c)
        e = E[idx.abs()]
        mf += torch.einsum("c,cabj->abj", w.clone(), e)
        g = w[:, None, None] * H[:, :, None] * Hs[:, None, :]
        v = torch.complex((e * g.real[:, None]).sum(0), (e * g.imag[:, None]).sum(0))
        mr += (H[i][:, None, None] * v).real
        e = E[z]
        wz = w * ok
        # T3 at (i, c): o n m = a b j;  H_j(i) of n = b, H_o = conj H_a(i + c), H_m -- m = j is f1's factor
        t = torch.einsum("c,cabj->abj", wz, e)
        mf += t.permute(2, 1, 0)
        g = wz[:, None, None] * Hs[:, :, None] * H[:, None, :]  # conj H_a(s) H_b(c)
        v = torch.complex((e * g.real[..., None]).sum(0), (e * g.imag[..., None]).sum(0))
        mr += (v * H[i][None, None, :]).real.permute(2, 1, 0)
        # T2 at (c, i): n o m = a b j;  H_j(c) H_a(i) conj H_b(s)
        mf += t.permute(2, 0, 1)
        g = wz[:, None, None] * Hs[:, :, None] * H[:, None, :]  # conj H_b(s) H_j(c)
        v = torch.complex((e * g.real[:, None]).sum(0), (e * g.imag[:, None]).sum(0))
        mr += (v * H[i][:, None, None]).real.permute(2, 0, 1)
    order = lambda x: x.permute(2, 1, 0).reshape(-1)  # m fastest
    return out + [order(mf), order(mr)]


def _bispectra(m, f1, f2, limit=None):
    """Force bispectra [p, o, n, m] at frequency pairs; S(f1 + f2) reads zero beyond `limit`."""
    nm, K = m.nm, m.l.shape[0]
    fr = torch.stack([f1, f2, f1 + f2]).abs()
    uniq, inv = torch.unique(fr, return_inverse=True)
    A = m.atable(uniq)
    B = torch.empty(len(f1), nm, nm, nm, dtype=torch.float64, device=m.dev)
    step = max(1, int(2e7 / (K * nm * nm)))
    for p in range(0, len(f1), step):
        X, Y, Z = (A[inv[c, p:p + step]] for c in range(3))
        if limit is not None:
            Z = Z * (fr[2, p:p + step] <= limit)[:, None, None]
        xy = (Y[:, :, :, None] * X[:, :, None, :]).reshape(len(X), K, -1)       # [k, (o, n)]
        qq = (Y[:, :, :, None] * m.q[:, None, :] + m.q[:, :, None] * X[:, :, None, :]).reshape(len(X), K, -1)
        b = xy.transpose(1, 2) @ m.q + qq.transpose(1, 2) @ Z
        B[p:p + step] = 2.0 * b.reshape(-1, nm, nm, nm)
    return B


def _frf3(m, f1, f2):
    """Re[H_m(f1) H_n(f2) conj H_o(f1 + f2)] as [p, o, n, m]."""
    h1, h2, h3 = m.frf(f1), m.frf(f2), m.frf(f1 + f2).conj()
    return (h3[:, :, None, None] * h2[:, None, :, None] * h1[:, None, None, :]).real


def exact(case, seed):
    kind = case["kind"]
    if kind == "mesher":
        return None  # every lattice point of the layout in 64 bits takes minutes
    dev = _device()
    st = prepare(case, seed)
    host = lambda t: t.cpu().numpy()
    if kind == "proposer":
        v = torch.as_tensor(st["net"].params(bf16=True), dtype=torch.float64, device=dev).requires_grad_()
        parts = torch.split(v, [128 * 13, 128, 128 * 128, 128, 128 * 128, 128, 128, 1])

        def net(x):
            a = torch.as_tensor(x, dtype=torch.float64, device=dev)
            for k in (0, 2, 4):
                a = torch.relu(a @ parts[k].reshape(128, -1).T + parts[k + 1])
            return a @ parts[6] + parts[7]

        y, w = (torch.as_tensor(st[k], dtype=torch.float64, device=dev) for k in ("y", "w"))
        z = net(st["x"])
        loss = (w * (torch.nn.functional.softplus(z) - y * z)).sum() / w.sum()
        grad, = torch.autograd.grad(loss, v)
        with torch.no_grad():
            return {"loss": float(loss), "grad": host(grad), "prob": host(torch.sigmoid(net(st["z"])))}
    if kind == "sweep":
        outs = [_classic_exact(p, False, False, dev) for p in st["probs"]]
        return {k: np.concatenate([host(o[i]) for o in outs]) for k, i in (("m3mf", 3), ("m3mr", 4), ("m2mr", 1))}
    p = st["prob"]
    if kind == "classic":
        outs = _classic_exact(p, case.get("diag"), case.get("analytic"), dev)
        return {k: host(o) for k, o in zip(("m2mf_cls", "m2mr_cls", "m2o2mr_cls", "m3mf_cls", "m3mr_cls"), outs)}
    m = _Model(p, dev)
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
    if kind == "bispectra":
        N = p.settings.nfreqs - 1
        f = torch.arange(-N, N + 1, device=dev).double() * float(p.settings.df)
        f1, f2 = f.repeat_interleave(len(f)), f.repeat(len(f))
        B = _bispectra(m, f1, f2, limit=float(p.settings.df) * (N + 0.5))
        n = len(f)
        return {"f": host(f), "bf": host(B.reshape(n, n, -1)), "br": host((B * _frf3(m, f1, f2)).reshape(n, n, -1))}
    if kind == "points":
        f1, f2 = t(st["f1"]), t(st["f2"])
        B = _bispectra(m, f1, f2)
        n = len(f1)
        return {"bf": host(B.reshape(n, -1)), "br": host((B * _frf3(m, f1, f2)).reshape(n, -1))}
    mf = mr = 0.0
    nb = nq = 0
    ax = lambda n: torch.arange(n, device=dev).double()
    ends = lambda n: torch.tensor([0.5] + [1.0] * (n - 2) + [0.5], dtype=torch.float64, device=dev)
    lat, f1s, f2s = [], [], []
    for z in st["zones"]:
        i, j = ax(z.ni).repeat_interleave(z.nj), ax(z.nj).repeat(z.ni)
        lat.append(len(i))
        f1s.append(z.fi0 + i * z.dIi + j * z.dJi)
        f2s.append(z.fj0 + i * z.dIj + j * z.dJj)
    Ball = torch.split(_bispectra(m, torch.cat(f1s), torch.cat(f2s)), lat)
    for z, B in zip(st["zones"], Ball):
        B = B.reshape(z.ni, z.nj, -1)
        dA = z.sym * math.hypot(z.dIi, z.dIj) * math.hypot(z.dJi, z.dJj) * TWO_PI ** 2
        mf = mf + dA * torch.einsum("i,j,ijx->x", ends(z.ni), ends(z.nj), B)
        NI, NJ = (z.ni - 1) * z.Fi + 1, (z.nj - 1) * z.Fj + 1
        # bilinear interpolation from lattice to fine lattice along each side
        hat = lambda n, F: torch.clamp(1.0 - (ax((n - 1) * F + 1)[:, None] / F - ax(n)[None, :]).abs(), min=0.0)
        Bq = torch.einsum("pi,qj,ijx->pqx", hat(z.ni, z.Fi), hat(z.nj, z.Fj), B)
        a, b = ax(NI).repeat_interleave(NJ) / z.Fi, ax(NJ).repeat(NI) / z.Fj
        G = _frf3(m, z.fi0 + a * z.dIi + b * z.dJi, z.fj0 + a * z.dIj + b * z.dJj).reshape(NI, NJ, -1)
        mr = mr + dA / (z.Fi * z.Fj) * torch.einsum("p,q,pqx->x", ends(NI), ends(NJ), Bq * G)
        nb, nq = nb + z.ni * z.nj, nq + NI * NJ
    return {"m3mf": host(mf), "m3mr": host(mr), "points": np.array([nb, nq], dtype=np.float64)}
