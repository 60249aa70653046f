"""The work that programs have this library do: single-point force evaluations, MD runs and
the allocation-free kinetic stress, through the public entry points, over the sizes, forms and
ensembles that the repository's workloads use.

A program keeps one configuration in the library (gb_init) and hands it positions and
velocities in pinned host arrays; `run` is one whole call sequence on such arrays: upload,
start-up (wrap, halo, Verlet list, forces), the MD steps if any, download.  The learned
multiple-time-step form is left out: it is slower than the plain mixed form on every workload
of the repository, so that nobody would choose it for speed.

A case: kind ("forces", "md" or "kinstress"), system ("nacl", "water", "eam"), n_side (lattice
sites, molecules or unit cells per edge), form ("fp64", "mixed", "native"), steps, ensemble.
The mixed form computes in single precision, and its results are kept in single precision, as
a trajectory frame is; the FP64 forms return float64.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dl-poly_gb300"))
import dlpoly_gb300 as gb  # noqa: E402
from dlpoly_gb300 import systems  # noqa: E402

FORMS = {"fp64": 0, "mixed": 1, "native": 2}
# bath temperature [K] and thermostat parameters (relaxation time [ps], Langevin friction [1/ps])
TEMP = {"nacl": 1500.0, "water": 300.0, "eam": 600.0}
TAU, CHI = 0.1, 5.0
SCALARS = ("engcpe_rc", "vircpe_rc", "engcpe_rl", "vircpe_rl", "engcpe_ex", "vircpe_ex", "engvdw", "virvdw",
           "engke", "vircon", "consv", "engmet", "virmet")


def listed():
    def c(name, kind, system="nacl", n_side=0, form="fp64", steps=0, ensemble="nve"):
        return {"name": name, "kind": kind, "system": system, "n_side": n_side, "form": form, "steps": steps,
                "ensemble": ensemble}

    return [
        # the kinetic stress of a host program whose device memory is not the library's to allocate
        {"name": "kinstress_98304", "kind": "kinstress", "n": 98304, "frozen": True},
        # the smallest single point: a geometry check of a small box, every launch counts
        c("forces_water_1536", "forces", "water", 8),
        # the small melt of the benchmark, production MD: launch and latency bound
        c("md_nacl_4096", "md", "nacl", 16, steps=50),
        # equilibration of a ragged water box (13^3 molecules) under a thermostat, mixed form
        c("md_nvt_water_6591_mixed", "md", "water", 13, "mixed", 20, "nose-hoover"),
        # a small alloy (13^3 fcc cells), MD
        c("md_eam_8788", "md", "eam", 13, steps=30),
        # the all-FP64 form, used to check the others, on a mid-size melt
        c("forces_nacl_13824_native", "forces", "nacl", 24, "native"),
        # a mid-size melt (36^3 sites, 108^3 grid), single point in the mixed form
        c("forces_nacl_46656_mixed", "forces", "nacl", 36, "mixed"),
        # a Fortran driver's first evaluation at scale: list build and forces, 160^3 grid
        c("forces_nacl_175616", "forces", "nacl", 56),
        # production MD at the benchmark's size, in the two forms meant for it
        c("md_nacl_262144", "md", "nacl", 64, steps=10),
        c("md_nacl_262144_mixed", "md", "nacl", 64, "mixed", 10),
        # rigid water at scale: SHAKE/RATTLE, exclusions, a list rebuild every few steps
        c("md_water_98304", "md", "water", 32, steps=8),
        # the EAM alloy at scale
        c("md_eam_256000", "md", "eam", 40, steps=4),
    ]


# edge range per system and form: from the smallest box the cutoff allows to the listed maximum
RANGE = {"nacl": (10, 64), "water": (8, 32), "eam": (5, 40)}


def draw(rng):
    if rng.random() < 0.1:
        return {"kind": "kinstress", "n": int(round(math.exp(rng.uniform(math.log(64), math.log(1048576))))),
                "frozen": rng.random() < 0.5}
    system = rng.choice(["nacl", "nacl", "nacl", "water", "water", "eam"])
    lo, hi = RANGE[system]
    n_side = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if system == "nacl":
        n_side -= n_side % 2  # a rock-salt box is periodic with even edges
    form = "fp64" if system == "eam" else rng.choice(["fp64", "fp64", "mixed", "mixed", "native"])
    ensemble = "nve"
    if rng.random() < 0.5:
        kind, steps = "forces", 0
    else:
        kind = "md"
        steps = rng.randint(1, 4 if system == "eam" or form == "native" else 8)
        if n_side <= hi // 3:
            steps *= rng.randint(2, 5)
        ensemble = rng.choice(["nve", "nve", "nve", "nose-hoover", "berendsen", "langevin"])
        if system == "eam" or n_side > hi // 2:
            ensemble = "nve"
    return {"kind": kind, "system": system, "n_side": n_side, "form": form, "steps": steps, "ensemble": ensemble}


def _grid(edge):
    """SPME points per dimension: the next even 2^a 3^b 5^c at one point per Angstrom or denser."""
    k = int(math.ceil(edge))
    while True:
        m = k
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1 and k % 2 == 0:
            return k
        k += 1


def _system(case, seed):
    """One configuration; the topology (types, charges, masses) does not depend on the seed."""
    n = case["n_side"]
    if case["system"] == "nacl":
        return systems.nacl_melt(n, seed=seed, kmax=_grid(n * 2.82))
    if case["system"] == "water":
        edge = (n ** 3 * (15.9994 + 2 * 1.008) / 0.6022140857) ** (1.0 / 3.0)
        return systems.spce_water(n, seed=seed, kmax=_grid(edge))
    s = systems.eam_alloy(n)
    t = systems.eam_alloy(n, seed=seed)
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        setattr(s, k, getattr(t, k))
    return s


_held = {"key": None, "lib": None}


def _library(case, s):
    """The library holding this case's configuration (it holds one at a time)."""
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _held["key"] != key:
        lib = _held["lib"] or gb.load()
        _held["key"], _held["lib"] = None, lib
        lib.init(s, precision=FORMS[case["form"]])
        if case["ensemble"] != "nve":
            lib.set_ensemble(case["ensemble"], temp=TEMP[case["system"]], tau_t=TAU, chi=CHI, seed=(1, 2, 3))
        _held["key"] = key
    return key


def _kin_inputs(case, seed):
    g = torch.Generator().manual_seed(int(seed))
    n = case["n"]
    w = torch.where(torch.arange(n) % 2 == 0, 22.99, 35.45).double()
    v = torch.randn(3, n, generator=g, dtype=torch.float64) * torch.sqrt(0.831451115 * 1500.0 / w)
    fr = (torch.arange(n) % 97 == 0).to(torch.int32) if case["frozen"] else None
    return v, w, fr


def prepare(case, seed):
    if case["kind"] == "kinstress":
        if _held["lib"] is None:
            _held["lib"] = gb.load()
        f = _held["lib"].lib.gb_kinstress_noalloc
        f.restype = ctypes.c_int
        f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
        v, w, fr = _kin_inputs(case, seed)
        v, w = v.cuda(), w.cuda()
        fr = None if fr is None else fr.cuda()
        return {"kind": "kinstress", "f": f, "v": v, "w": w, "fr": fr, "n": case["n"],
                "out": torch.empty(9, dtype=torch.float64, device="cuda")}
    s = _system(case, seed)
    key = _library(case, s)
    rows = torch.empty((6, s.natms), dtype=torch.float64).pin_memory()
    rows.copy_(torch.from_numpy(np.stack([s.x, s.y, s.z, s.vx, s.vy, s.vz])))
    frame = torch.empty((9, s.natms), dtype=torch.float64).pin_memory()
    views = frame.numpy()
    return {"kind": case["kind"], "key": key, "steps": case["steps"], "single": case["form"] == "mixed",
            "in": list(rows.numpy()), "rows": rows, "frame": frame,
            "out": dict(zip(_held["lib"].STATE_KEYS, views))}


def run(state):
    if state["kind"] == "kinstress":
        v, fr = state["v"], state["fr"]
        rc = state["f"](v[0].data_ptr(), v[1].data_ptr(), v[2].data_ptr(), state["w"].data_ptr(),
                        None if fr is None else fr.data_ptr(), state["n"], state["out"].data_ptr(),
                        torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("gb_kinstress_noalloc: status %d" % rc)
        return state["out"]
    lib = _held["lib"]
    if _held["key"] != state["key"]:
        raise RuntimeError("the library holds another configuration")
    lib.upload(*state["in"])
    lib.set_step(0)
    lib.set_thermostat_state(0.0, 0.0)
    eng, stress = lib.start()
    res = {"eng": np.array(list(eng.values())), "stress": stress}
    if state["steps"]:
        st = lib.md_vv(state["steps"])
        res["md_scalars"] = np.array([[getattr(t, k) for k in SCALARS] for t in st])
        res["md_stress"] = np.array([t.stress[:] for t in st])
        res["md_strkin"] = np.array([t.strkin[:] for t in st])
        res["md_strcon"] = np.array([t.strcon[:] for t in st])
        res["md_counts"] = np.array([[t.list_rebuilt, t.shake_iters, t.rattle_iters] for t in st], dtype=np.int32)
    lib.download(state["out"])
    frame = state["frame"]
    if state["single"]:
        frame = frame.to(torch.float32)
        res = {k: v if v.dtype == np.int32 else v.astype(np.float32) for k, v in res.items()}
    res["pos"], res["vel"], res["force"] = frame[0:3], frame[3:6], frame[6:9]
    return res


# ------------------------------------------------------------------ what a pass cannot do without
def _shape(case):
    n = case["n_side"]
    if case["system"] == "nacl":
        natms, edge, rc, skin = n ** 3, n * 2.82, 12.0, 1.0
    elif case["system"] == "water":
        natms, edge, rc, skin = 3 * n ** 3, (n ** 3 * 18.0154 / 0.6022140857) ** (1.0 / 3.0), 10.0, 1.0
    else:
        natms, edge, rc, skin = 4 * n ** 3, n * 3.565, 7.0, 0.5
    return natms, edge, rc, skin


def work(case):
    if case["kind"] == "kinstress":
        n = case["n"]
        return {"bytes": n * (36.0 if case["frozen"] else 32.0) + 72, "flops": 13.0 * n}
    natms, edge, rc, skin = _shape(case)
    dens = natms / edge ** 3
    pairs = natms * dens * 2.0 / 3.0 * math.pi * rc ** 3
    entries = natms * dens * 2.0 / 3.0 * math.pi * (rc + skin) ** 3
    evals = 1 + case["steps"]
    flops = evals * pairs * (84.0 if case["system"] == "eam" else 55.0) + 10.0 * entries
    nbytes = natms * (48.0 + 72.0) + case["steps"] * natms * 208.0 + evals * (entries * 4.0 + natms * 48.0)
    if case["system"] != "eam":
        k = _grid(edge)
        word = 4.0 if case["form"] == "mixed" else 8.0
        flops += evals * (natms * (10.0 * 8 ** 3 + 3 * 88) + 5.0 * k ** 3 * 3 * math.log2(k))
        nbytes += evals * k ** 3 * word * 2
    if case["system"] == "water":
        flops += case["steps"] * natms * 120 * 40.0
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------- the same passes in plain torch, 64 bits
def exact(case, seed):
    if case["kind"] == "kinstress":
        v, w, fr = _kin_inputs(case, seed)
        if fr is not None:
            w = torch.where(fr != 0, torch.zeros_like(w), w)
        return (v * w) @ v.T
    if case["ensemble"] == "langevin":
        return None  # its noise is the library's own random stream
    natms = _shape(case)[0]
    if (1 + case["steps"]) * natms > 3.2e6:
        return None
    return _Exact(case, _system(case, seed)).run(case)


class _Exact:
    R4PIE0 = 138935.4835

    def __init__(self, case, s):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.s = s
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        self.x = t(np.stack([s.x, s.y, s.z], 1))
        self.v = t(np.stack([s.vx, s.vy, s.vz], 1))
        self.q, self.w = t(s.chge), t(s.weight)[:, None]
        self.type = t(s.ltype.astype(np.int64)) - 1
        self.L, self.n, self.dt = float(s.cell[0]), s.natms, s.tstep
        self.charged = bool((s.chge != 0).any())
        self.ens = case["ensemble"]
        self.chi_t = self.cint = 0.0
        deg = 3.0 * self.n - 3.0 - s.ntcons
        self.sigma = 0.5 * deg * 0.831451115 * TEMP[case["system"]]
        self.qmass = 2.0 * self.sigma * TAU * TAU
        if s.ntcons:
            lc = s.listcon.reshape(-1, 3).astype(np.int64)
            self.ci, self.cj = t(lc[:, 1] - 1), t(lc[:, 2] - 1)
            self.d0 = t(s.prmcon)[t(lc[:, 0] - 1)]
        self._tables()
        if self.charged:
            self._spme_setup()
        if s.eam:
            self._eam_setup()

    # interpolation tables of the real-space terms: value and force, points r = i h
    def _tables(self):
        s, rc = self.s, self.s.rcut
        n = max(1004, int(round(rc / 0.01)) + 4)
        self.h = rc / (n - 4)
        i = np.arange(n + 3, dtype=np.float64)
        i[0] = 1.0
        r = i * self.h
        a = s.alpha * r
        tt = 1.0 / (1.0 + 0.3275911 * a)
        erfc = tt * (0.254829592 + tt * (-0.284496736 + tt * (1.421413741 + tt * (-1.453152027 + tt * 1.061405429))))
        erfc = erfc * np.exp(-a * a)
        te = erfc / r
        td = (erfc / r + s.alpha * 2.0 * np.exp(-a * a) / math.sqrt(math.pi)) / (r * r)
        to = lambda v: torch.as_tensor(v, device=self.dev)  # noqa: E731
        self.te, self.td = to(te), to(td)
        nt = s.ntypes
        prm = s.vdw_prm.reshape(-1, 3)
        vp, vf = np.zeros((nt * nt, n + 3)), np.zeros((nt * nt, n + 3))
        for p in range(nt):
            for b in range(nt):
                k, eps, sig = prm[max(p, b) * (max(p, b) + 1) // 2 + min(p, b)]
                if k == 1:
                    s6 = (sig / r) ** 6
                    vp[p * nt + b], vf[p * nt + b] = 4 * eps * s6 * (s6 - 1), 24 * eps * s6 * (2 * s6 - 1)
        self.vp, self.vf = to(vp.reshape(-1)), to(vf.reshape(-1))
        self.nvdw, self.has_vdw = n + 3, bool((prm[:, 0] != 0).any())

    @staticmethod
    def _interp(tab, base, l, f):
        p1, p2, p3 = tab[base + l], tab[base + l + 1], tab[base + l + 2]
        t1 = p1 + (p2 - p1) * f
        t2 = p2 + (p3 - p2) * (f - 1.0)
        return t1 + (t2 - t1) * f * 0.5

    def _image(self, d):
        return d - self.L * torch.round(d / self.L)

    def _pairs(self, rc):
        """Batches of (i, j, d, r^2) over unique pairs within rc."""
        x, L, dev = self.x, self.L, self.dev
        nc = int(L / rc)
        if nc < 3:
            for a in range(0, self.n, 512):
                i = torch.arange(a, min(self.n, a + 512), device=dev)
                d = self._image(x[i][:, None, :] - x[None, :, :])
                r2 = (d * d).sum(-1)
                hit = (r2 <= rc * rc) & (i[:, None] < torch.arange(self.n, device=dev)[None, :])
                p, j = hit.nonzero(as_tuple=True)
                yield i[p], j, d[p, j], r2[p, j]
            return
        u = x / L + 0.5
        c = torch.clamp(((u - torch.floor(u)) * nc).long(), 0, nc - 1)
        cell = (c[:, 2] * nc + c[:, 1]) * nc + c[:, 0]
        order = torch.argsort(cell, stable=True)
        count = torch.bincount(cell, minlength=nc ** 3)
        start = torch.cumsum(count, 0) - count
        m = int(count.max())
        slot = torch.arange(self.n, device=dev) - start[cell[order]]
        table = torch.full((nc ** 3, m), -1, dtype=torch.int64, device=dev)
        table[cell[order], slot] = order
        g = torch.arange(nc, device=dev)
        cz, cy, cx = torch.meshgrid(g, g, g, indexing="ij")
        half = [(0, 0, 0)] + [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
                              if (dz, dy, dx) > (0, 0, 0)]
        step = max(1, int(4.0e7 // (m * m)))
        for dx, dy, dz in half:
            other = ((((cz + dz) % nc) * nc + (cy + dy) % nc) * nc + (cx + dx) % nc).reshape(-1)
            for a in range(0, nc ** 3, step):
                ti, tj = table[a:a + step], table[other[a:a + step]]
                ok = (ti[:, :, None] >= 0) & (tj[:, None, :] >= 0)
                if (dx, dy, dz) == (0, 0, 0):
                    ok &= ti[:, :, None] < tj[:, None, :]
                r2 = torch.zeros(ok.shape, dtype=torch.float64, device=dev)
                for k in range(3):
                    e = self._image(x[ti.clamp(min=0), k][:, :, None] - x[tj.clamp(min=0), k][:, None, :])
                    r2 += e * e
                b, p, o = (ok & (r2 <= rc * rc)).nonzero(as_tuple=True)
                i, j = ti[b, p], tj[b, o]
                d = self._image(x[i] - x[j])
                yield i, j, d, (d * d).sum(-1)

    def _spme_setup(self):
        s, dev = self.s, self.dev
        K, p = s.kmax[0], s.nsplines
        m = torch.arange(K, device=dev, dtype=torch.int64)
        ms = torch.where(2 * m > K, m - K, m).double() / self.L
        c = np.zeros(p + 1)
        c[2] = 1.0
        for k in range(3, p + 1):
            for j in range(k, 1, -1):
                c[j] = ((j - 1) * c[j] + (k - j + 1) * c[j - 1]) / (k - 1)
        i = np.arange(K)
        t = sum(c[k + 2] * np.exp(2j * np.pi * ((i * k) % K) / K) for k in range(p - 1))
        b = torch.as_tensor(1.0 / np.abs(t) ** 2, device=dev)
        k2 = ms[:, None, None] ** 2 + ms[None, :, None] ** 2 + ms[None, None, :] ** 2
        cut = 0.5 * 1.05 * K / self.L
        f2 = k2 * (math.pi / s.alpha) ** 2
        keep = (k2 <= cut * cut) & (k2 > 0)
        infl = b[:, None, None] * b[None, :, None] * b[None, None, :] * torch.exp(-f2) / (math.sqrt(math.pi) * f2)
        self.infl = torch.where(keep, infl, torch.zeros_like(infl))
        psi = self.infl * -2.0 * (1.0 + f2) / k2
        self.psi = torch.where(keep, psi, torch.zeros_like(psi))
        self.ms, self.K = ms, K
        self.scale = math.pi ** 1.5 / s.alpha ** 2 * 0.5 / self.L ** 3 * self.R4PIE0 / s.epsq
        self.self_energy = -float((s.chge ** 2).sum()) * self.R4PIE0 / s.epsq * s.alpha / math.sqrt(math.pi)

    def _splines(self, c):
        """Values and derivatives of the order-p B-spline at its p grid points; c (n, 3)."""
        p = self.s.nsplines
        z = [None] + [torch.zeros_like(c) for _ in range(p + 1)]
        z[p], z[p - 1] = c.clone(), 1.0 - c
        dv = None
        for k in range(p - 2, 0, -1):
            if k == 1:
                dv = [z[j] - z[j + 1] for j in range(1, p)] + [z[p].clone()]
            for j in range(1, p):
                pt = c + (p - j)
                z[j] = (pt * z[j] + ((p - k + 1) - pt) * z[j + 1]) / (p - k)
            z[p] = z[p] * c / (p - k)
        return torch.stack(z[1:p + 1], 1), torch.stack(dv, 1)  # (n, p, 3)

    def _spme(self, f, stress):
        s, K, p, n = self.s, self.K, self.s.nsplines, self.n
        u = K * (self.x / self.L + 0.5)
        grid = torch.zeros(K ** 3, dtype=torch.float64, device=self.dev)
        chunk = 32768
        o = torch.arange(p, device=self.dev) + 1 - p

        def stencil(base):
            g = (base[:, None, :] + o[None, :, None]) % K
            return (g[:, :, None, None, 2] * K + g[:, None, :, None, 1]) * K + g[:, None, None, :, 0]

        for a in range(0, n, chunk):
            b = torch.floor(u[a:a + chunk])
            sv, _ = self._splines(u[a:a + chunk] - b)
            wt = (self.q[a:a + chunk, None] * sv[:, :, 2])[:, :, None, None] * sv[:, None, :, None, 1] * sv[:, None, None, :, 0]
            grid.index_add_(0, stencil(b.long()).reshape(-1), wt.reshape(-1))
        G = torch.fft.fftn(grid.reshape(K, K, K))
        pv = self.psi * (G.real ** 2 + G.imag ** 2)
        st = torch.zeros((3, 3), dtype=torch.float64, device=self.dev)
        axis = [self.ms[None, None, :], self.ms[None, :, None], self.ms[:, None, None]]
        for a in range(3):
            for b in range(a, 3):
                st[a, b] = st[b, a] = (pv * axis[a] * axis[b]).sum()
        del pv
        phi = torch.fft.ifftn(G * self.infl).real.reshape(-1) * float(K) ** 3
        del G
        cf = torch.empty((n, 3), dtype=torch.float64, device=self.dev)
        energy = 0.0
        for a in range(0, n, chunk):
            b = torch.trunc(u[a:a + chunk])  # toward zero, as the gather of the reference does
            sv, dv = self._splines(u[a:a + chunk] - b)
            ph = phi[stencil(b.long())]
            q = self.q[a:a + chunk]
            x0, x1 = (ph * sv[:, None, None, :, 0]).sum(-1), (ph * dv[:, None, None, :, 0]).sum(-1)
            y00, y10 = (x0 * sv[:, None, :, 1]).sum(-1), (x0 * dv[:, None, :, 1]).sum(-1)
            y01 = (x1 * sv[:, None, :, 1]).sum(-1)
            z0, z1 = sv[:, :, 2], dv[:, :, 2]
            cf[a:a + chunk, 0] = q * (y01 * z0).sum(-1)
            cf[a:a + chunk, 1] = q * (y10 * z0).sum(-1)
            cf[a:a + chunk, 2] = q * (y00 * z1).sum(-1)
            energy += float((q * (y00 * z0).sum(-1)).sum())
        cf *= K / self.L
        f += -(cf - cf.mean(0)) * (2.0 * self.scale)
        eng = energy * self.scale
        stt = st * self.scale + eng * torch.eye(3, dtype=torch.float64, device=self.dev)
        stress += stt
        return eng + self.self_energy, -float(torch.trace(stt))

    def _eam_setup(self):
        """Tables by point: start, spacing, values and (minus r times, but for the embedding) derivatives."""
        self.tab = {}
        for t in self.s.eam:
            y = np.asarray(t["values"], np.float64)
            ng = len(y)
            h = (t["finish"] - t["start"]) / (ng - 1)
            d = np.zeros(ng)
            for i in range(2, ng - 2):
                d[i] = self._derivative(y, i, h, 0)
            d[0], d[1] = self._derivative(y, 2, h, -2), self._derivative(y, 2, h, -1)
            d[ng - 2], d[ng - 1] = self._derivative(y, ng - 3, h, 1), self._derivative(y, ng - 3, h, 2)
            base = t["start"] - 5.0 * h
            if t["kind"] != "embe":
                d = -((np.arange(ng) + 5.0) * h + base) * d
            pad = lambda v: torch.as_tensor(np.concatenate([np.zeros(5), v, np.zeros(4)]), device=self.dev)  # noqa: E731
            self.tab[(t["kind"], tuple(sorted(t["types"])))] = (base, h, ng, t["start"], t["finish"], pad(y), pad(d))

    @staticmethod
    def _derivative(y, i, h, at):
        if y[i] == 0.0:
            return 0.0
        f0, f1, f2, f3, f4 = y[i - 2] / y[i], y[i - 1] / y[i], 1.0, y[i + 1] / y[i], y[i + 2] / y[i]
        d1, d2, d3 = f1 - f0, (f2 - f1) - (f1 - f0), (f3 - f0) + 3.0 * (f1 - f2)
        d4 = (f4 - f3) + 3.0 * (f2 - f3) + 3.0 * (f2 - f1) + (f0 - f1)
        a4 = d4 / 24.0
        a3 = (d3 + 12.0 * a4) / 6.0
        a2 = (d2 + 6.0 * a3 - 14.0 * a4) / 2.0
        a1 = d1 + 3.0 * a2 - 7.0 * a3 + 15.0 * a4
        return (a1 + 2.0 * at * a2 + 3.0 * at * at * a3 + 4.0 * at ** 3 * a4) * y[i] / h

    def _eam_interp(self, tab, values, r, density=False):
        base, h, ng = tab[0], tab[1], tab[2]
        u = (r - base) / h
        l = torch.clamp(torch.floor(u + 0.5).long(), max=ng + 3)
        f = u - l
        v0, v1, v2 = values[l - 1], values[l], values[l + 1]
        t1, t2 = v1 + f * (v1 - v0), v1 + f * (v2 - v1)
        lo, hi = t1 + 0.5 * (t2 - t1) * (f + 1.0), t2 + 0.5 * (t2 - t1) * (f - 1.0)
        if density:
            lo, hi = torch.where(lo < 0, t1, lo), torch.where(hi < 0, t2, hi)
        return torch.where(f < 0, lo, torch.where(l == 5, t2, hi))

    def _eam(self, f, stress):
        nt = self.s.ntypes
        rho = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        batches = list(self._pairs(self.s.rcut))
        for i, j, d, r2 in batches:
            r = torch.sqrt(r2)
            for a, b in ((i, j), (j, i)):  # b's density at a
                for t in range(nt):
                    tab = self.tab[("dens", (t + 1, t + 1))]
                    k = ((self.type[b] == t) & (r <= tab[4])).nonzero(as_tuple=True)[0]
                    rho.index_add_(0, a[k], self._eam_interp(tab, tab[5], r[k], True))
        engden, fp = 0.0, torch.zeros_like(rho)
        for t in range(nt):
            tab = self.tab[("embe", (t + 1, t + 1))]
            k = (self.type == t).nonzero(as_tuple=True)[0]
            engden += float(self._eam_interp(tab, tab[5], rho[k]).sum())
            fp[k] = self._eam_interp(tab, tab[6], rho[k])
        engmet = virmet = 0.0
        for i, j, d, r2 in batches:
            r = torch.sqrt(r2)
            gamma, eng = torch.zeros_like(r), torch.zeros_like(r)
            for a in range(nt):
                for b in range(nt):
                    k = ((self.type[i] == a) & (self.type[j] == b)).nonzero(as_tuple=True)[0]
                    pt = self.tab[("pair", (min(a, b) + 1, max(a, b) + 1))]
                    da, db = self.tab[("dens", (a + 1, a + 1))], self.tab[("dens", (b + 1, b + 1))]
                    eng[k] = self._eam_interp(pt, pt[5], r[k])
                    gamma[k] = self._eam_interp(pt, pt[6], r[k]) + self._eam_interp(db, db[6], r[k]) * fp[i[k]] \
                        + self._eam_interp(da, da[6], r[k]) * fp[j[k]]
            gamma /= r2
            F = gamma[:, None] * d
            f.index_add_(0, i, F)
            f.index_add_(0, j, -F)
            engmet += float(eng.sum())
            virmet -= float((gamma * r2).sum())
            stress += d.T @ F
        return engmet + engden, virmet

    def _forces(self):
        s, nt = self.s, self.s.ntypes
        f = torch.zeros_like(self.x)
        stress = torch.zeros((3, 3), dtype=torch.float64, device=self.dev)
        e = np.zeros(8)
        met = (0.0, 0.0)
        if self.charged:
            e[0], e[1] = self._spme(f, stress)
        if s.eam:
            met = self._eam(f, stress)
        if self.charged or self.has_vdw:
            qs = self.q * (self.R4PIE0 / s.epsq)
            for i, j, d, r2 in self._pairs(s.rcut):
                if s.ntcons:  # the three sites of a molecule exclude one another
                    k = (i // 3 != j // 3).nonzero(as_tuple=True)[0]
                    i, j, d, r2 = i[k], j[k], d[k], r2[k]
                r = torch.sqrt(r2)
                u = r / self.h
                l = u.long()
                u = u - l
                qq = qs[i] * self.q[j]
                gam = qq * self._interp(self.td, 0, l, u)
                e[2] += float((qq * self._interp(self.te, 0, l, u)).sum())
                e[3] -= float((gam * r2).sum())
                if self.has_vdw:
                    base = (self.type[i] * nt + self.type[j]) * self.nvdw
                    gv = self._interp(self.vf, base, l, u)
                    e[6] += float(self._interp(self.vp, base, l, u).sum())
                    e[7] -= float(gv.sum())
                    gam = gam + gv / r2
                F = gam[:, None] * d
                f.index_add_(0, i, F)
                f.index_add_(0, j, -F)
                stress += d.T @ F
        if s.ntcons:
            for a, b in ((0, 1), (0, 2), (1, 2)):
                i = 3 * torch.arange(self.n // 3, device=self.dev) + a
                j = i + (b - a)
                d = self._image(self.x[i] - self.x[j])
                r2 = (d * d).sum(-1)
                r = torch.sqrt(r2)
                qq = qs[i] * self.q[j]
                tt = 1.0 / (1.0 + 0.3275911 * s.alpha * r)
                ex = torch.exp(-(s.alpha * r) ** 2)
                poly = tt * (0.254829592 + tt * (-0.284496736 + tt * (1.421413741 + tt * (-1.453152027 + tt * 1.061405429))))
                erf = qq * (1.0 - poly * ex) / r
                gam = -(erf - 2.0 * qq * (s.alpha / math.sqrt(math.pi)) * ex) / r2
                F = gam[:, None] * d
                f.index_add_(0, i, F)
                f.index_add_(0, j, -F)
                e[4] -= float(erf.sum())
                e[5] -= float((gam * r2).sum())
                stress += d.T @ F
        return f, e, met, stress

    def _wrap(self):
        u = self.x / self.L
        u = u - torch.round(u)
        self.x = self.L * torch.where(u >= 0.5, -u, u)
        self.x0 = self.x.clone()

    def _kinetic(self):
        st = (self.v * self.w).T @ self.v
        return st, 0.5 * float(torch.trace(st))

    def _nose_hoover(self, dt):
        h, q = 0.5 * dt, 0.25 * dt
        ek = self._kinetic()[1]
        self.cint += q * self.chi_t
        self.chi_t += h * (2.0 * ek - 2.0 * self.sigma) / self.qmass
        self.cint += h * self.chi_t
        scale = math.exp(-dt * self.chi_t)
        self.v *= scale
        ek *= scale * scale
        self.chi_t += h * (2.0 * ek - 2.0 * self.sigma) / self.qmass
        self.cint += q * self.chi_t
        return ek

    def _spread_bonds(self, a, b):
        out = torch.zeros_like(self.x)
        out.index_add_(0, self.ci, a)
        out.index_add_(0, self.cj, b)
        return out

    def _shake(self, bond):
        s, dt = self.s, self.dt
        x0 = self.x.clone()
        str_ = torch.zeros((3, 3), dtype=torch.float64, device=self.dev)
        ai, aj = dt * dt / self.w[self.ci, 0], dt * dt / self.w[self.cj, 0]
        it = 0
        while it < s.shake_maxit:
            it += 1
            d = self._image(self.x[self.ci] - self.x[self.cj])
            t = (d * d).sum(-1) - self.d0 ** 2
            if bool((0.5 * t.abs() < s.shake_tol * self.d0).all()):
                break
            gamma = t / ((ai + aj) * (bond * d).sum(-1))
            str_ -= (gamma[:, None] * bond).T @ bond
            self.x = self.x + self._spread_bonds(bond * (-0.5 * gamma * ai)[:, None], bond * (0.5 * gamma * aj)[:, None])
        self.v = self.v + (self.x - x0) / dt
        return it, str_

    def _rattle(self, bond):
        s, dt = self.s, self.dt
        bond = bond / bond.norm(dim=1, keepdim=True)
        ai, aj = dt / self.w[self.ci, 0], dt / self.w[self.cj, 0]
        it = 0
        while it < s.shake_maxit:
            it += 1
            gamma = (bond * (self.v[self.ci] - self.v[self.cj])).sum(-1)
            if float(gamma.abs().max()) * 0.5 * dt < s.shake_tol:
                break
            gamma = gamma / (ai + aj)
            self.v = self.v + self._spread_bonds(bond * (-gamma * ai)[:, None], bond * (gamma * aj)[:, None])
        return it

    def run(self, case):
        s, dt = self.s, self.dt
        cons = s.ntcons > 0
        bonds = lambda: self._image(self.x[self.ci] - self.x[self.cj]) if cons else None  # noqa: E731
        self._wrap()
        f, e, met, stress = self._forces()
        res = {"eng": e, "stress": stress.T.reshape(9).cpu().numpy()}
        rows = {k: [] for k in ("md_scalars", "md_stress", "md_strkin", "md_strcon", "md_counts")}
        for _ in range(case["steps"]):
            it1 = it2 = 0
            strcon = torch.zeros((3, 3), dtype=torch.float64, device=self.dev)
            b = bonds()
            if self.ens == "nose-hoover":
                self._nose_hoover(0.5 * dt)
            self.v = self.v + (0.5 * dt) / self.w * f
            self.x = self.x + dt * self.v
            if cons:
                it1, strcon = self._shake(b)
            moved = self._image(self.x - self.x0).norm(dim=1).max()
            rebuilt = int(float(moved) >= 0.5 * s.rpad)
            if rebuilt:
                self._wrap()
            f, e, met, stress = self._forces()
            b = bonds()
            self.v = self.v + (0.5 * dt) / self.w * f
            if cons:
                it2 = self._rattle(b)
            consv = 0.0
            if self.ens == "berendsen":
                for last in (False, True):
                    sk, ek = self._kinetic()
                    if not last:
                        self.v *= math.sqrt(1.0 + dt / TAU * (self.sigma / ek - 1.0))
                        self.v = self.v - (self.w * self.v).sum(0) / self.w.sum()
            elif self.ens == "nose-hoover":
                ek = self._nose_hoover(0.5 * dt)
                consv = 0.5 * self.qmass * self.chi_t ** 2 + 2.0 * self.sigma * self.cint
                sk = self._kinetic()[0]
            else:
                sk, ek = self._kinetic()
            rows["md_scalars"].append(list(e) + [ek, -float(torch.trace(strcon)), consv, met[0], met[1]])
            rows["md_stress"].append(stress.T.reshape(9).cpu().numpy())
            rows["md_strkin"].append(sk.reshape(9).cpu().numpy())
            rows["md_strcon"].append(strcon.reshape(9).cpu().numpy())
            rows["md_counts"].append([rebuilt, it1, it2])
        if case["steps"]:
            for k, v in rows.items():
                res[k] = np.array(v, dtype=np.int32 if k == "md_counts" else np.float64)
        for k, v in (("pos", self.x), ("vel", self.v), ("force", f)):
            res[k] = v.T.contiguous().cpu()
        return res
