"""The work that this framework is used for, as cases that can be timed and compared.

A case is one call sequence of a host program on the C ABI (include/orbc_gpu.h): the reference's containers (x, n, v,
o) go in, a stretch of the main loop (or another entry point) runs on the GPU, the containers come back.

call      run       set_state, step(steps), download: a host program that owns the containers
          resident  step(steps), download: a run that goes on from where the last pass left it, read back for a frame
          forces    set_state, forces: the forces / torques / energies of a given configuration
          minimize  set_state, minimize(steps), download: the relaxation that precedes a run
          rdf       the pair-distance histogram of the current state
system    lattice   flat jittered lipid sheet, periodic in the plane
          vesicle   spherical lipid vesicle in the reference's open +-1000 box
          rbc       red-cell membrane with spectrin anchors, bonds and the area / volume constraint
          vesicles  a batch of vesicles, each in its own periodic box, advanced in one launch per step
form      orbc_params.kernel_variant: 0 is what a program gets that chooses nothing; 55 is what the autotuner picks on
          large mixed systems, 51 the same for FP64 and Nose-Hoover, 115 with compensated sums
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from openrbc_gb300 import RTParameter, Simulation, workloads
from openrbc_gb300 import _native as N

DT, ETA, SEED = 0.01, 0.01, 0xBAD5EED


def _case(name, call, system, n, **kw):
    c = {"name": name, "call": call, "system": system, "n": n, "precision": "mixed", "integrator": "langevin",
         "form": 55, "skin": 0.8, "kT": 1.0, "steps": 20, "energy": False}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one step of a small patch whose containers the host owns (latency and launches)
        _case("patch_step1", "run", "lattice", 2048, form=0, skin=0.4, steps=1),
        # the plain small workload: the 32,768-lipid periodic lattice, mixed precision
        _case("lattice_mixed", "run", "lattice", 32768, skin=0.5),
        # the same in plain FP64, the form that matches the reference's FP64 build
        _case("lattice_fp64", "run", "lattice", 32768, precision="fp64", form=51, skin=0.5, steps=10),
        # the command-line driver's default vesicle with nothing chosen: untuned form and skin, the reference's kBT
        _case("vesicle_default", "resident", "vesicle", 131946, form=0, skin=0.4, kT=0.22),
        # relaxation before a run, with the default form
        _case("vesicle_minimize", "minimize", "vesicle", 20011, form=0, skin=0.4, steps=5),
        # whole cell in FP64: the precise run that mixed runs are checked against
        _case("cell_fp64", "run", "rbc", 250000, precision="fp64", form=51, steps=5),
        # the FP64 check of a configuration: forces, torques and energies of the host's state
        _case("cell_forces_fp64", "forces", "rbc", 120001, precision="fp64", form=51),
        # Nose-Hoover cell with compensated sums and the energy kept, as the long constant-temperature run has it
        _case("cell_nose_hoover", "resident", "rbc", 500000, integrator="nose-hoover", form=115, kT=0.22,
              energy=True),
        # many systems of uneven size in one launch per step
        _case("vesicle_batch", "run", "vesicles", 1000000, skin=1.0),
        # host containers stay the source of truth: state in, one step, state out
        _case("cell_host_loop", "run", "rbc", 1000000, steps=1),
        # the flagship: the 4.03M-particle red cell
        _case("cell_4m", "run", "rbc", 4000000),
        # pair statistics of a snapshot
        _case("lattice_rdf", "rdf", "lattice", 32768, form=0, skin=0.4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["run", "run", "run", "resident", "forces", "minimize", "rdf"])
    fp64 = call != "rdf" and rng.random() < 0.3
    prec = "fp64" if fp64 else "mixed"
    if call == "rdf":
        return _drawn("rdf", "lattice", size(1000, 40000), form=0, skin=0.4)
    if call == "minimize":
        return _drawn("minimize", rng.choice(["vesicle", "rbc"]), size(3000, 60000 if fp64 else 400000),
                      precision=prec, form=rng.choice([0, 3]), skin=rng.choice([0.4, 0.6]),
                      steps=rng.randint(10, 20) if fp64 else rng.randint(2, 5))
    if call == "forces":
        # the mixed hook returns FP32 forces in FP64 arrays: the FP64 hook is the one that is compared in 64 bits
        return _drawn("forces", rng.choice(["lattice", "vesicle", "rbc"]), size(2000, 250000), precision="fp64",
                      form=rng.choice([0, 51]), skin=rng.choice([0.4, 0.8]))
    system = rng.choice(["lattice", "vesicle", "rbc", "vesicles"])
    lo = {"lattice": 1500, "vesicle": 3000, "rbc": 8000, "vesicles": 60000}[system]
    hi = 200000 if fp64 else 1500000
    nh = rng.random() < 0.35
    if call == "resident" or nh:
        call, kT = "resident", 0.22
    else:
        kT = rng.choice([0.22, 1.0])
    form = rng.choice([0, 3, 19, 51] if fp64 else ([0, 19, 51, 115] if nh else [0, 7, 23, 51, 55]))
    return _drawn(call, system, size(lo, hi), precision=prec, integrator="nose-hoover" if nh else "langevin",
                  form=form, skin=rng.choice([0.3, 0.4, 0.5, 0.6, 0.8, 1.0]), kT=kT,
                  steps=rng.randint(1, 8) if fp64 else rng.randint(1, 20), energy=nh and rng.random() < 0.5)


def _drawn(call, system, n, **kw):
    c = _case("", call, system, n, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _geometry(system, n):
    """The generator's particles and topology of one workload (its seed belongs to the workload, as in the benchmark)."""
    if system == "lattice":
        ncol = max(8, int(round(math.sqrt(n))))
        rows = -(-n // ncol)
        w = workloads.lattice(n=n, ncol=ncol, spacing=1.1, jitter=0.05, tilt=0.05, kT=1.0, seed=1)
        w["systems"] = [{"lo": (0.0, 0.0, -20.0), "hi": (1.1 * ncol, 1.1 * rows, 20.0), "periodic": (1, 1, 1)}]
    elif system == "rbc":
        w = workloads.rbc(n_lipid=n, freq=max(4, int(round(57 * math.sqrt(n / 4.0e6)))), kT=1.0, seed=2)
        w["systems"] = [{"lo": (-1000.0,) * 3, "hi": (1000.0,) * 3, "periodic": (0, 0, 0), **w["constraint"]}]
    else:
        w = _vesicles(system, n)
    if "offsets" not in w:
        w["offsets"] = np.array([0, len(w["x"])], np.int64)
    return w


def _system(case, seed):
    """One case's containers: the workload's geometry as it is within a run -- positions and normals moved and tilted by
    the thermal motion, velocities and angular velocities of the case's temperature -- all drawn from the seed."""
    w, sd = dict(_geometry(case["system"], case["n"])), math.sqrt(case["kT"])
    g = np.random.default_rng(int(seed))
    w["x"] = w["x"] + 0.02 * g.standard_normal(w["x"].shape)
    w["n"] = w["n"] + 0.1 * g.standard_normal(w["x"].shape)
    w["n"] /= np.sqrt(np.einsum("ij,ij->i", w["n"], w["n"]))[:, None]
    w["v"] = sd * g.standard_normal(w["x"].shape)  # lipids and anchors have mass 1
    w["o"] = 0.5 * sd * g.standard_normal(w["x"].shape)
    return w


def _vesicles(system, n):
    """Spherical vesicles of the surface density 1.05: one in the reference's open box, or a batch of log-normal sizes,
    each in a periodic box of edge 2.5 diameters."""
    lib = N.lib()
    sizes = np.array([n], np.int64)
    if system == "vesicles":
        sizes = np.zeros(max(3, n // 42000), np.int64)
        k = len(sizes)
        if lib.orbc_gen_vesicle_sizes(k, max(2000, n // (4 * k)), max(4000, 6 * n // k), int(0.8 * n / k), n, 4,
                                      sizes.ctypes.data):
            raise ValueError("orbc_gen_vesicle_sizes failed")
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    m = int(off[-1])
    x, nn, v, o = (np.zeros((m, 3)) for _ in range(4))
    ty, tg = np.zeros(m, np.int32), np.zeros(m, np.int32)
    systems = []
    for k, (a, b) in enumerate(zip(off[:-1], off[1:])):
        R = C.c_double()
        if lib.orbc_gen_vesicle(int(b - a), 1.05, 1.0, 4000 + k, int(a) + 1,
                                *[q[a:].ctypes.data for q in (x, nn, v, o, ty, tg)], C.byref(R)):
            raise ValueError("orbc_gen_vesicle failed")
        half = 2.5 * R.value if system == "vesicles" else 1000.0
        systems.append({"lo": (-half,) * 3, "hi": (half,) * 3,
                        "periodic": (1, 1, 1) if system == "vesicles" else (0, 0, 0)})
    return {"x": x, "n": nn, "v": v, "o": o, "type": ty, "tag": tg, "offsets": off, "systems": systems}


def _containers(m, dtype, count=4):
    """Page-locked host arrays, as a host program that exchanges them every step keeps them."""
    return [torch.empty((m, 3), dtype=dtype, pin_memory=True) for _ in range(count)]


def prepare(case, seed):
    w = _system(case, seed)
    fp64 = case["precision"] == "fp64"
    p = RTParameter(init="trimesh", mesh="synthetic", kBT=case["kT"], dt=DT, eta=ETA, precision=case["precision"],
                    integrator=case["integrator"], rseed=SEED)
    sim = Simulation(p, skin=case["skin"], kernel_variant=case["form"], energy=case["energy"],
                     bond_table=workloads.RBC_BOND_TABLE)
    sim.upload_batch(w["systems"], w["x"], w["n"], w["v"], w["o"], w["type"], w["tag"], w["offsets"],
                     bonds=w.get("bonds"), bond_r0=w.get("bond_r0"), faces=w.get("faces"))
    m = len(w["x"])
    dtype = torch.float64 if fp64 else torch.float32
    state = {"case": case, "sim": sim, "m": m}
    if case["call"] in ("run", "forces", "minimize"):
        state["in"] = _containers(m, dtype)
        for h, a in zip(state["in"], (w["x"], w["n"], w["v"], w["o"])):
            h.copy_(torch.from_numpy(a))
    if case["call"] in ("run", "resident", "minimize"):
        state["out"] = _containers(m, dtype)
    return state


def run(state):
    case, sim, m = state["case"], state["sim"], state["m"]
    lib, h, fp64 = N.lib(), sim.h, case["precision"] == "fp64"
    if "in" in state:
        ptr = [a.data_ptr() for a in state["in"]]
        N.check(lib.orbc_gpu_set_state(h, *ptr) if fp64 else lib.orbc_gpu_set_state_f32(h, 0, m, 3, *ptr), h)
    if case["call"] == "forces":
        f, t, e = sim.forces()
        return {"f": f, "t": t, "e": e}
    if case["call"] == "rdf":
        counts, dropped = sim.rdf(dr=0.1, nbins=10000)
        return {"counts": counts.astype(np.int64), "dropped": dropped}
    out = {}
    if case["call"] == "minimize":
        sim.minimize(case["steps"], 0.05, 0.05)
    elif case["call"] == "resident":
        # a run prints its temperature, area and volume where it writes a frame
        th = sim.step(case["steps"])
        out = {k: th[k] for k in ("temperature", "area", "volume")}
    else:
        N.check(lib.orbc_gpu_step(h, case["steps"], None), h)
    ptr = [a.data_ptr() for a in state["out"]]
    N.check(lib.orbc_gpu_download(h, *ptr) if fp64 else lib.orbc_gpu_download_f32(h, 0, m, 3, *ptr), h)
    out.update(zip(("x", "n", "v", "o"), state["out"]))
    return out


def work(case):
    """Bytes: the state in and out of each step (x, n, v, o as 16-byte records, the tag and the displacement reference:
    104 B in FP32, 192 B in FP64) and the containers over the host link; flops: 106 per interacting pair, each pair
    once, with the 21 partners in range that a lipid of these membranes has on average."""
    n, k, fp64 = case["n"], case["steps"], case["precision"] == "fp64"
    host = 12 * (8 if fp64 else 4) * n
    if case["call"] == "rdf":
        return {"bytes": 16 * n, "flops": 0.5 * n * n * 9}
    if case["call"] == "forces":
        return {"bytes": host + (7 * 8 + (64 if fp64 else 32)) * n, "flops": 106 * 10.5 * n}
    moved = host * (1 if case["call"] == "resident" else 2)
    return {"bytes": moved + (192 if fp64 else 104) * n * k, "flops": 106 * 10.5 * n * k}


# ---------------------------------------------------------------------------------------------------------------------
# What run() returns, in 64 bits, in plain torch (src/pairwise_kernel.h:30-68, src/compute_bonded.h:89-146,
# src/integrate_langevin.h:99-149, src/integrate_nh.h:146-273, src/openrbc.cpp:88-146).
# Particle types here are lipids (0) and spectrin anchors (3).
def _pairs(x, sysid, systems, reach):
    """All i < j of one system closer than `reach`, with the periodic image's shift of x_i - x_j."""
    out_i, out_j, out_s = [], [], []
    for s, d in enumerate(systems):
        idx = torch.nonzero(sysid == s)[:, 0] if len(systems) > 1 else torch.arange(len(x), device=x.device)
        p = x[idx]
        per = [bool(v) for v in d["periodic"]]
        lo = p.new_tensor([d["lo"][a] if per[a] else float(p[:, a].min()) for a in range(3)])
        L = [d["hi"][a] - d["lo"][a] if per[a] else float(p[:, a].max()) - float(lo[a]) + 1e-6 for a in range(3)]
        nc = [max(1, min(2000, int(L[a] / reach))) for a in range(3)]
        q = p - lo
        for a in range(3):
            if per[a]:
                q[:, a] -= torch.floor(q[:, a] / L[a]) * L[a]
        c = [torch.clamp((q[:, a] * (nc[a] / L[a])).long(), 0, nc[a] - 1) for a in range(3)]
        key = (c[0] * nc[1] + c[1]) * nc[2] + c[2]
        order = torch.argsort(key, stable=True)
        skey = key[order]
        for off in range(27):
            o = (off // 9 - 1, off // 3 % 3 - 1, off % 3 - 1)
            if o < (0, 0, 0):
                continue
            t, shift, ok = [], torch.zeros_like(p), torch.ones(len(p), dtype=torch.bool, device=x.device)
            for a in range(3):
                v = c[a] + o[a]
                if per[a]:
                    shift[:, a] = L[a] * ((v < 0).to(p.dtype) - (v >= nc[a]).to(p.dtype))
                    v = v % nc[a]
                else:
                    ok &= (v >= 0) & (v < nc[a])
                t.append(v)
            tk = (t[0] * nc[1] + t[1]) * nc[2] + t[2]
            b, e = torch.searchsorted(skey, tk), torch.searchsorted(skey, tk, right=True)
            cnt = torch.where(ok, e - b, 0)
            for k0 in range(0, len(p), 400000):
                kk = torch.arange(k0, min(len(p), k0 + 400000), device=x.device)
                m = cnt[kk]
                i = torch.repeat_interleave(kk, m)
                j = torch.arange(len(i), device=x.device) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
                j = order[j + torch.repeat_interleave(b[kk], m)]
                d3 = q[i] - q[j] + shift[i]
                keep = (d3 * d3).sum(1) < reach * reach
                if off == 13:
                    keep &= i < j
                i, j = i[keep], j[keep]
                out_i.append(idx[i])
                out_j.append(idx[j])
                # x_i - x_j + s is the image distance in the caller's own coordinates
                out_s.append((q[i] - q[j] + shift[i]) - (p[i] - p[j]))
    return torch.cat(out_i), torch.cat(out_j), torch.cat(out_s)


class _Exact:
    def __init__(self, case, seed):
        dev = torch.device("cuda")
        w = _system(case, seed)
        fp64 = case["precision"] == "fp64"
        given = case["call"] in ("run", "forces", "minimize")

        def put(a):
            t = torch.from_numpy(np.ascontiguousarray(a)).to(dev).double()
            return t.float().double() if given and not fp64 else t

        self.case, self.w, self.dev = case, w, dev
        self.x, self.n, self.v, self.o = (put(w[k]) for k in ("x", "n", "v", "o"))
        self.ty = torch.from_numpy(w["type"]).to(dev).long()
        self.tag = torch.from_numpy(w["tag"]).to(dev).long()
        off = torch.from_numpy(np.asarray(w["offsets"])).to(dev)
        self.sysid = torch.bucketize(torch.arange(len(self.x), device=dev), off[1:], right=True)
        self.ref = None
        if "bonds" in w:
            b = torch.from_numpy(w["bonds"]).to(dev).long()
            self.bi, self.bj, self.r0 = b[:, 1] - 1, b[:, 2] - 1, torch.from_numpy(w["bond_r0"]).to(dev)
            self.face = torch.from_numpy(w["faces"]).to(dev).long() - 1

    def mesh(self):
        a, b, c = (self.x[self.face[:, k]] for k in range(3))
        area = 0.5 * torch.linalg.norm(torch.linalg.cross(b - a, c - a), dim=1).sum()
        vol = (a * torch.linalg.cross(b, c)).sum() / 6.0
        return float(area), float(vol)

    def forces(self):
        x, n = self.x, self.n
        if self.ref is None or float(((x - self.ref) ** 2).sum(1).max()) > 0.2 ** 2:
            self.i, self.j, self.s = _pairs(x, self.sysid, self.w["systems"], 2.6 + 0.4)
            self.ref = x.clone()
        d = x[self.i] - x[self.j] + self.s
        near = (d * d).sum(1) < 2.6 * 2.6
        i, j, d = self.i[near], self.j[near], d[near]
        r = torch.linalg.norm(d, dim=1)
        prot = (self.ty[i] != 0).long() + (self.ty[j] != 0).long()  # proteins in the pair
        eps, alpha = x.new_tensor([1.2, 2.8, 1.0])[prot], x.new_tensor([1.55, 5.0, 0.0])[prot]
        rep, att = eps / (2.6 - 1.1225) ** 8, -2.0 * eps / (2.6 - 1.1225) ** 4
        att = torch.where(prot == 2, torch.zeros_like(att), att)
        u = d / r[:, None]
        ni, nj = n[i], n[j]
        nn, niu, nju = (ni * nj).sum(1), (ni * u).sum(1), (nj * u).sum(1)
        A = 1.0 + alpha * (nn - niu * nju - 1.0)
        rc = 2.6 - r
        pi, pj = ni - niu[:, None] * u, nj - nju[:, None] * u
        aa = alpha * att * rc ** 4
        f = (8.0 * rep * rc ** 7 + A * 4.0 * att * rc ** 3)[:, None] * u
        f = f + (aa / r)[:, None] * (nju[:, None] * pi + niu[:, None] * pj)
        e = 0.5 * (rep * rc ** 8 + A * att * rc ** 4)
        F, T, E = torch.zeros_like(x), torch.zeros_like(x), torch.zeros(len(x), dtype=x.dtype, device=self.dev)
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        T.index_add_(0, i, -aa[:, None] * pj)
        T.index_add_(0, j, -aa[:, None] * pi)
        E.index_add_(0, i, e)
        E.index_add_(0, j, e)
        if "bonds" in self.w:
            K, ratio = 1.0, 2.2
            d = x[self.bj] - x[self.bi]
            r = torch.linalg.norm(d, dim=1)
            lmax = ratio * self.r0
            z, z0 = r / lmax, 1.0 / ratio
            fw = K * (0.25 / (1 - z) ** 2 - 0.25 + z)
            fw0 = K * (0.25 / (1 - z0) ** 2 - 0.25 + z0)
            q = self.r0 / r
            g = ((fw - fw0 * q * q) / r)[:, None] * d
            F.index_add_(0, self.bi, g)
            F.index_add_(0, self.bj, -g)
            ub = 0.5 * (K * lmax * (0.5 * z * z + 0.25 / (1 - z) - 0.25 * z - 0.25) + fw0 * self.r0 * q)
            E.index_add_(0, self.bi, ub)
            E.index_add_(0, self.bj, ub)
            c = self.w["constraint"]
            area, vol = self.mesh()
            cv, ca = -c["kv"] * (vol - c["V0"]) / c["V0"], -c["ka"] * (area - c["A0"]) / c["A0"]
            for k in range(3):
                va, vb, vc = (self.face[:, (k + m) % 3] for m in range(3))
                b, cc = x[vb] - x[va], x[vc] - x[va]
                nv = torch.linalg.cross(b, cc)
                g = torch.linalg.cross(b - cc, nv / torch.linalg.norm(nv, dim=1, keepdim=True))
                F.index_add_(0, va, cv / 6.0 * nv + 0.5 * ca * g)
        return F, T, E

    def noise(self, step):
        m32 = 0xFFFFFFFF

        def mul(a, c):
            return ((a * (c >> 16) + ((a * (c & 0xFFFF)) >> 16)) >> 16) & m32, (a * (c & 0xFFFF) + ((a * (c >> 16) & 0xFFFF) << 16)) & m32

        c = [self.tag, torch.full_like(self.tag, step & m32), torch.zeros_like(self.tag), self.sysid.long()]
        k0, k1 = SEED & m32, SEED >> 32
        for _ in range(10):
            h0, l0 = mul(0xD2511F53, c[0])
            h1, l1 = mul(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        return torch.stack([(q >> 8).double() / 8388608.0 - 1.0 for q in c[:3]], 1)

    def turn(self, o):
        g = self.n + torch.linalg.cross(o, self.n) * DT
        return g / torch.linalg.norm(g, dim=1, keepdim=True)

    def langevin(self, steps):
        gam = 6.0 * math.pi * ETA * 0.56125
        sig = math.sqrt(2.0 * self.case["kT"] * gam) * math.sqrt(3.0 / DT)
        for k in range(steps):
            F, T, _ = self.forces()
            self.o = self.o + DT * torch.linalg.cross(self.n, T)
            self.n = self.turn(self.o)
            self.v = self.v + DT * (F - gam * self.v - sig * self.noise(k))
            self.x = self.x + DT * self.v

    def nose_hoover(self, steps):
        count = torch.bincount(self.sysid, minlength=len(self.w["systems"])).double()
        zeta = torch.zeros_like(count)

        def thermostat():
            ke = torch.zeros_like(count).index_add_(0, self.sysid, (self.v * self.v).sum(1))
            return 0.5 * DT / (0.01 * count) * (0.5 * ke - 1.5 * count * self.case["kT"])

        def final():
            F, T, _ = self.forces()
            T = torch.linalg.cross(self.n, T)
            self.v = self.v + 0.5 * DT * (F - zeta[self.sysid][:, None] * self.v)
            self.o = self.o + 0.5 * DT * T
            return F, T

        F, T = final()
        zeta += thermostat()
        for _ in range(steps):
            g = 1.0 / (1.0 + 0.5 * DT * zeta[self.sysid])[:, None]
            self.v = (self.v + 0.5 * DT * F) * g
            self.x = self.x + DT * self.v
            self.o = self.o + 0.5 * DT * T
            self.n = self.turn(self.o)
            zeta += thermostat()
            F, T = final()
            zeta += thermostat()

    def minimize(self, steps):
        for _ in range(steps):
            F, T, _ = self.forces()
            dn = torch.linalg.cross(torch.linalg.cross(self.n, T), self.n)
            a, b = torch.linalg.norm(F, dim=1), torch.linalg.norm(dn, dim=1)
            h = torch.where((a > 0.05) | (b > 0.05), torch.minimum(0.05 / a, 0.05 / b), torch.full_like(a, DT))[:, None]
            self.x = self.x + F * h
            g = self.n + dn * h
            self.n = g / torch.linalg.norm(g, dim=1, keepdim=True)


def exact(case, seed):
    if case["call"] == "rdf" or case["n"] * max(1, case["steps"]) > 1.0e8:
        return None
    ex = _Exact(case, seed)
    if case["call"] == "forces":
        F, T, E = ex.forces()
        return {"f": F.cpu(), "t": T.cpu(), "e": E.cpu()}
    out = {}
    if case["call"] == "minimize":
        ex.minimize(case["steps"])
    elif case["integrator"] == "nose-hoover":
        ex.nose_hoover(case["steps"])
    else:
        ex.langevin(case["steps"])
    if case["call"] == "resident":
        area, vol = ex.mesh() if "faces" in ex.w else (None, None)
        out = {"temperature": float((ex.v ** 2).sum() / (3.0 * len(ex.x))), "area": area, "volume": vol}
    for k in ("x", "n", "v", "o"):
        out[k] = getattr(ex, k).cpu()
    if any(any(d["periodic"]) for d in ex.w["systems"]) and case["system"] == "lattice":
        out["x"] = None  # a lipid at the box's edge comes back on the side where the last sort found it
    return out
