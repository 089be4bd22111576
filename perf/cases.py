"""Performance cases of hemepure_b200: what a user of the framework has it do.

A case is one lattice (or a batch of lattices) driven through the public Python
interface: `LBM` steps and hands back its fields, `Batch` admits, steps and
retires many small lattices.  Geometries are voxelised once into a temporary
folder by `hemepure_b200.vessels` and shared by every case of the same shape;
the initial state (or, for a batch, the iolet conditions) comes from the seed.
`exact` computes the same fields in FP64 with plain torch from its own reading of
the geometry file.
"""

import concurrent.futures as cf
import hashlib
import json
import math
import os
import tempfile

import numpy as np
import torch

from hemepure_b200 import lbm, vessels

CS2 = 1.0 / 3.0
BYTES = {"fp64": 8, "fp32": 4, "fp16": 2}
MEMBER_KINDS = (("pipe", "LBGK", "SBB", "pressure"), ("pipe", "TRT", "BFL", "velocity"),
                ("stenosis", "LBGK", "BFL", "velocity"), ("bifurcation", "TRT", "SBB", "pressure"))


def _single(name, shape, r, length, kernel, wall, precision, tau, inlet, steps, outlet="pressure", drive="run",
            stress=False, state=False):
    c = {"shape": shape, "r": float(r), "length": int(length), "kernel": kernel, "wall": wall, "precision": precision,
         "tau": float(tau), "inlet": inlet, "outlet": outlet, "steps": int(steps), "drive": drive, "stress": stress,
         "state": state}
    return {"name": name, **c} if name else c


def _batch(name, members, r_lo, r_hi, precision, steps):
    c = {"shape": "batch", "members": int(members), "r_lo": float(r_lo), "r_hi": float(r_hi), "precision": precision,
         "steps": int(steps)}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The small rigid pipe of the configurations (13k sites): a parameter scan's
        # single run, where the latency of a step counts.
        _single("small_pipe_fp64", "pipe", 8, 64, "LBGK", "SBB", "fp64", 0.8, "pressure", 500),
        # A host that couples another model step by step: it hands over the iolet
        # densities and advances one step per call.
        _single("coupled_steps_fp64", "pipe", 12.5, 131, "LBGK", "BFL", "fp64", 0.7, "velocity", 200, drive="coupled"),
        # The large straight pipe (4.0M sites), the benchmark workload, in each storage
        # precision: a thousand steps between two outputs of the macroscopic fields.
        _single("large_pipe_fp64", "pipe", 40, 800, "LBGK", "BFL", "fp64", 0.55, "velocity", 1000),
        _single("large_pipe_fp32", "pipe", 40, 800, "LBGK", "BFL", "fp32", 0.55, "velocity", 1000),
        _single("large_pipe_fp16", "pipe", 40, 800, "LBGK", "BFL", "fp16", 0.55, "velocity", 1000),
        # Y-bifurcation with Guo-Zheng-Shi walls and Windkessel outlets, TRT: the
        # configuration's physics at 0.6 and 0.4 of its size.
        _single("bifurcation_fp64", "bifurcation", 19, 240, "TRT", "GZS", "fp64", 0.8, "pressure", 200, outlet="wk3"),
        _single("bifurcation_fp32", "bifurcation", 13, 160, "TRT", "GZS", "fp32", 0.8, "pressure", 300, outlet="wk3"),
        # Stenosed artery with the LES sponge kernel, two sizes and precisions.
        _single("stenosis_les_fp64", "stenosis", 24, 300, "LBGKLESSL", "BFL", "fp64", 0.6, "velocity", 200),
        _single("stenosis_les_fp32", "stenosis", 31, 411, "LBGKLESSL", "BFL", "fp32", 0.6, "velocity", 200),
        # A ragged medium pipe whose distributions are handed back at the end (a
        # checkpoint, or a host that analyses them).
        _single("ragged_state_fp32", "pipe", 17.3, 211, "TRT", "BFL", "fp32", 0.65, "velocity", 300, state=True),
        # Monitoring: short bursts, then the macroscopic fields, stresses and conserved sums.
        _single("monitor_fp64", "pipe", 20, 203, "LBGK", "BFL", "fp64", 0.7, "velocity", 25, stress=True),
        # Serving: eight small vessels of mixed physics prepared on host threads,
        # admitted, stepped together and retired with their fields.
        _batch("serving_batch_fp32", 8, 6, 20, "fp32", 2000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pipe", "pipe", "pipe", "stenosis", "bifurcation", "batch"])
    if kind == "batch":
        lo = rng.uniform(5.0, 9.0)
        return _batch(None, rng.randint(3, 10), lo, lo + rng.uniform(3.0, 11.0), rng.choice(["fp32", "fp32", "fp16"]),
                      200 * rng.randint(4, 10))
    precision = rng.choice(["fp64", "fp64", "fp32", "fp32", "fp16"])
    if kind == "bifurcation":
        r = _log(rng, 7.0, 22.0)
        return _single(None, kind, round(r, 2), int(r * rng.uniform(8.0, 13.0)), rng.choice(["TRT", "LBGK"]),
                       rng.choice(["GZS", "GZS", "BFL", "SBB"]), precision, rng.uniform(0.75, 0.95), "pressure",
                       rng.randint(60, 240), outlet=rng.choice(["wk3", "pressure"]))
    r = _log(rng, 5.5, 38.0)
    length = int(r * _log(rng, 6.0, 19.0))
    if kind == "stenosis":
        r = max(r, 8.0)
        length = max(length, int(8 * r))
        kernel, tau = rng.choice([("LBGKLESSL", 0.6), ("LBGK", 0.7), ("TRT", 0.7)])
        return _single(None, kind, round(r, 2), length, kernel, rng.choice(["BFL", "SBB"]), precision, tau, "velocity",
                       rng.randint(60, 300))
    drive = rng.choice(["run", "run", "run", "coupled"])
    inlet = rng.choice(["velocity", "pressure"])
    return _single(None, kind, round(r, 2), length, rng.choice(["LBGK", "TRT"]), rng.choice(["BFL", "SBB", "BFL", "GZS"]),
                   precision, rng.uniform(0.6 if inlet == "velocity" else 0.75, 0.95), inlet, rng.randint(60, 300), drive=drive,
                   stress=rng.random() < 0.15, state=rng.random() < 0.15)


# -- geometries ----------------------------------------------------------------

def _vessel(shape, r, length):
    if shape == "pipe":
        return vessels.Pipe(r, length)
    if shape == "stenosis":
        return vessels.Stenosis(r, length, 0.6 * r, 3.0 * r)
    return vessels.YBifurcation(r, length, 0.78 * r, length, 35.0)


def _folder(shape, r, length):
    """Folder holding the voxelised geometry and its decoded tables (made once)."""
    key = hashlib.sha256(json.dumps([shape, r, length, 3]).encode()).hexdigest()[:20]
    root = os.path.join(tempfile.gettempdir(), "hemepure_b200_cases")
    path = os.path.join(root, key)
    if not os.path.isdir(path):
        os.makedirs(root, exist_ok=True)
        tmp = tempfile.mkdtemp(dir=root)
        vessels.voxelise(_vessel(shape, r, length), os.path.join(tmp, "vessel.gmy"))
        for name, a in _read_gmy(os.path.join(tmp, "vessel.gmy")).items():
            np.save(os.path.join(tmp, name + ".npy"), a)
        try:
            os.rename(tmp, path)
        except OSError:
            pass
    return path


def _table(path, name):
    return np.load(os.path.join(path, name + ".npy"))


_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, -1, 0),
      (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
_INV = [0] + [i + 1 if i % 2 else i - 1 for i in range(1, 19)]
_W = [1.0 / 3.0] + [1.0 / 18.0] * 6 + [1.0 / 36.0] * 12


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _read_gmy(path):
    """The site tables of a geometry file in the solver's contiguous site order
    (sites binned by collision type, block order within a bin); all blocks are
    walked side by side."""
    import zlib
    raw = open(path, "rb").read()
    pre = np.frombuffer(raw, ">u4", 8)
    nb, bs = [int(v) for v in pre[3:6]], int(pre[6])
    hdr = np.frombuffer(raw, ">u4", 3 * nb[0] * nb[1] * nb[2], 32).reshape(-1, 3).astype(np.int64)
    blocks = np.nonzero(hdr[:, 0])[0]
    off = 32 + 12 * len(hdr) + np.concatenate([[0], np.cumsum(hdr[:, 1])])
    bodies = [zlib.decompress(raw[off[b]:off[b] + hdr[b, 1]]) for b in blocks]
    start = np.concatenate([[0], np.cumsum([len(x) // 4 for x in bodies])])[:-1]
    dev = _device()
    words = torch.from_numpy(np.frombuffer(b"".join(bodies) + bytes(1024), ">u4").astype(np.uint32).view(np.int32)).to(dev)
    cur = torch.from_numpy(start.astype(np.int64)).to(dev)
    B, S = len(blocks), bs ** 3
    fluid = torch.zeros((B, S), dtype=torch.bool, device=dev)
    wall = torch.zeros((B, S), dtype=torch.int32, device=dev)
    iolet, iid = torch.zeros_like(wall), torch.zeros_like(wall)
    kind = torch.zeros((B, S), dtype=torch.int8, device=dev)
    q = torch.zeros((B, S, 18), dtype=torch.float32, device=dev)
    nrm = torch.zeros((B, S, 3), dtype=torch.float32, device=dev)
    order = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) != (0, 0, 0)]
    for s in range(S):
        is_f = words[cur] == 1
        cur = cur + 1
        if not bool(is_f.any()):
            continue
        fluid[:, s] = is_f
        one = is_f.long()
        for c in order:
            ty = words[cur] * one.int()
            w, io = ty == 1, ty > 1
            if c in _C:
                d = _C.index(c) - 1
                nxt = words[cur + 1]
                wall[:, s] |= w.int() << d
                iolet[:, s] |= io.int() << d
                kind[:, s] = torch.where(io, torch.maximum(kind[:, s], (ty == 2).to(torch.int8) * 2 + (ty == 3).to(torch.int8)),
                                         kind[:, s])
                iid[:, s] = torch.where(io, nxt, iid[:, s])
                q[:, s, d] = torch.where(w, nxt.view(torch.float32), q[:, s, d])
            cur = cur + one + w.long() + 2 * io.long()
        has = (words[cur] == 1) & is_f
        for k in range(3):
            nrm[:, s, k] = torch.where(has, words[cur + 1 + k].view(torch.float32), nrm[:, s, k])
        cur = cur + one + 3 * has.long()
    sel = fluid.reshape(-1)
    b, s = torch.nonzero(fluid, as_tuple=True)
    g = torch.from_numpy(blocks).to(dev)[b]
    xyz = torch.stack([g // (nb[1] * nb[2]) * bs + s // (bs * bs), g // nb[2] % nb[1] * bs + s // bs % bs, g % nb[2] * bs + s % bs], 1)
    wall, iolet, iid, kind = (t.reshape(-1)[sel] for t in (wall, iolet, iid, kind))
    q, nrm = q.reshape(-1, 18)[sel], nrm.reshape(-1, 3)[sel]
    nrm = nrm / torch.sqrt((nrm * nrm).sum(1, keepdim=True)).clamp_min(1e-30)
    stype = torch.where(kind == 2, 1, torch.where(kind == 1, 2, 0))  # 0 fluid, 1 inlet, 2 outlet
    ct = torch.where(wall == 0, torch.where(stype == 0, 0, stype + 1), torch.where(stype == 0, 1, stype + 3))
    p = torch.argsort(ct, stable=True)
    out = {"xyz": xyz.to(torch.int32), "wall": wall, "iolet": iolet, "stype": stype, "iid": iid, "q": q, "nrm": nrm}
    return {k: v[p].cpu().numpy() for k, v in out.items()}


# -- case files and initial states ---------------------------------------------

def _conditions(case):
    """(inlet conditions, outlet conditions, wk3 list) in lattice units."""
    v = _vessel(case["shape"], case["r"], case["length"])
    n_out = sum(io.kind == "outlet" for io in v.iolets)
    if case["inlet"] == "velocity":
        inlet = vessels.VelocityBC(case.get("u", 0.01))
    else:
        inlet = vessels.PressureBC(1.0 + case.get("dp", 5e-4), 2e-4, 4000.0)
    outs = []
    for k in range(n_out):
        if case.get("outlet") == "wk3":
            mu, area = (case["tau"] - 0.5) / 3.0, math.pi * v.rd ** 2
            r_par, r_dau = (8.0 * mu * a / (math.pi * b ** 4) for a, b in ((v.lp, v.rp), (v.ld, v.rd)))
            r_tot = CS2 / (CS2 * 5e-4 / (2.0 * r_par + r_dau)) * (0.9 + 0.2 * k)
            rc = math.sqrt(CS2) / area
            outs.append(vessels.WK3BC(r_c=rc, r_p=r_tot - rc, c_p=2e5 / (r_tot - rc), area=area))
        else:
            outs.append(vessels.PressureBC(1.0 - (case.get("dp", 5e-4) if case["inlet"] == "pressure" else 0.0)))
    return v, [inlet], outs


def _sponge(case):
    return {"viscosity_ratio": 10.0, "width": 1.5 * case["r"], "lifetime": 4000} if case["kernel"] == "LBGKLESSL" else None


def _case_file(case, tag, warmup=0):
    """XML case file of a single lattice beside its geometry."""
    path = _folder(case["shape"], case["r"], case["length"])
    v, ins, outs = _conditions(case)
    fd, xml = tempfile.mkstemp(prefix="case_%s_" % tag, suffix=".xml", dir=path)
    os.close(fd)
    vessels.write_case_xml(xml, "vessel.gmy", v, vessels.CaseUnits(tau=case["tau"]), 1000000, ins, outs, warmup=warmup,
                           relaxation_parameter=3.0 / 16.0 if case["kernel"] == "TRT" else None, sponge=_sponge(case))
    return path, xml


def _feq(rho, m):
    """Second-order equilibrium [19, n] of density [n] and momentum [3, n]."""
    c = torch.tensor(_C, dtype=m.dtype, device=m.device)
    w = torch.tensor(_W, dtype=m.dtype, device=m.device)[:, None]
    e = c @ m
    return w * ((rho - 1.5 * (m * m).sum(0) / rho) + (4.5 / rho) * e * e + 3.0 * e)


def _initial(case, xyz, seed):
    """A smooth seeded state near rest [19, n]: what a run meets while its flow develops."""
    g = torch.Generator().manual_seed(int(seed))
    dev = _device()
    x = torch.from_numpy(xyz).to(dev).double().T
    a_u, a_rho = (2e-5, 1e-4) if case["outlet"] == "wk3" else (4e-3, 5e-4)
    fields = []
    for amp in (a_rho, a_u, a_u, a_u):
        v = torch.zeros(x.shape[1], dtype=torch.float64, device=dev)
        for _ in range(3):
            k = (torch.rand(3, generator=g, dtype=torch.float64) * 2 - 1) * 0.25
            ph = float(torch.rand(1, generator=g, dtype=torch.float64)) * 2 * math.pi
            v += amp / 3.0 * torch.sin(k[0].item() * x[0] + k[1].item() * x[1] + k[2].item() * x[2] + ph)
        fields.append(v)
    rho = 1.0 + fields[0]
    return _feq(rho, torch.stack(fields[1:]) * rho)


def _densities(case, seed, k):
    """Iolet densities a coupled host hands over at its k-th step."""
    return 1.0 + 1e-4 * math.sin(0.05 * k + seed % 7), 1.0 - 1e-4 * math.sin(0.03 * k)


def _member(case, k, seed):
    """The k-th lattice of a batch: shapes and sizes from the case, conditions from the seed."""
    shape, kernel, wall, inlet = MEMBER_KINDS[k % len(MEMBER_KINDS)]
    f = k / max(1, case["members"] - 1)
    r = round(case["r_lo"] + f * (case["r_hi"] - case["r_lo"]), 2)
    rng = np.random.default_rng([int(seed), k])
    return {"shape": shape, "r": r, "length": int(r * (10 if shape == "bifurcation" else 18)), "kernel": kernel, "wall": wall,
            "precision": case["precision"], "tau": (0.62 if inlet == "velocity" else 0.75) + 0.2 * f, "inlet": inlet, "outlet": "pressure", "steps": case["steps"],
            "u": float(rng.uniform(0.008, 0.012)), "dp": float(rng.uniform(4e-4, 6e-4))}


# -- the cases -----------------------------------------------------------------

def _prepare_one(case, xml):
    return lbm.PreparedLattice(xml, kernel=case["kernel"], wall=case["wall"], steps=case["steps"])


def prepare(case, seed):
    if case["shape"] == "batch":
        members = [_member(case, k, seed) for k in range(case["members"])]
        files = [_case_file(m, "b%d" % k, warmup=500) for k, m in enumerate(members)]
        wall = [np.nonzero(_table(p, "wall"))[0] for p, _ in files]
        sites = sum(len(_table(p, "stype")) + 64 for p, _ in files)
        general = sum(int(np.count_nonzero(_table(p, "wall") | _table(p, "iolet"))) for p, _ in files)
        batch = lbm.Batch(sites + 1024, 2 * general + 1024, max_lattices=case["members"], precision=case["precision"])
        batch.set_tuning(1, 128, "split")
        return {"case": case, "batch": batch, "members": members, "files": [x for _, x in files], "wall": wall,
                "pool": cf.ThreadPoolExecutor(8)}
    path, xml = _case_file(case, "s")
    sim = lbm.LBM(xml, kernel=case["kernel"], wall=case["wall"], precision=case["precision"])
    os.remove(xml)
    sim.SetFs(_initial(case, _table(path, "xyz"), seed).T.contiguous().cpu().numpy())
    return {"case": case, "sim": sim, "seed": int(seed), "k": 0, "wall": np.nonzero(_table(path, "wall"))[0]}


def run(state):
    case = state["case"]
    if case["shape"] == "batch":
        batch, out = state["batch"], {}
        preps = list(state["pool"].map(_prepare_one, state["members"], state["files"]))
        slots = [batch.add_prepared(p) for p in preps]
        left = set(slots)
        while left:
            left -= set(batch.run(200))
        for k, s in enumerate(slots):
            rho, u, w = batch.macro(s)
            out["m%d" % k] = {"rho": rho, "u": u, "wss": w[state["wall"][k]]}
            batch.remove(s)
        for p in preps:
            p.close()
        return out
    sim, n = state["sim"], case["steps"]
    if case["drive"] == "coupled":
        for j in range(n):
            a, b = _densities(case, state["seed"], state["k"])
            sim.SetIoletDensities([a], [b])
            sim.step(1, macro=(j == n - 1), stress=case["stress"])
            state["k"] += 1
    else:
        sim.step(n, macro=True, stress=case["stress"])
    rho, u, w = sim.GetPropertyCache()
    out = {"rho": rho, "u": u, "wss": w[state["wall"]]}
    if case["stress"]:
        out["shearrate"] = sim.GetStress("shearrate")
        out["traction"] = sim.GetStress("traction")[state["wall"]]
        out["sums"] = sim.moment_sums()
    if case["state"]:
        out["f"] = sim.GetFOld()
    return out


def _shapes(case):
    return [_member(case, k, 0) for k in range(case["members"])] if case["shape"] == "batch" else [case]


def _site_count(c):
    """Sites of a vessel from its analytic volume (no file is made for it)."""
    if c["shape"] == "bifurcation":
        return math.pi * c["length"] * (c["r"] ** 2 + 2 * (0.78 * c["r"]) ** 2)
    return math.pi * c["length"] * c["r"] ** 2 * (1.0 - (0.5 * 3.0 * c["r"] / c["length"] * 0.5 if c["shape"] == "stenosis" else 0.0))


def work(case):
    sites = sum(_site_count(c) for c in _shapes(case))
    # Each step reads and writes the 19 distributions of every site once; the
    # collision takes about 250 operations a site.
    nbytes = case["steps"] * sites * 38 * BYTES[case["precision"]] + sites * 40
    if case.get("state"):
        nbytes += sites * 152
    if case.get("stress"):
        nbytes += sites * 40
    return {"bytes": nbytes, "flops": case["steps"] * sites * 250}


def tolerance(case):
    # About four times the largest error of any output against `exact`: the wall shear
    # stress (a root of a cancelling difference) in FP64, the traction (which holds
    # rho - 1) in FP32, the wall shear stress in FP16.
    return {"fp64": {"rel": 1e-7, "max": 1e-5}, "fp32": {"rel": 3e-4, "max": 3e-2}, "fp16": {"rel": 5e-3, "max": 0.3}}[case["precision"]]


# -- the same in FP64 with plain torch -------------------------------------------

def _closest(n):
    c = np.array(_C, dtype=np.float64)
    c[1:] /= np.linalg.norm(c[1:], axis=1, keepdims=True)
    return int(np.argmin(((c - np.asarray(n)) ** 2).sum(1)))


class _Lattice:
    """One lattice stepped in FP64: collision, then every slot filled by its streaming rule."""

    def __init__(self, case, warmup=0):
        path = _folder(case["shape"], case["r"], case["length"])
        T = {k: _table(path, k) for k in ("xyz", "wall", "iolet", "stype", "iid", "q", "nrm")}
        self.case, self.warmup, self.t = case, warmup, 1
        vessel, ins, outs = _conditions(case)
        self.dev = dev = _device()
        n = self.n = len(T["xyz"])
        xyz = torch.from_numpy(T["xyz"]).to(dev).long()
        wall, iolet = (torch.from_numpy(T[k]).to(dev) for k in ("wall", "iolet"))
        stype, iid = (torch.from_numpy(T[k]).to(dev).long() for k in ("stype", "iid"))
        q = torch.from_numpy(T["q"]).to(dev)
        self.wall_sites = torch.nonzero(wall)[:, 0]
        self.nrm = torch.from_numpy(T["nrm"]).to(dev).double().T
        dims = (xyz.max(0).values + 3).tolist()
        flat = ((xyz[:, 0] + 1) * dims[1] + xyz[:, 1] + 1) * dims[2] + xyz[:, 2] + 1
        grid = torch.full((dims[0] * dims[1] * dims[2],), -1, dtype=torch.int32, device=dev)
        grid[flat] = torch.arange(n, dtype=torch.int32, device=dev)
        site = torch.arange(n, device=dev)
        self.src = torch.empty((19, n), dtype=torch.int64, device=dev)
        self.src[0] = site
        rows = {"bfl": [], "io": [], "gzs": []}
        for i in range(1, 19):
            d, c = _INV[i], _C[_INV[i]]
            bw, bi = (wall >> (d - 1)) & 1 == 1, (iolet >> (d - 1)) & 1 == 1
            nb = grid[flat + (c[0] * dims[1] + c[1]) * dims[2] + c[2]].long()
            self.src[i] = torch.where(bw | bi, d * n + site, i * n + nb)
            behind = torch.where(((wall >> (i - 1)) & 1 == 1), 1, torch.where((iolet >> (i - 1)) & 1 == 1, 2, 0))
            x = torch.nonzero(bi)[:, 0]
            rows["io"].append(torch.stack([x, torch.full_like(x, d), torch.where(stype[x] == 1, 0, 16) + iid[x]]))
            x = torch.nonzero(bw)[:, 0]
            if case["wall"] == "BFL":
                x = x[behind[x] != 1]
                rows["bfl"].append((torch.stack([x, torch.full_like(x, d)]), q[x, d - 1].double()))
            elif case["wall"] == "GZS":
                qq, bh = q[x, d - 1].double(), behind[x]
                gio = torch.where(bh == 2, torch.where(stype[x] == 1, 0, 16) + iid[x], -1)
                ci = _C[i]
                far = grid[flat[x] + (ci[0] * dims[1] + ci[1]) * dims[2] + ci[2]].long()
                rows["gzs"].append((torch.stack([x, torch.full_like(x, d), bh, far, gio]), qq))
        self.io = torch.cat(rows["io"], 1)
        cat = lambda k: (torch.cat([a for a, _ in rows[k]], 1), torch.cat([b for _, b in rows[k]])) if rows[k] else None  # noqa: E731
        self.bfl, self.gzs = cat("bfl"), cat("gzs")
        self.c = torch.tensor(_C, dtype=torch.float64, device=dev)
        self.w = torch.tensor(_W, dtype=torch.float64, device=dev)[:, None]
        self.inv = torch.tensor(_INV, device=dev)
        lam = 3.0 / 16.0
        self.om, self.om_minus = -1.0 / case["tau"], -1.0 / (0.5 + lam / (case["tau"] - 0.5))
        # Iolet links: the Ladd profile factor, or the Nash normal (kept in float).
        self.kinds, self.dens, self.wk = {}, torch.ones(32, dtype=torch.float64, device=dev), {}
        ios = [io for g in ("inlet", "outlet") for io in vessel.iolets if io.kind == g]
        ids = list(range(len(ins))) + [16 + k for k in range(len(outs))]
        nrm = torch.zeros((32, 3), dtype=torch.float64, device=dev)
        pos = torch.zeros((32, 3), dtype=torch.float64, device=dev)
        rad = torch.ones(32, dtype=torch.float64, device=dev)
        for idx, io, bc in zip(ids, ios, list(ins) + list(outs)):
            unit = io.normal / np.linalg.norm(io.normal)
            nrm[idx], pos[idx] = torch.from_numpy(unit).to(dev), torch.from_numpy(np.asarray(io.position)).to(dev)
            rad[idx] = io.radius
            self.kinds[idx] = bc
            if isinstance(bc, vessels.WK3BC):
                dir0 = _closest(unit)
                sel = (self.io[2] == idx) & (self.inv[self.io[1]] == dir0)
                x = torch.sort(self.io[0][sel]).values
                box = ((xyz.double() - pos[idx]).abs() <= 1.0).all(1)
                centre = int(torch.nonzero(box)[0, 0]) if bool(box.any()) else -1
                self.wk[idx] = {"x": x, "n": nrm[idx], "bc": bc, "new": 1.0, "old": 0.0, "flow": None,
                                "couples": bool((x == centre).any())}
        x, d, idx = self.io
        self.ladd = torch.zeros(len(x), dtype=torch.bool, device=dev)
        for k, bc in self.kinds.items():
            if isinstance(bc, vessels.VelocityBC):
                self.ladd |= idx == k
        half = xyz[x].double() + 0.5 * self.c[d] - pos[idx]
        z = (half * nrm[idx]).sum(1)
        self.profile = 1.0 - ((half * half).sum(1) - z * z) / rad[idx] ** 2
        self.rho_min = min(bc.mean_rho - bc.amp_rho if isinstance(bc, vessels.PressureBC) else 1.0 for bc in self.kinds.values())
        self.u_max = max([bc.u_max for bc in ins if isinstance(bc, vessels.VelocityBC)] or [0.0])
        self.ladd_c = (nrm[idx] * self.c[d]).sum(1)
        self.nash_n = nrm.float().double()[idx]
        self.prof_n = nrm
        self.prof = (pos, rad)
        self.xyz = xyz.double()
        self.vtau = None
        sponge = _sponge(case)
        if sponge:
            vr = torch.ones(n, dtype=torch.float64, device=dev)
            for k in range(len(outs)):
                o = torch.tensor([int(v) for v in ios[len(ins) + k].position], device=dev)
                dist = ((xyz - o) ** 2).sum(1).double().sqrt()
                fac = 1.0 + (sponge["viscosity_ratio"] - 1.0) * (dist / sponge["width"] - 1.0) ** 2
                vr = torch.where(dist <= sponge["width"], vr * fac, vr)
            self.vtau, self.lifetime = vr * (case["tau"] - 0.5) + 0.5, sponge["lifetime"]

    def _iolet_densities(self, override):
        t0 = self.t - 1
        for idx, bc in self.kinds.items():
            if isinstance(bc, vessels.PressureBC):
                v = bc.mean_rho + bc.amp_rho * math.cos(2.0 * math.pi / bc.period_steps * t0 + bc.phase)
                if t0 < self.warmup:
                    v = v * t0 / self.warmup + (1.0 - t0 / self.warmup) * self.rho_min
                self.dens[idx] = v
                if override is not None:
                    self.dens[idx] = override[0] if idx < 16 else override[1]
        for idx, k in self.wk.items():
            flow = 0.0 if k["flow"] is None else float(k["flow"]) * k["bc"].area / len(k["x"])
            rho, bc = k["new"], k["bc"]
            self.dens[idx] = rho
            if k["couples"]:
                p = rho * CS2
                pn = (bc.r_p * bc.c_p * p + (bc.r_c + bc.r_p) * (2.0 * flow - k["old"])
                      + bc.r_c * bc.r_p * bc.c_p * (flow - k["old"])) / (1.0 + bc.r_p * bc.c_p)
                k["new"], k["old"] = pn / CS2, flow

    def _relax(self, f, fneq, om):
        if self.case["kernel"] != "TRT":
            return f + fneq * om
        opp = fneq[self.inv]
        return f + 0.5 * self.om * (fneq + opp) + 0.5 * self.om_minus * (fneq - opp)

    def _ramp(self):
        return self.u_max * (self.t / self.warmup if self.t < self.warmup else 1.0)

    def step(self, f, override=None, last=False):
        case, n = self.case, self.n
        self._iolet_densities(override)
        rho, m = f.sum(0), self.c.T @ f
        feq = _feq(rho, m)
        fneq = f - feq
        tau, om = case["tau"], self.om
        if self.vtau is not None:
            q12 = torch.zeros(n, dtype=torch.float64, device=self.dev)
            for a in range(3):
                for b in range(3):
                    q12 += ((self.c[:, a] * self.c[:, b])[None] @ fneq)[0] ** 2
            les = 0.5 * (tau + torch.sqrt(tau * tau + 18.0 * math.sqrt(2.0) * 0.01 * q12.sqrt()))
            if self.t <= self.lifetime // 2:
                tau = torch.where(self.vtau == case["tau"], les, self.vtau)
            elif self.t < self.lifetime:
                tau = (les - self.vtau) * 2.0 / self.lifetime * self.t + (2.0 * self.vtau - les)
            else:
                tau = les
            om = -1.0 / tau
        post = self._relax(f, fneq, om)
        u = m / rho
        new = post.reshape(-1)[self.src.reshape(-1)].reshape(19, n)
        x, d, idx = self.io
        i = self.inv[d]
        rb = self.dens[idx]
        comp = (u[:, x] * self.nash_n.T).sum(0)
        mg = self.nash_n.T * comp * rb
        e = (self.c[i] * mg.T).sum(1)
        w = self.w[i, 0]
        nash = w * ((rb - 1.5 * (mg * mg).sum(0) / rb) + 4.5 / rb * e * e + 3.0 * e)
        ladd = post[d, x] - 2.0 * w * (self._ramp() * self.profile * self.ladd_c * rho[x]) / CS2
        new[i, x] = torch.where(self.ladd, ladd, nash)
        if self.bfl is not None:
            (x, d), q = self.bfl
            i = self.inv[d]
            far = (post[d, x] + (2.0 * q - 1.0) * post[i, x]) / (2.0 * q)
            near = 2.0 * q * post[d, x] + (1.0 - 2.0 * q) * new[d, x]
            new[i, x] = torch.where(q < 0.5, near, far)
        if self.gzs is not None:
            (x, d, behind, far, gio), q = self.gzs
            i = self.inv[d]
            near = q < 0.75
            vel = torch.zeros_like(near)
            for k, bc in self.kinds.items():
                if isinstance(bc, vessels.VelocityBC):
                    vel |= gio == k
            ok = near & (behind == 0)
            far = torch.where(ok, far, x)
            io = gio.clamp_min(0)
            p = self.xyz[x] + self.c[i] - self.prof[0][io]
            z = (p * self.prof_n[io]).sum(1)
            speed = self._ramp() * (1.0 - ((p * p).sum(1) - z * z) / self.prof[1][io] ** 2)
            vn = torch.where(ok, u[:, far], self.prof_n[io].T * speed)
            r, mw = rho[x], m[:, x] * (1.0 - 1.0 / q)
            use = ok | (near & vel)
            mw = torch.where(use, q * mw + (1.0 - q) * r * (vn * (q - 1.0) / (q + 1.0)), mw)
            fi = torch.where(ok, q * fneq[i, x] + (1.0 - q) * fneq[i, far], fneq[i, x])
            fd = torch.where(ok, q * fneq[d, x] + (1.0 - q) * fneq[d, far], fneq[d, x])
            e = (self.c[i] * mw.T).sum(1)
            v = self.w[i, 0] * ((r - 1.5 * (mw * mw).sum(0) / r) + 4.5 / r * e * e + 3.0 * e) + fi
            if case["kernel"] == "TRT":
                v = v + 0.5 * self.om * (fi + fd) + 0.5 * self.om_minus * (fi - fd)
            else:
                v = v + fi * self.om
            bounce = near & ~use
            new[i, x] = torch.where(bounce, post[d, x], v)
        for k in self.wk.values():
            k["flow"] = -(u[:, k["x"]] * k["n"][:, None]).sum()
        self.t += 1
        if not last:
            return new, None
        c, dev = self.c, post - f
        tt = tau if torch.is_tensor(tau) else torch.full((n,), tau, dtype=torch.float64, device=self.dev)
        pi = torch.stack([torch.stack([((c[:, a] * c[:, b])[None] @ dev)[0] for b in range(3)]) for a in range(3)]) * -(tt - 0.5)
        ws = self.wall_sites
        nr = self.nrm[:, ws]
        s = (pi[:, :, ws] * nr[None]).sum(1)
        wss = torch.sqrt(((s * s).sum(0) - (s * nr).sum(0) ** 2).clamp_min(0.0))
        out = {"rho": rho.cpu().numpy(), "u": u.T.contiguous().cpu().numpy(), "wss": wss.cpu().numpy()}
        if case.get("stress"):
            out["shearrate"] = (torch.sqrt((pi * pi).sum((0, 1))) / (-2.0 * CS2 * rho) / (tt - 0.5))[:, None].cpu().numpy()
            st = -pi[:, :, ws] - torch.eye(3, dtype=torch.float64, device=self.dev)[:, :, None] * (rho[ws] - 1.0) * CS2
            out["traction"] = (st * nr[None]).sum(1).T.contiguous().cpu().numpy()
            out["sums"] = np.concatenate([[float(new.sum())], (self.c.T @ new).sum(1).cpu().numpy()])
        if case.get("state"):
            out["f"] = new.T.contiguous().cpu().numpy()
        return new, out


def exact(case, seed):
    if case["shape"] == "batch":
        if case["members"] * case["steps"] > 20000:
            return None
        out = {}
        for k in range(case["members"]):
            m = _member(case, k, seed)
            lat = _Lattice(m, warmup=500)
            f = _feq(torch.ones(lat.n, dtype=torch.float64, device=lat.dev), torch.zeros((3, lat.n), dtype=torch.float64, device=lat.dev))
            for j in range(m["steps"]):
                f, res = lat.step(f, last=j == m["steps"] - 1)
            out["m%d" % k] = res
        return out
    lat = _Lattice(case)
    f = _initial(case, _table(_folder(case["shape"], case["r"], case["length"]), "xyz"), seed)
    res = None
    for j in range(case["steps"]):
        over = _densities(case, int(seed), j) if case["drive"] == "coupled" else None
        f, res = lat.step(f, over, last=j == case["steps"] - 1)
    return res
