"""Performance cases of the pose scorer, its GSO driver and its surrogate.

A case is one call (or one short sequence of calls) that a docking program
makes; ``run`` makes it through the package's public entry points.

* Receptors: a ball of jittered lattice points, 2,000 to 101,000 atoms, either
  at the benchmark's random-chain density (0.0155 atoms / A^3) or at a
  protein's density with hydrogens (0.09).  AMBER well depths and radii,
  charges U[-0.8, 0.8] shifted to a net +10, as in ``synth.globule``.
* Ligands: a B-DNA-like cylinder (62 atoms a base pair, 3.38 A rise, charge -1
  on each phosphorus, 0 elsewhere: ``synth.duplex``), or for the large cpydock
  complex, whose receptor is eight balls at the corners of a cube, another
  ball with every atom charged (``synth.config4``).
* Poses: swarms of glowworms around points at the setup's distance from the
  receptor's centre, +-1 A, random quaternions (``synth.setup_poses``).

``exact`` restates the scoring formulas in 64-bit torch.
"""
import importlib
import math

import numpy as np
import torch

lkg = importlib.import_module("lklight-gpu_b200")
compat = importlib.import_module("lklight-gpu_b200.compat")

CHAIN, PROTEIN = 0.0155, 0.09   # atoms / A^3
FLAGS = {"dna": 7, "pydock": 3, "vdw": 0}


def _case(path, family, n_rec, n_lig, n_pose, density=CHAIN, precision="fast", complexes=1, ball=False):
    return dict(path=path, family=family, n_rec=n_rec, n_lig=n_lig, n_pose=n_pose, density=density,
                precision=precision, complexes=complexes, ball=ball)


def listed():
    return [
        # Score::energy for a single pose (rescoring, a minimiser's inner loop): the smallest call, all latency
        dict(_case("energy", "dna", 12625, 1240, 1), name="energy_one_pose"),
        # one swarm's step of a docking run as the reference calls its scorer: 200 glowworms, host buffers
        dict(_case("score", "dna", 12625, 1240, 200), name="swarm_dna_200"),
        # the same on a small protein-protein-sized complex at a protein's density, where pairs dominate; ragged sizes
        dict(_case("score", "pydock", 4999, 811, 301, density=PROTEIN), name="swarm_protein_301"),
        # six swarms of 300 in one call, van der Waals only (no far field, no charges)
        dict(_case("score", "vdw", 12625, 1240, 1800), name="swarms_vdw_1800"),
        # a reference program linked against the compatible C symbols: one swarm of 300 a call
        dict(_case("compat", "pydock", 9973, 1301, 300), name="compat_pydock_300"),
        # the f64 parity mode on one swarm (rescoring final poses, checks against the CPU path)
        dict(_case("score", "dna", 12625, 1240, 200, precision="exact"), name="exact_dna_200"),
        # cpydock with its desolvation minima: six swarms of 300
        dict(_case("score", "cpydock", 12625, 1240, 1800), name="cpydock_1800"),
        # a large assembly: every ligand atom charged, far field larger than L2, 50 swarms of 500 on device buffers
        dict(_case("device", "cpydock", 101000, 12000, 25000, ball=True), name="cpydock_assembly"),
        # many complexes in one launch group, host buffers, half dna and half pydock: the batch screening workload
        dict(_case("multi", "mixed", 40000, 5000, 2000, complexes=16), name="batch_16_complexes"),
        # restraints and a membrane collected in the batch kernels
        dict(_case("restraints", "dna", 12625, 1240, 3000), name="restraints_3000"),
        # a short GSO run on the device from creation to read-back: n_pose glowworms in swarms of 200, ten steps
        dict(_case("gso", "dna", 12625, 1240, 2000), name="gso_ten_swarms"),
        # the surrogate: two epochs over n_pose scored poses, then a prediction of four times as many
        dict(_case("surrogate", "dna", 12625, 1240, 8192), name="surrogate_fit_predict"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["energy", "score", "score", "score", "compat", "device", "device", "multi", "restraints", "gso",
                       "surrogate"])
    family = rng.choice(["dna", "pydock", "vdw", "cpydock"])
    dense = rng.random() < 0.4
    n_rec, n_lig = _log(rng, 2000, 12000 if dense else 40000), _log(rng, 300, 2000 if dense else 5000)
    n_pose = _log(rng, 20, 6000)
    precision = "exact" if path == "score" and rng.random() < 0.25 else "fast"
    complexes = 1
    if path == "energy":
        n_pose = 1
    if path == "compat" and family == "cpydock":
        family = "pydock"   # its desolvation is another symbol
    if path == "multi":
        family, complexes, n_pose = "mixed", rng.randint(3, 12), _log(rng, 100, 2000)
    if path == "gso":
        family, n_pose = rng.choice(["dna", "pydock"]), 200 * rng.randint(1, 10)
    if path == "surrogate":
        family, n_pose = rng.choice(["dna", "pydock"]), _log(rng, 2000, 8192)
    if path == "restraints" and family == "vdw":
        family = "dna"
    if precision == "exact":
        n_pose = min(n_pose, 600)
    if family == "cpydock":
        n_pose = min(n_pose, 2000)
    return _case(path, family, n_rec, n_lig, n_pose, PROTEIN if dense else CHAIN, precision, complexes)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
# AMBER (well depth, radius, is hydrogen): H, HC, HA, C, CT, N, O, OH, P
_TYPES = [(0.0157, 0.6, 1), (0.0157, 1.487, 1), (0.015, 1.459, 1), (0.086, 1.908, 0), (0.1094, 1.908, 0),
          (0.17, 1.824, 0), (0.21, 1.6612, 0), (0.2104, 1.721, 0), (0.2, 2.1, 0)]


def _params(rng, n):
    t = np.array(_TYPES)[rng.integers(0, len(_TYPES), n)]
    return dict(vdw=t[:, 0].copy(), radius=t[:, 1].copy(), heavy=(1 - t[:, 2]).astype(np.uint8))


def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _ball(rng, n, density, net):
    a = density ** (-1.0 / 3.0)
    r = (3.0 * n / (4.0 * math.pi * density)) ** (1.0 / 3.0)
    m = int(math.ceil(r / a)) + 2
    g = np.arange(-m, m + 1)
    p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).astype(float) * a
    keep = np.argsort((p * p).sum(1), kind="stable")[:n]
    p = p[rng.permutation(keep)] + rng.uniform(-0.12 * a, 0.12 * a, (n, 3))
    q = rng.uniform(-0.8, 0.8, n)
    if net is not None:
        q += (net - q.sum()) / n
    return dict(coords=_f32(p - p.mean(0)), ele=q, **_params(rng, n))


def _assembly(rng, n, density):
    """Eight balls at the corners of a cube, just apart."""
    parts = [_ball(rng, n // 8 + (k < n % 8), density, 10.0) for k in range(8)]
    r = 1.18 * max(float(np.sqrt((m["coords"] ** 2).sum(1)).max()) for m in parts)
    for k, m in enumerate(parts):
        m["coords"] = _f32(m["coords"] + r * np.array([(k & 1) * 2 - 1, ((k >> 1) & 1) * 2 - 1, (k >> 2) * 2 - 1]))
    return {key: np.concatenate([m[key] for m in parts]) for key in parts[0]}


def _duplex(rng, n):
    k = np.arange(n)
    bp, shell = k // 62, rng.integers(0, 3, n)
    r = np.where(shell == 0, 9.4, np.where(shell == 1, rng.uniform(5.8, 8.2, n), rng.uniform(0.6, 5.4, n)))
    ph = bp * math.radians(36.0) + rng.integers(0, 2, n) * math.pi + rng.uniform(-0.4, 0.6, n)
    z = bp * 3.38 + rng.uniform(-1.2, 1.2, n)
    p = np.stack([r * np.cos(ph), r * np.sin(ph), z], 1) + rng.uniform(-0.2, 0.2, (n, 3))
    m = dict(coords=_f32(p - p.mean(0)), **_params(rng, n))
    phos = k % 31 == 0
    m["ele"] = np.where(phos, -1.0, 0.0)
    m["vdw"][phos], m["radius"][phos], m["heavy"][phos] = 0.2, 2.1, 1
    return m


def _desolvation(rng, m):
    n, heavy = len(m["ele"]), m["heavy"].astype(bool)
    des = np.where(heavy, rng.choice([0.01918, 0.1108, -0.0391, -0.12604, -0.03128, -0.06877, -0.04255], n), 0.0)
    m.update(hyd=heavy.astype(np.int32), des=des, asa=np.where(heavy, rng.uniform(0.0, 70.0, n), -1.0))
    return m


def _sizes(case):
    """(receptor atoms, ligand atoms, family) of each complex of a case."""
    if case["path"] != "multi":
        return [(case["n_rec"], case["n_lig"], case["family"])]
    n = case["complexes"]
    f = [(k + 0.5) / n for k in range(n)]
    return [(int(2000 * (case["n_rec"] / 2000) ** f[k]), int(300 * (case["n_lig"] / 300) ** f[(5 * k + 3) % n]),
             "dna" if k < n // 2 else "pydock") for k in range(n)]


def _complexes(case, seed):
    out = []
    for k, (nr, nl, fam) in enumerate(_sizes(case)):
        rng = np.random.default_rng([seed, k])
        rec = _assembly(rng, nr, case["density"]) if case["ball"] else _ball(rng, nr, case["density"], 10.0)
        lig = _ball(rng, nl, case["density"], None) if case["ball"] else _duplex(rng, nl)
        if fam == "cpydock":
            rec, lig = _desolvation(rng, rec), _desolvation(rng, lig)
        out.append((fam, rec, lig))
    return out


def _poses(rng, rec, n, swarm, cap):
    """n x 7 (w, x, y, z, tx, ty, tz): swarms around points at the mean atom distance + 3 A (cap: within 18 degrees
    of an axis of the assembly's cube, as the first swarms of a setup sphere are)."""
    avg = float(np.sqrt((rec["coords"] ** 2).sum(1)).mean()) + 3.0
    c = rng.normal(size=((n + swarm - 1) // swarm, 3))
    if cap:
        c = 0.3 * c / np.linalg.norm(c, axis=1, keepdims=True) + np.eye(3)[rng.integers(0, 3, len(c))]
    c *= avg / np.linalg.norm(c, axis=1, keepdims=True)
    t = np.repeat(c, swarm, 0)[:n] + rng.uniform(-1.0, 1.0, (n, 3))
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    return np.round(np.hstack([q, t]), 6)


def _all_poses(case, seed, cx, factor=1):
    swarm = {"gso": 200, "device": 500}.get(case["path"], 300)
    return [_poses(np.random.default_rng([seed, k, 1]), rec, factor * case["n_pose"], swarm, case["ball"])
            for k, (_, rec, _) in enumerate(cx)]


def _restraints(case, seed, rec, poses):
    """Restraint residues (blocks of 10 receptor / 30 ligand atoms) and membrane beads near the swarms."""
    rng = np.random.default_rng([seed, 2])
    nr, nl = case["n_rec"], case["n_lig"]
    near = np.zeros(nr, bool)
    for c in poses[::300, 4:7]:
        near |= ((rec["coords"] - c) ** 2).sum(1) < 400.0
    idx = np.nonzero(near)[0]
    rres, lres = np.arange(nr) // 10, np.arange(nl) // 30
    ra = rng.choice(np.unique(rres[idx]), min(20, len(np.unique(rres[idx]))), replace=False)
    la = rng.choice(lres.max() + 1, min(6, lres.max() + 1), replace=False)
    lut_r, lut_l = np.full(rres.max() + 1, -1), np.full(lres.max() + 1, -1)
    lut_r[ra], lut_l[la] = np.arange(len(ra)), np.arange(len(la))
    mem = np.sort(rng.choice(idx, min(300, len(idx)), replace=False))
    return lut_r[rres].astype(np.int32), lut_l[lres].astype(np.int32), mem.astype(np.int32)


# ---------------------------------------------------------------------------
# what a program holds, and its call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    path = case["path"]
    cx = _complexes(case, seed)
    poses = _all_poses(case, seed, cx, 5 if path == "surrogate" else 1)
    fam, rec, lig = cx[0]
    s = dict(path=path)
    if path == "compat":
        lkg.lib().lkg_compat_cache_clear()   # its device copies are keyed on the host arrays of the last complex
        s["field"] = lkg.field_build(rec["coords"], rec["ele"]) if FLAGS[fam] & 1 else None
        s["rec"] = compat.CudaReceptor(rec["coords"], rec["ele"], np.sqrt(rec["vdw"]), rec["radius"], rec["heavy"])
        s["lig"] = compat.CudaLigand(lig["coords"], lig["ele"], np.sqrt(lig["vdw"]), lig["radius"], lig["heavy"])
        s["poses"], s["flags"] = poses[0], FLAGS[fam]
        return s
    if path in ("energy", "score"):
        s["scorer"] = lkg.Scorer(fam, rec, lig, precision=case["precision"])
        s["t"], s["q"] = poses[0][:, 4:7].copy(), poses[0][:, 0:4].copy()
        return s
    # the large batches run with the shapes the autotuner picks for them
    tuned = dict(tile=256, group=16, cell=7.0) if path == "multi" else dict(tile=128, group=16, cell=8.0)
    ctx = s["ctx"] = lkg.Context(**(tuned if path in ("multi", "device") else {}))
    s["ids"] = [ctx.add_complex(f, r, l) for f, r, l in cx]
    if path == "multi":
        s["counts"] = [len(p) for p in poses]
        s["poses"] = torch.from_numpy(np.vstack(poses)).pin_memory()
        s["scores"] = torch.empty(sum(s["counts"]), dtype=torch.float64).pin_memory()
    elif path == "device":
        s["poses"] = torch.from_numpy(poses[0]).cuda()
        s["scores"] = torch.empty(len(poses[0]), dtype=torch.float64, device="cuda")
        s["plan"] = ctx.plan(s["ids"], [len(poses[0])])
    elif path == "restraints":
        ctx.set_restraints(s["ids"][0], *_restraints(case, seed, rec, poses[0]))
        s["poses"] = poses[0]
    elif path == "gso":
        s["groups"] = [(s["ids"][0], case["n_pose"] // 200, 200)]
        s["positions"] = np.hstack([poses[0][:, 4:7], poses[0][:, 0:4]])
    else:   # surrogate
        n = case["n_pose"]
        known = ctx.score(s["ids"][0], poses[0][:n])
        s["sur"] = lkg.Surrogate(ctx, s["ids"][0], seed=seed)
        s["sur"].set_target_scale(known)
        s["poses"], s["known"] = torch.from_numpy(poses[0]).cuda(), torch.from_numpy(known).cuda()
        s["pred"] = torch.empty(4 * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()   # the context's stream is not torch's
    return s


def run(s):
    path = s["path"]
    if path == "energy":
        return s["scorer"].energy(s["t"][0], s["q"][0])
    if path == "score":
        return s["scorer"].batch_energy(s["t"], s["q"])
    if path == "compat":
        return compat.batch_raw(s["field"], s["rec"], s["lig"], s["poses"], s["flags"])
    if path == "multi":
        return s["ctx"].score_multi(s["ids"], s["counts"], s["poses"], s["scores"])
    if path == "device":
        s["plan"].launch(s["poses"].data_ptr(), s["scores"].data_ptr())
        return s["scores"]
    if path == "restraints":
        return s["ctx"].score_interface(s["ids"][0], s["poses"])
    if path == "gso":
        g = lkg.GSO(s["ctx"], s["groups"], s["positions"], [42])
        g.run(10, device=True)
        return g.state()
    n = len(s["known"])
    loss = s["sur"].train_device(n, s["poses"].data_ptr(), s["known"].data_ptr(), epochs=2, batch=1024)
    s["sur"].predict_device(4 * n, s["poses"][n:].data_ptr(), s["pred"].data_ptr())
    return dict(loss=loss, params=s["sur"].params(), pred=s["pred"])


def work(case):
    """The poses and atoms in, the results out; the near pairs' arithmetic
    (about 24 operations a pair; half of a ligand atom's 10 A sphere holds
    receptor for a duplex at the surface, a twelfth for the assembly's ball), the
    surrogate's products where there is one."""
    n_pose, nbytes, flops = case["n_pose"], 0, 0
    steps = 10 if case["path"] == "gso" else 1
    for nr, nl, fam in _sizes(case):
        nbytes += 40 * (nr + nl) + n_pose * 64
        if case["path"] != "surrogate":
            pairs = n_pose * nl * case["density"] * 4189.0 * (1.0 / 12.0 if case["ball"] else 0.5)
            flops += steps * 24 * pairs
    if case["path"] == "surrogate":
        weights = 64 * 256 + 2 * 256 * 256 + 256
        flops = 2 * weights * n_pose * (2 * 3 + 4)
        nbytes += n_pose * 4 * 64 + 4 * weights * 2
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
_CAP = 4.0 / 332.0


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _rotate(p, x):
    """p: n x 7 poses, x: m x 3 -> n x m x 3 (no normalisation)."""
    w, i, j, k = (p[:, a] for a in range(4))
    m = torch.stack([1 - 2 * (j * j + k * k), 2 * (i * j - w * k), 2 * (i * k + w * j),
                     2 * (i * j + w * k), 1 - 2 * (i * i + k * k), 2 * (j * k - w * i),
                     2 * (i * k - w * j), 2 * (j * k + w * i), 1 - 2 * (i * i + j * j)], 1).reshape(-1, 3, 3)
    return torch.einsum("nab,mb->nma", m, x) + p[:, None, 4:7]


def _phi(points, rc, rq):
    """sum of q / d^2 over receptor atoms with 10 < d <= 30 at each point."""
    out = torch.zeros(len(points), dtype=torch.float64, device=points.device)
    step = max(1, (1 << 26) // max(1, len(rc)))
    for a in range(0, len(points), step):
        x = points[a:a + step]
        d2 = (x[:, None, 0] - rc[None, :, 0]) ** 2
        d2 += (x[:, None, 1] - rc[None, :, 1]) ** 2
        d2 += (x[:, None, 2] - rc[None, :, 2]) ** 2
        out[a:a + step] = torch.where((d2 > 100.0) & (d2 <= 900.0), rq / d2, 0.0).sum(1)
    return out


def _far(x, q, rc, rq):
    """q phi(x), phi interpolated trilinearly from its 0.5 A grid; x: n x 3."""
    lo = torch.floor(rc.min(0).values - 31.0)
    dims = ((torch.ceil(rc.max(0).values + 31.0) - lo) / 0.5).long() + 1
    f = (x - lo) / 0.5
    i = torch.floor(f)
    ok = ((i >= 0) & (i + 1 < dims)).all(1)
    t, i, q = (f - i)[ok], i[ok].long(), q[ok]
    corner = torch.stack([i + torch.tensor([b & 1, (b >> 1) & 1, b >> 2], device=x.device) for b in range(8)], 1)
    flat = (corner[..., 2] * dims[1] + corner[..., 1]) * dims[0] + corner[..., 0]
    uniq, inv = torch.unique(flat, return_inverse=True)
    g = torch.stack([uniq % dims[0], (uniq // dims[0]) % dims[1], uniq // (dims[0] * dims[1])], 1)
    phi = _phi(lo + 0.5 * g.double(), rc, rq)[inv]
    w = torch.stack([(t[:, 0] if b & 1 else 1 - t[:, 0]) * (t[:, 1] if b & 2 else 1 - t[:, 1])
                     * (t[:, 2] if b & 4 else 1 - t[:, 2]) for b in range(8)], 1)
    out = torch.zeros(len(x), dtype=torch.float64, device=x.device)
    out[ok] = q * (w * phi).sum(1)
    return out


def _excluded(hyd):
    e = np.zeros(len(hyd), bool)
    e[0::2] = np.asarray(hyd)[:(len(hyd) + 1) // 2] != 0
    return e


def _score64(fam, rec, lig, poses, tags=None):
    """(raw electrostatics, LJ + clash, desolvation, interface counts) of every pose."""
    dev = _dev()
    T = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    rc, lc, P = T(rec["coords"]), T(lig["coords"]), T(poses)
    rq, lq = T(rec["ele"]), T(lig["ele"])
    re, le, rr, lr = T(rec["vdw"]), T(lig["vdw"]), T(rec["radius"]), T(lig["radius"])
    rh, lh = T(rec["heavy"]) != 0, T(lig["heavy"]) != 0
    n, nr, nl = len(P), len(rc), len(lc)
    elec, vdw, solv = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(3))
    frac = None
    if tags is not None:
        rt, lt, mem = (torch.as_tensor(t, device=dev).long() for t in tags)
        mb = torch.full((nr,), -1, device=dev).long()
        mb[mem] = torch.arange(len(mem), device=dev)
        groups = [int(rt.max()) + 1, int(lt.max()) + 1, len(mem)]
        frac = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    if fam == "cpydock":
        rx, lx = (torch.as_tensor(_excluded(m["hyd"]), device=dev) for m in (rec, lig))
        rd, ra, ld, la = T(rec["des"]), T(rec["asa"]), T(lig["des"]), T(lig["asa"])
    rf = torch.cat([rc, (rc * rc).sum(1, keepdim=True), torch.ones(nr, 1, dtype=torch.float64, device=dev)], 1).float()
    step = max(1, (1 << 27) // (nr * nl))
    for a in range(0, n, step):
        x = _rotate(P[a:a + step], lc).reshape(-1, 3)
        m = len(x) // nl
        if fam != "vdw":
            c = torch.nonzero(lq.repeat(m))[:, 0]
            elec[a:a + m].index_add_(0, c // nl, _far(x[c], lq.repeat(m)[c], rc, rq))
        xf = torch.cat([-2 * x, torch.ones(len(x), 1, dtype=torch.float64, device=dev), (x * x).sum(1, keepdim=True)],
                       1).float()
        i, k = torch.nonzero(xf @ rf.T < 101.0, as_tuple=True)   # a superset, decided in 64 bits below
        d2 = ((x[i] - rc[k]) ** 2).sum(1)
        i, k, d2 = (v[d2 <= 100.0] for v in (i, k, d2))
        p, j = i // nl, i % nl
        if fam != "vdw":
            elec[a:a + m].index_add_(0, p, torch.clamp(lq[j] * rq[k] / d2, -_CAP, _CAP))
        s = rr[k] + lr[j]
        p6 = (s * s / d2) ** 3
        v = torch.clamp(torch.sqrt(re[k] * le[j]) * (p6 * p6 - 2 * p6), max=1.0)
        if fam == "dna":
            d = torch.sqrt(d2)
            v = v + torch.where(rh[k] & lh[j] & (d < 0.75 * s), 6.0 * (0.75 * s - d), 0.0)
        vdw[a:a + m].index_add_(0, p, v)
        if tags is not None:
            c = d2 <= 3.9 * 3.9
            for b, (bit, size) in enumerate(zip((rt[k], lt[j], mb[k]), groups)):
                use = c & (bit >= 0)
                seen = torch.zeros(m, size, dtype=torch.bool, device=dev)
                seen[p[use], bit[use]] = True
                frac[a:a + m, b] = seen.sum(1).double() / size
        if fam == "cpydock":
            c = ~(rx[k] | lx[j]) & (d2 <= 6.4 * 6.4)
            for idx, size, des, asa in ((p * nr + k, nr, rd, ra), (i, nl, ld, la)):
                lo = torch.full((m * size,), 1e300, dtype=torch.float64, device=dev)
                lo = lo.scatter_reduce(0, idx[c], d2[c], "amin").reshape(m, size)
                g = torch.where((lo <= 6.4 * 6.4) & (lo > 0) & (asa > 0), 65.0 - 10.0 * torch.sqrt(lo), 0.0)
                solv[a:a + m] += (torch.where(asa > 0, torch.minimum(g, asa), 0.0) * des).sum(1)
    if fam == "cpydock":
        for asa, des in ((ra, rd), (la, ld)):
            solv += (torch.where(asa < 0, asa, 0.0) * des).sum()
    return elec, vdw, solv, frac


def _total(fam, elec, vdw, solv):
    ek = elec * 332.0 / 4.0
    if fam == "cpydock":
        return -(ek + 0.1 * vdw - solv)
    return -vdw if fam == "vdw" else -(ek + vdw)


def exact(case, seed):
    path = case["path"]
    # a GSO run and a fit are sequences of roundings and choices; the large
    # assembly would take minutes in 64 bits
    if path in ("gso", "surrogate") or case["n_rec"] * case["n_lig"] * case["n_pose"] > 2e12:
        return None
    cx = _complexes(case, seed)
    poses = _all_poses(case, seed, cx)
    if path == "compat":   # its parameters come as f32
        fam, rec, lig = cx[0]
        for m in (rec, lig):
            m["vdw"] = _f32(np.sqrt(m["vdw"])) ** 2
            m["ele"], m["radius"] = _f32(m["ele"]), _f32(m["radius"])
        elec, vdw, _, _ = _score64(fam, rec, lig, poses[0])
        return torch.stack([elec, vdw], 1).cpu().numpy()
    if path == "restraints":
        fam, rec, lig = cx[0]
        elec, vdw, solv, f = _score64(fam, rec, lig, poses[0], _restraints(case, seed, rec, poses[0]))
        s = _total(fam, elec, vdw, solv)
        s = s + f[:, 0] * s + f[:, 1] * s - torch.where(f[:, 2] > 0, 999.0 * f[:, 2], 0.0)
        return s.cpu().numpy(), f.cpu().numpy()
    out = torch.cat([_total(f, *_score64(f, r, l, p)[:3]) for (f, r, l), p in zip(cx, poses)]).cpu()
    if path == "energy":
        return float(out[0])
    return out.numpy() if path == "score" else out
