"""Performance cases of the library: what its users have it do, through its public entry points.

Each case names a kind of call and its sizes.  A kind's inputs come from seeded generators: atoms
uniform in a box (the two plain-kernel workloads with their own boxes, every other protein at the
heavy-atom density of a real one, 0.05 per cubic Angstrom), ligand atoms within 5 A of the origin,
34 forcefield types, poses with angles over the full circle and translations within 3 A.
"""
import ctypes
import math

import numpy as np
import torch

from minibude_gb300 import capi
from minibude_gb300.deck import (BatchDeck, Deck, synthetic_forcefield, synthetic_ligand, synthetic_poses,
                                 synthetic_protein)
from minibude_gb300.model import Gb300Bude, GpuContext, launch_cfg

NTYPES = 34
EXTENT, SPACING = 11.0, 1.25  # the surrogate's field grid, as GpuContext.surrogate_init has it


def listed():
    return [
        # An interactive rescoring: a handful of poses of one ligand from host buffers; latency.
        {"name": "host-938x26x64", "kind": "host", "natpro": 938, "half_box": 20.0, "natlig": 26, "nposes": 64,
         "tune": False},
        # The bm1-sized workload, poses in and energies out, with the autotuner's launch shape.
        {"name": "host-938x26x65536", "kind": "host", "natpro": 938, "half_box": 20.0, "natlig": 26,
         "nposes": 65536, "tune": True},
        # The headline workload, end to end from pinned host memory.
        {"name": "host-4096x64x1048576", "kind": "host", "natpro": 4096, "half_box": 30.0, "natlig": 64,
         "nposes": 1048576, "tune": True},
        # What the reference's driver does per launch shape: context, upload, 8 + 2 evaluations, download.
        {"name": "fasten-938x26x65536", "kind": "fasten", "natpro": 938, "half_box": 20.0, "natlig": 26,
         "nposes": 65536, "ppwi": 8, "wgsize": 64, "iterations": 8, "warmup": 2},
        # A pose set too large to stage at once, streamed from the host in chunks; odd count.
        {"name": "stream-2672x48x400003", "kind": "stream", "natpro": 2672, "half_box": 18.8, "natlig": 48,
         "nposes": 400003, "chunk": 65536},
        # A plugin inside another framework: device buffers, no allocation; odd sizes everywhere.
        {"name": "noalloc-1237x37x12345", "kind": "noalloc", "natpro": 1237, "half_box": 14.6, "natlig": 37,
         "nposes": 12345},
        # A virtual screen scored exhaustively: ragged ligands, uploaded, scored with the autotuner's
        # launch shape and read back.
        {"name": "batch-64x12to96", "kind": "batch", "natpro": 2672, "half_box": 18.8, "nligands": 64,
         "atoms_lo": 12, "atoms_hi": 96, "poses_lo": 1024, "poses_hi": 16384},
        # A few dozen conformers with a few hundred poses each: less work than the chip has room for.
        {"name": "batch-24x20to40-small", "kind": "batch", "natpro": 938, "half_box": 13.3, "nligands": 24,
         "atoms_lo": 20, "atoms_hi": 40, "poses_lo": 256, "poses_hi": 1024},
        # The learned pre-screen over held-out ligands.
        {"name": "score-64x16384", "kind": "score", "natpro": 938, "half_box": 20.0, "nligands": 64,
         "atoms_lo": 16, "atoms_hi": 64, "poses_lo": 16384, "poses_hi": 16384},
        # One loss gradient of the pre-screen (forward and backward) over a training batch.
        {"name": "gradient-8192", "kind": "gradient", "natpro": 938, "half_box": 20.0, "nligands": 64,
         "atoms_lo": 16, "atoms_hi": 64, "poses_lo": 512, "poses_hi": 512, "batch": 8192},
        # One training epoch in steps of 8,192 poses.
        {"name": "train-64x2048", "kind": "train", "natpro": 938, "half_box": 20.0, "nligands": 64,
         "atoms_lo": 16, "atoms_hi": 64, "poses_lo": 2048, "poses_hi": 2048, "batch": 8192},
        # The whole screen: pre-screen, selection, exact rescoring of the picks, audit.
        {"name": "screen-128x8192", "kind": "screen", "natpro": 2672, "half_box": 18.8, "nligands": 128,
         "atoms_lo": 16, "atoms_hi": 80, "poses_lo": 8192, "poses_hi": 8192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(natpro):
    return round(0.5 * (natpro / 0.05) ** (1.0 / 3.0), 3)


def draw(rng):
    """One more case of the listed kinds, sizes over their whole ranges."""
    kind = rng.choice(["host", "host", "host", "fasten", "stream", "noalloc", "batch", "batch", "score", "gradient",
                       "train", "screen"])
    natpro = _log(rng, 300, 4096)
    c = {"kind": kind, "natpro": natpro, "half_box": _box(natpro)}
    if kind == "host":
        c.update(natlig=_log(rng, 6, 96), nposes=_log(rng, 64, 400000), tune=rng.random() < 0.25)
        if c["natpro"] * c["natlig"] * c["nposes"] > 4e10:
            c["nposes"] = int(4e10 / (c["natpro"] * c["natlig"]))
    elif kind == "fasten":
        c.update(natlig=_log(rng, 6, 64), nposes=_log(rng, 512, 65536), ppwi=rng.choice([1, 2, 4, 8, 16]),
                 wgsize=rng.choice([32, 64, 128, 256]), iterations=8, warmup=2)
    elif kind == "stream":
        c.update(natlig=_log(rng, 12, 64), nposes=_log(rng, 30000, 300000), chunk=rng.choice([16384, 65536, 131072]))
    elif kind == "noalloc":
        c["natpro"] = natpro = min(natpro, 3800)
        c.update(half_box=_box(natpro), natlig=_log(rng, 6, 96), nposes=_log(rng, 64, 65536))
    elif kind == "batch":
        n, lo, hi = _log(rng, 4, 96), rng.randint(8, 24), rng.randint(24, 96)
        plo = _log(rng, 64, 2048)
        c.update(nligands=n, atoms_lo=lo, atoms_hi=hi, poses_lo=plo, poses_hi=plo * rng.randint(1, 8))
    else:
        p = _log(rng, 512, 4096)
        c.update(nligands=_log(rng, 16, 96), atoms_lo=rng.randint(8, 20), atoms_hi=rng.randint(24, 64), poses_lo=p,
                 poses_hi=p + rng.randint(0, 700))
        if kind in ("gradient", "train"):
            c["batch"] = _log(rng, 1024, 8192)
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _protein(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 11]))
    ff = synthetic_forcefield(rng, NTYPES)
    return rng, ff, synthetic_protein(rng, case["natpro"], case["half_box"], NTYPES)


def _deck(case, seed, nposes=None):
    rng, ff, protein = _protein(case, seed)
    ligand = synthetic_ligand(rng, case["natlig"], 5.0, NTYPES)
    n = case["nposes"] if nposes is None else nposes
    return Deck(protein, ligand, ff, synthetic_poses(rng, n), None, n, "perf")


def _batch(case, seed):
    rng, ff, protein = _protein(case, seed)
    shape = np.random.Generator(np.random.PCG64(10))  # a case's atom and pose counts are the same for every seed
    ligands, poses = [], []
    for _ in range(case["nligands"]):
        natlig = int(shape.integers(case["atoms_lo"], case["atoms_hi"] + 1))
        n = int(round(math.exp(shape.uniform(math.log(case["poses_lo"]), math.log(case["poses_hi"])))))
        ligands.append(synthetic_ligand(rng, natlig, 5.0, NTYPES))
        poses.append(synthetic_poses(rng, n))
    return BatchDeck(protein, ff, ligands, poses, "perf")


def _params(seed):
    """Network parameters in the library's layout.  A pass costs the same for any weights; these
    give scores of the spread that a network has at the start of its training."""
    rng = np.random.Generator(np.random.PCG64([seed, 12]))
    sizes = [(64 * 16, None), (128 * 32, 32), (128, 32), (128 * 128, 128), (128, 128), (128 * 128, 128), (128, 128),
             (128, 128), (4, None)]
    parts = [rng.normal(0, 1, n) if k is None else rng.uniform(-1, 1, n) / math.sqrt(k) for n, k in sizes]
    parts[-1][1:] = 0.0
    return np.concatenate(parts).astype(np.float32)


def _labels(n, seed):
    return np.random.Generator(np.random.PCG64([seed, 13])).normal(0.0, 200.0, n).astype(np.float32)


def _picked(total, k, seed):
    return np.random.Generator(np.random.PCG64([seed, 14])).permutation(total)[:k].astype(np.int32)


def _pinned(shape, values=None):
    """A page-locked float32 array that owns its memory."""
    a = torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()
    if values is not None:
        a[...] = values
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("host", "fasten", "stream", "noalloc"):
        deck = _deck(case, seed)
        s = {"case": case, "deck": deck}
        if kind in ("host", "stream"):
            s["ctx"] = GpuContext(0)
            s["ctx"].upload(deck)
            s["cfg"] = s["ctx"].autotune()[0] if case.get("tune") else s["ctx"].default_cfg(8, 128)
            s["poses"], s["energies"] = _pinned(deck.poses.shape, deck.poses), _pinned((deck.nposes,))
        elif kind == "noalloc":
            dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()  # noqa: E731
            s["dev"] = [dev(deck.protein), dev(deck.ligand), dev(deck.forcefield), dev(deck.poses)]
            s["energies"] = torch.empty(deck.nposes, device="cuda")
        return s
    batch = _batch(case, seed)
    s = {"case": case, "ctx": GpuContext(0), "nligands": batch.nligands}
    if kind in ("batch", "screen"):
        s["arrays"] = (batch.protein, batch.forcefield, batch.atoms(), batch.ligand_offsets())
        s["pose_off"], s["poses"] = batch.pose_offsets(), _pinned((6, batch.total_poses), batch.pose_block())
        s["energies"] = _pinned((batch.total_poses,))
    s["ctx"].upload_batch(batch)
    if kind == "batch":
        s["cfg"] = s["ctx"].autotune_batch()[0]
    else:
        s["ctx"].surrogate_init(batch.protein, batch.forcefield, EXTENT, SPACING, seed=seed)
        s["ctx"].surrogate_params(_params(seed))
    if kind in ("gradient", "train"):
        s["labels"] = _labels(batch.total_poses, seed)
        s["picked"] = _picked(batch.total_poses, case["batch"], seed)
    return s


# ---- one pass -------------------------------------------------------------------------------

def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "host":
        return s["ctx"].score_host(s["cfg"], s["poses"], s["energies"], ligand=s["deck"].ligand)
    if kind == "fasten":
        return Gb300Bude(case["ppwi"]).fasten(s["deck"], case["wgsize"], 0, case["iterations"],
                                              case["warmup"]).energies
    if kind == "stream":
        s["ctx"].score_stream(s["cfg"], s["poses"], s["energies"], chunk=case["chunk"])
        return s["energies"]
    if kind == "noalloc":
        d, p = s["deck"], [ctypes.c_void_p(t.data_ptr()) for t in s["dev"]]
        capi.check(capi.lib().bude_gpu_fasten_noalloc(p[0], d.natpro, p[1], d.natlig, p[2], d.ntypes, p[3], d.nposes,
                                                      d.nposes, ctypes.c_void_p(s["energies"].data_ptr()),
                                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return s["energies"]
    ctx = s["ctx"]
    if kind == "batch":
        protein, ff, atoms, lig_off = s["arrays"]
        ctx.upload_batch_arrays(protein, ff, atoms, lig_off, s["poses"], s["pose_off"])
        ctx.run_batch(s["cfg"])
        return ctx.download_batch(s["energies"])
    if kind == "score":
        ctx.surrogate_score()
        return ctx.surrogate_download()
    if kind == "gradient":
        grads, pred = ctx.surrogate_gradient(s["picked"], s["labels"])
        return {"grads": grads, "pred": pred}
    if kind == "train":
        loss, _ = ctx.surrogate_train(1, batch_poses=case["batch"], lr=1e-3, labels=s["labels"], seed=1)
        return {"params": ctx.surrogate_params(), "loss": loss}
    protein, ff, atoms, lig_off = s["arrays"]
    ctx.upload_batch_arrays(protein, ff, atoms, lig_off, s["poses"], s["pose_off"])
    # An audit tolerance no rank correlation exceeds: as with a trained network, nothing falls back.
    ctx.screen(launch_cfg(16, 128, 21, 32, 1, cluster=0), top_frac=0.02, audit_frac=0.005, audit_tol=2.5, seed=1)
    final, rescored, err = ctx.screen_download(s["nligands"])
    return {"final": final, "rescored": rescored, "audit_error": err}


# ---- the work a pass cannot do without --------------------------------------------------------

def _pair_terms(ff, lt, pt):
    """radij, charge weight and 1/reach, desolvation weight and 1/reach of ligand type lt against the
    protein types pt (float64 arrays), and the distance past which all three terms are zero."""
    f = {k: ff[k].astype(np.float64) for k in ("radius", "hphb", "elsc")}
    hb = ff["hbtype"]
    radij = f["radius"][pt] + f["radius"][lt]
    both_f = (hb[pt] == 70) & (hb[lt] == 70)
    c = f["elsc"][lt] * f["elsc"][pt]
    kc = 45.0 * np.where((hb[pt] == 69) | (hb[lt] == 69), -np.abs(c), c)
    hp, hl = f["hphb"][pt], f["hphb"][lt]
    d = hp * np.where((hp < 0) & (hl > 0), -1.0, 1.0) + hl * np.where((hp > 0) & (hl < 0), -1.0, 1.0)
    dist = np.where(hp < 0, np.where(hl < 0, 5.5, 1.0), np.where(hl < 0, 1.0, 0.0))
    on = (hp != 0) & (dist > 0)
    ic, idv = np.where(both_f, 0.25, 0.5), np.where(on, 1.0 / np.where(on, dist, 1.0), 1.0)
    kd = np.where(on, d, 0.0)
    reach = radij + np.maximum(np.where(kc != 0, 1.0 / ic, 0.0), np.where(on, dist, 0.0))
    return radij, kc, ic, kd, idv, reach


def _rotations(poses):
    p = poses.astype(np.float64)
    (sx, sy, sz), (cx, cy, cz) = np.sin(p[:3]), np.cos(p[:3])
    return np.array([[cy * cz, sx * sy * cz - cx * sz, cx * sy * cz + sx * sz],
                     [cy * sz, sx * sy * sz + cx * cz, cx * sy * sz - sx * cz], [-sy, sx * cy, cx * cy]]), p[3:]


def _xyz(a):
    return np.stack([a["x"], a["y"], a["z"]], 1).astype(np.float64)


def work(case):
    """Pairs of a ligand and a protein atom that lie within reach of each other cost the reference's
    30 operations each (src/main.cpp:359); their share is counted on a sample of the geometry.  A
    row of the pre-screen network costs 73,984 operations, three times that with its gradient."""
    kind = case["kind"]
    natpro = case["natpro"]
    one = dict(case, natlig=case.get("natlig", 24), nposes=24)
    d = _deck(one, 0)
    R, t = _rotations(d.poses)
    P, pt = _xyz(d.protein), d.protein["type"]
    near = 0
    for a in d.ligand[:24]:
        pos = (np.einsum("abn,b->an", R, np.array([a["x"], a["y"], a["z"]], np.float64)) + t).T
        reach = _pair_terms(d.forcefield, int(a["type"]), pt)[5]
        near += int((((pos[:, None] - P[None]) ** 2).sum(2) < reach ** 2).sum())
    per_point = near / (24.0 * min(24, d.natlig)) * 30 + 18
    if "natlig" in case:
        n, points, deck_bytes = case["nposes"], case["nposes"] * case["natlig"], 16 * (natpro + case["natlig"] + NTYPES)
        times = case.get("iterations", 1) + case.get("warmup", 0)
        return {"bytes": times * 28 * n + deck_bytes, "flops": times * (points * per_point + 28 * n)}
    atoms = 0.5 * (case["atoms_lo"] + case["atoms_hi"])
    lo, hi = case["poses_lo"], case["poses_hi"]
    n = case["nligands"] * (lo if hi <= lo else (hi - lo) / math.log(hi / lo))
    row = 73984.0
    if kind == "batch":
        return {"bytes": 28 * n, "flops": n * atoms * per_point + 28 * n}
    if kind == "score":
        return {"bytes": 28 * n, "flops": n * atoms * row}
    if kind in ("gradient", "train"):
        n = min(n, case["batch"]) if kind == "gradient" else n
        return {"bytes": 32 * n + 8 * 38404, "flops": 3 * n * atoms * row}
    return {"bytes": 33 * n, "flops": n * atoms * row + 0.025 * n * (atoms * per_point + 28)}


# ---- the same in 64 bits ----------------------------------------------------------------------

def _energies64(protein, ff, ligand, poses):
    R, t = (torch.from_numpy(v).cuda() for v in _rotations(poses))
    P, pt = _xyz(protein), protein["type"]
    out = torch.zeros(poses.shape[1], dtype=torch.float64, device="cuda")
    for a in ligand:
        pos = (torch.einsum("abn,b->an", R, torch.tensor([a["x"], a["y"], a["z"]], dtype=torch.float64).cuda()) + t).T
        terms = _pair_terms(ff, int(a["type"]), pt)
        lo, hi = pos.min(0).values.cpu().numpy(), pos.max(0).values.cpu().numpy()
        gap = np.maximum(0.0, np.maximum(lo - P, P - hi))
        keep = (gap ** 2).sum(1) < terms[5] ** 2  # the others' terms are zero at every pose
        if not keep.any():
            continue
        Q = torch.from_numpy(P[keep]).cuda()
        radij, kc, ic, kd, idv = (torch.from_numpy(v[keep]).cuda() for v in terms[:5])
        for b in range(0, len(out), 16384):
            r = torch.cdist(pos[b:b + 16384].contiguous(), Q, compute_mode="donot_use_mm_for_euclid_dist")
            e = 76.0 * (1 - r / radij).clamp_(0, 1)
            r -= radij
            e += kc * (1 - r * ic).clamp_(0, 1)
            e += kd * (1 - r * idv).clamp_(0, 1)
            out[b:b + 16384] += 0.5 * e.sum(1)
    return out


def _field64(protein, ff):
    """[n, n, n, 13] scaled field channels at the grid points (x, y, z order)."""
    n = int(math.ceil(2 * EXTENT / SPACING)) + 1
    axis = torch.arange(n, dtype=torch.float64, device="cuda") * SPACING - EXTENT
    pts = torch.stack(torch.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3)
    t = protein["type"]
    g = lambda v: torch.from_numpy(np.asarray(v, np.float64)).cuda()  # noqa: E731
    rad, q, h, is_f = g(ff["radius"][t]), g(ff["elsc"][t]), g(ff["hphb"][t]), g(ff["hbtype"][t] == 70)
    r = torch.cdist(pts, g(_xyz(protein)), compute_mode="donot_use_mm_for_euclid_dist")
    bb = r - (1.75 + rad)
    s2, s4, s55, s1 = ((1 - bb * k).clamp(0, 1) for k in (0.5, 0.25, 1 / 5.5, 1.0))
    neg, pos = h.clamp(max=0), h.clamp(min=0)
    c = [(1 - r / (p + rad)).clamp(min=0).sum(1) for p in (1.0, 1.5, 2.0, 2.5)]
    c += [(w * s).sum(1) for w, s in ((q, s2), (q, s4), (q.abs(), s2), (q.abs(), s4), (q * is_f, s4), (neg, s55),
                                      (pos, s1), (neg, s1))]
    c.append((r - rad).min(1).values.clamp(-3.0, 8.0))
    c = torch.stack(c, 1)
    sd = c.std(0, unbiased=False)
    return (c / torch.where(sd > 1e-6, sd, torch.ones_like(sd))).reshape(n, n, n, 13)


def _rows64(batch, field, which):
    """Types and features 16..31 of the rows of ligand l's poses which[l] (an index array), ligand by
    ligand."""
    n = field.shape[0]
    for l, idx in which:
        lig = batch.ligands[l]
        R, t = (torch.from_numpy(v).cuda() for v in _rotations(batch.poses[l][:, idx]))
        x = torch.einsum("abn,ib->nia", R, torch.from_numpy(_xyz(lig)).cuda()) + t.T[:, None]
        u = (x + EXTENT) / SPACING
        i0 = torch.floor(u)
        f = u - i0
        val = 0
        for c in range(8):
            bit = torch.tensor([c & 1, c >> 1 & 1, c >> 2], device="cuda")
            i = (i0.long() + bit).clamp(0, n - 1)
            w = torch.where(bit == 1, f, 1 - f).prod(-1, keepdim=True)
            val = val + w * field[i[..., 0], i[..., 1], i[..., 2]]
        types = torch.from_numpy(lig["type"].astype(np.int64)).cuda().expand(len(idx), -1)
        yield types, torch.cat([0.1 * x, val], -1)


def _network64(p, types, feats):
    act = lambda z: z * (z / 6 + 0.5).clamp(0, 1)  # noqa: E731
    o, parts = 0, []
    for shape in ((64, 16), (128, 32), (128,), (128, 128), (128,), (128, 128), (128,), (128,), (4,)):
        k = math.prod(shape)
        parts.append(p[o:o + k].reshape(shape))
        o += k
    emb, w1, b1, w2, b2, w3, b3, w4, b4 = parts
    h = act(torch.cat([emb[types], feats], -1) @ w1.T + b1)
    return (act(act(h @ w2.T + b2) @ w3.T + b3) @ w4 + b4[0]).sum(-1)


def exact(case, seed):
    kind = case["kind"]
    if "natlig" in case:
        d = _deck(case, seed)
        e = _energies64(d.protein, d.forcefield, d.ligand, d.poses)
        return e if kind == "noalloc" else e.cpu().numpy()
    if kind in ("train", "screen"):
        return None  # they follow from 16-bit roundings: updates over many steps, and which poses are picked
    batch = _batch(case, seed)
    if kind == "batch":
        return np.concatenate([_energies64(batch.protein, batch.forcefield, batch.ligands[l], batch.poses[l]).cpu()
                               .numpy() for l in range(batch.nligands)])
    field = _field64(batch.protein, batch.forcefield)
    p = torch.from_numpy(_params(seed).astype(np.float64)).cuda()
    if kind == "score":
        parts = []
        for l in range(batch.nligands):
            every = np.arange(batch.poses[l].shape[1])
            for b in range(0, len(every), 2048):
                for types, feats in _rows64(batch, field, [(l, every[b:b + 2048])]):
                    parts.append(_network64(p, types, feats).cpu().numpy())
        return np.concatenate(parts)
    p.requires_grad_(True)
    off, picked = batch.pose_offsets(), _picked(batch.total_poses, case["batch"], seed)
    lig = np.searchsorted(off, picked, side="right") - 1
    labels = torch.from_numpy(_labels(batch.total_poses, seed).astype(np.float64)).cuda()
    scale = lambda e: 20.0 * torch.asinh(e / 20.0)  # noqa: E731
    pred = torch.zeros(len(picked), dtype=torch.float64, device="cuda")
    for l in np.unique(lig):
        at = np.nonzero(lig == l)[0]
        for types, feats in _rows64(batch, field, [(int(l), picked[at] - off[l])]):
            got = _network64(p, types, feats)
            where = torch.from_numpy(at).cuda()
            pred[where] = got.detach()
            loss = (scale(got) - scale(labels[torch.from_numpy(picked[at].astype(np.int64)).cuda()])) ** 2
            (loss.sum() / len(picked)).backward()
    grads = p.grad.clone()
    grads[-3:] = 0.0
    return {"grads": grads.cpu().numpy(), "pred": pred.cpu().numpy()}
