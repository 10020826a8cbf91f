"""What a user of this library runs, as timed cases.

Each case is one call (or one call sequence) through the package's public
functions on seeded data: `prepare` makes the inputs and the objects a
program keeps, `run` makes the call, `work` states the bytes that the call
cannot do without, and `exact` gives the numbers in 64 bits where a short
formula has them.  The snapshots are the synthetic workloads 1 to 5 of
csrc/synth.c at the scales given here.
"""
import importlib
import math

import numpy as np
import torch

rk = importlib.import_module("mpi-rockstar_gb300")

SYNTH_SEED = 20261203

# Largest scale of each workload in a drawn case: no more time than the
# largest listed case takes.
BATCHED_MAX = {1: 16.0, 2: 8.0, 3: 0.03, 4: 0.25, 5: 0.2}
PLAIN_MAX = {1: 1.0, 2: 0.25, 3: 0.005, 4: 1 / 256, 5: 0.004}
HOST_MAX = {1: 8.0, 2: 4.0, 3: 0.03, 4: 1 / 16, 5: 0.1}
SMALLEST = 20000  # particles of the smallest drawn snapshot
PER_UNIT = {1: 262144, 2: 2097152, 3: 81158533, 4: 134217728, 5: 25000000}


def listed():
    return [
        # The whole path on particles in HBM, batched form: what a program
        # that keeps its snapshot on the GPU calls once per snapshot.
        # The smallest snapshot (64^3): launches and host round trips count.
        {"name": "path_64cube", "kind": "path", "workload": 1, "scale": 1.0, "batched": True,
         "a": 1.0},
        # 128^3 with substructure: an ordinary chunk.
        {"name": "path_128cube", "kind": "path", "workload": 2, "scale": 1.0, "batched": True,
         "a": 1.0},
        # Isolated groups of very uneven sizes, no background.
        {"name": "path_groups", "kind": "path", "workload": 3, "scale": 0.03, "batched": True,
         "a": 1.0},
        # The benchmark's snapshot (512^3) at a quarter of its volume: the
        # largest call.
        {"name": "path_512cube_quarter", "kind": "path", "workload": 4, "scale": 0.25,
         "batched": True, "a": 1.0},
        # One cluster holding most particles: a zoom run, one group's levels
        # and no others to fill the chip.
        {"name": "path_cluster", "kind": "path", "workload": 5, "scale": 0.2, "batched": True,
         "a": 1.0},
        # The plain form (the reference's results bit for bit) on a small
        # chunk at z = 1.
        {"name": "path_plain", "kind": "path", "workload": 2, "scale": 0.25, "batched": False,
         "a": 0.5},
        # The drop-in calls on host arrays, as the C program makes them: the
        # 3D FOF of one chunk ...
        {"name": "fof_host", "kind": "fof_host", "workload": 4, "scale": 0.0625, "a": 1.0},
        # ... and the substructure step over the groups of a chunk.
        {"name": "subs_host", "kind": "subs_host", "workload": 2, "scale": 0.5, "a": 1.0},
        # The allocation-free 3D FOF inside a simulation step, at its limit
        # of 65,536 particles.
        {"name": "fof_noalloc", "kind": "fof_noalloc", "workload": 1, "scale": 0.25, "a": 1.0},
        # The id sort before halo finding, records in HBM (256^3 less an odd
        # number, ids of a larger run).
        {"name": "sort_256cube", "kind": "sort", "n": 16777141, "id_bits": 29},
        # Potentials of one halo by the reference's call, reference arithmetic.
        {"name": "potential_halo", "kind": "potential", "n": 3001, "form": 0},
        # Potentials of a cluster, FP32 Kahan form.
        {"name": "potential_cluster", "kind": "potential", "n": 500000, "form": 1},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["path", "path", "path", "plain", "fof_host", "subs_host", "fof_noalloc",
                       "sort", "potential"])
    a = rng.choice([1.0, 1.0, 0.5])
    if kind == "sort":
        n = int(_log_uniform(rng, 1000, 16777216))
        return {"kind": "sort", "n": n, "id_bits": rng.randint(max(n - 1, 1).bit_length(), 62)}
    if kind == "potential":
        form = rng.choice([0, 1])
        return {"kind": "potential", "n": int(_log_uniform(rng, 100, 500000 if form else 50000)),
                "form": form}
    if kind == "fof_noalloc":
        w = rng.choice([1, 2])
        return {"kind": kind, "workload": w, "a": a,
                "scale": _log_uniform(rng, 4096, 65536) / PER_UNIT[w]}
    w = rng.randint(1, 5)
    top = {"path": BATCHED_MAX, "plain": PLAIN_MAX}.get(kind, HOST_MAX)[w]
    case = {"workload": w, "scale": _log_uniform(rng, min(SMALLEST / PER_UNIT[w], top), top),
            "a": a}
    if kind in ("path", "plain"):
        return dict(case, kind="path", batched=kind == "path")
    return dict(case, kind=kind)


def _snapshot(case, seed):
    """The workload's structures as another snapshot: every particle displaced
    by a fiftieth of the linking length, the box mirrored along axes that the
    seed picks, the particles numbered in another order.  (records on the
    GPU, configuration); the particle count is the workload's."""
    p, box, mp, _ = rk.synth(case["workload"], case["scale"], SYNTH_SEED)
    n = len(p)
    cfg = rk.Config(particle_mass=mp, box_size=box, total_particles=n, scale_now=case["a"])
    link = cfg.fof_linking_length * rk.setup_config(cfg).avg_particle_spacing
    g = torch.Generator(device="cuda").manual_seed(seed)
    at = torch.randperm(n, device="cuda", generator=g)
    rec = torch.from_numpy(p.view(np.uint8).reshape(n, 32)).cuda()[at]
    f = rec.view(torch.float32)
    f[:, 2:5] += torch.randn(n, 3, device="cuda", generator=g) * (0.02 * link)
    for axis in range(3):
        if (seed >> axis) & 1:
            f[:, 2 + axis] = box - f[:, 2 + axis]
            f[:, 5 + axis].neg_()
    rec.view(torch.int64)[:, 0] = torch.arange(n, device="cuda")
    torch.cuda.synchronize()  # the library works on a stream of its own
    return rec, cfg


def _to_host(rec):
    return rec.cpu().numpy().reshape(-1).view(rk.PARTICLE)


def _sort_input(case, seed):
    """Shuffled records whose ids are spread over id_bits bits, all distinct."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    step = max(1, (1 << case["id_bits"]) // n)
    ids = torch.arange(n, device="cuda") * step
    if step > 1:
        ids += torch.randint(0, step, (n,), device="cuda", generator=g)
    ids = ids[torch.randperm(n, device="cuda", generator=g)]
    rec = torch.empty(n, 32, dtype=torch.uint8, device="cuda")
    rec.view(torch.int64)[:, 0] = ids
    rec.view(torch.float32)[:, 2:5] = torch.rand(n, 3, device="cuda", generator=g) * 500
    rec.view(torch.float32)[:, 5:8] = torch.randn(n, 3, device="cuda", generator=g) * 300
    return rec


def _potential_input(case, seed):
    """One NFW halo (c = 8, 200 times the critical density) about a point of
    the box; `flags` holds each record's place, since the call leaves the
    records in tree order."""
    r = np.random.default_rng(seed)
    n, c, mp = case["n"], 8.0, 1e9
    r200 = (3 * n * mp / (4 * math.pi * 200 * 2.77519737e11)) ** (1 / 3)
    x = np.linspace(0, c, 20001)
    m = np.log1p(x) - x / (1 + x)
    dist = np.interp(r.random(n) * m[-1], m, x) * (r200 / c)
    v = r.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    po = np.zeros(n, rk.POTENTIAL)
    po["pos"][:, :3] = r.uniform(5, 35, 3) + dist[:, None] * v
    po["pos"][:, 3:] = r.normal(scale=300.0, size=(n, 3))
    po["flags"] = np.arange(n)
    return po, rk.Config(particle_mass=mp)


def _device_path(n, cfg, batched):
    path = rk.DevicePath(n, cfg, batched=batched)
    for t in (path.out, path.halos, path.extra):
        t.zero_()  # capacity beyond what a pass writes
    return path


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "sort":
        # the call sorts in place: each pass sorts the records afresh, as a
        # reader would leave them
        s["source"] = _sort_input(case, seed)
        s["records"] = torch.empty_like(s["source"])
    elif kind == "potential":
        s["records"], s["cfg"] = _potential_input(case, seed)
        s["form"] = case["form"]
    else:
        rec, cfg = _snapshot(case, seed)
        n = len(rec)
        s["cfg"] = cfg
        if kind == "path":
            s["input"] = rec
            s["path"] = _device_path(n, cfg, case["batched"])
        elif kind in ("fof_host", "subs_host"):
            # both calls permute the particles in place: each pass takes them
            # afresh from `source`
            s["source"] = _to_host(rec)
            s["particles"] = s["source"].copy()
            s["offsets"] = np.zeros(n // 10 + 1, np.int64)
            s["sizes"] = np.zeros(n // 10 + 1, np.int64)
            if kind == "subs_host":
                _, s["offsets"], s["sizes"] = rk.rockstar_fof(s["source"], cfg, inplace=True)
                s["halos"] = np.zeros(n // 8 + 64, rk.HALO)
                s["extra"] = np.zeros(n // 8 + 64, rk.EXTRA)
        else:
            s["n"] = n
            s["cap"] = n // 2 + 1
            s["input"] = rec
            s["cfg"] = rk.setup_config(cfg)
            s["out"] = torch.zeros(n, 32, dtype=torch.uint8, device="cuda")
            s["offsets"] = torch.zeros(s["cap"], dtype=torch.int64, device="cuda")
            s["sizes"] = torch.zeros(s["cap"], dtype=torch.int64, device="cuda")
            s["stream"] = torch.cuda.Stream()
    torch.cuda.synchronize()
    return s


# The halo record by columns of 4 bytes (floats) and 8 bytes (counts, flags,
# links), so that large fields do not hide small ones.
_F = {}
for _name in rk.HALO.names:
    if rk.HALO[_name].base == np.dtype("<f4"):
        _o = rk.HALO.fields[_name][1] // 4
        _F[_name] = (_o, _o + (rk.HALO[_name].itemsize // 4))
_FLOAT_GROUPS = [("pos",), ("corevel", "bulkvel"), ("m", "mgrav"), ("r", "child_r", "vmax_r"),
                 ("vmax", "vrms"), ("rvmax", "rs", "klypin_rs"), ("J",), ("energy",), ("spin",),
                 ("alt_m",), ("Xoff",), ("Voff",), ("b_to_a", "c_to_a"), ("A",),
                 ("b_to_a2", "c_to_a2"), ("A2",), ("bullock_spin", "kin_to_pot"),
                 ("m_pe_b", "m_pe_d"), ("halfmass_radius",),
                 ("min_pos_err", "min_vel_err", "min_bulkvel_err"), ("inertia_tensor",),
                 ("inertia_tensor2",), ("chi2",)]
_INTS = (rk.HALO.fields["num_p"][1] // 8, rk.HALO.fields["n_core"][1] // 8 + 1)


def _columns(ids, rec_f, halo_f, halo_i, extra_i, extra_f):
    out = {"ids": ids, "pos": rec_f[:, 2:8], "halo_ints": halo_i[:, _INTS[0]:_INTS[1]],
           "links": extra_i[:, :5], "max_metric": extra_f[:, 10]}
    for names in _FLOAT_GROUPS:
        out["_".join(names)] = halo_f[:, _F[names[0]][0]:_F[names[-1]][1]]
    return out


def _device_columns(path):
    rec, h, e = path.out, path.halos, path.extra
    return _columns(rec.view(torch.int64).view(-1, 4)[:, 0],
                    rec.view(torch.float32).view(-1, 8),
                    h.view(torch.float32).view(-1, 78), h.view(torch.int64).view(-1, 39),
                    e.view(torch.int64).view(-1, 6), e.view(torch.float32).view(-1, 12))


def _host_columns(p, h, e):
    return _columns(p["id"], p.view("<f4").reshape(-1, 8),
                    h.view("<f4").reshape(-1, 78), h.view("<i8").reshape(-1, 39),
                    e.view("<i8").reshape(-1, 6), e.view("<f4").reshape(-1, 12))


def _refill(s):
    """The host particles as the reader left them (several threads copy)."""
    torch.from_numpy(s["particles"].view(np.uint8)).copy_(
        torch.from_numpy(s["source"].view(np.uint8)))
    return s["particles"]


def run(s):
    kind = s["kind"]
    if kind == "path":
        num_p, num_fofs, num_halos = s["path"].run(s["input"].data_ptr())
        return dict(_device_columns(s["path"]), counts=[num_p, num_fofs, num_halos])
    if kind == "fof_host":
        p = _refill(s)
        q, off, sz = rk.rockstar_fof(p, s["cfg"], inplace=True)
        s["offsets"][:len(off)] = off
        s["sizes"][:len(sz)] = sz
        return {"ids": p["id"], "pos": p["pos"], "offsets": s["offsets"], "sizes": s["sizes"],
                "counts": [len(q), len(off)]}
    if kind == "subs_host":
        p, h, e = rk.find_subs(_refill(s), s["offsets"], s["sizes"], s["cfg"], batched=True,
                               inplace=True)
        s["halos"][:len(h)] = h
        s["extra"][:len(e)] = e
        return dict(_host_columns(p, s["halos"], s["extra"]), counts=[len(h)])
    if kind == "fof_noalloc":
        num_p, nf = rk.rockstar_fof_noalloc(s["input"].data_ptr(), s["n"], s["cfg"],
                                            s["out"].data_ptr(), s["offsets"].data_ptr(),
                                            s["sizes"].data_ptr(), s["cap"],
                                            s["stream"].cuda_stream)
        return {"ids": s["out"].view(torch.int64)[:, 0],
                "pos": s["out"].view(torch.float32)[:, 2:], "offsets": s["offsets"],
                "sizes": s["sizes"], "counts": [num_p, nf]}
    if kind == "sort":
        rec = s["records"].copy_(s["source"])
        rk.sort_by_id_device(rec.view(-1))
        return {"ids": rec.view(torch.int64)[:, 0], "pos": rec.view(torch.float32)[:, 2:]}
    q = rk.compute_potential(s["records"], s["cfg"], form=s["form"])
    pe = np.empty(len(q))
    pe[q["flags"]] = q["pe"]
    return {"order": q["flags"], "pe": pe}


def work(case):
    """Each input record read once, each output record written once."""
    kind = case["kind"]
    if kind == "sort":
        # the sorted records; the copy that refills them is not the sort's
        return {"bytes": 64 * case["n"], "flops": 0}
    if kind == "potential":
        return {"bytes": 96 * case["n"], "flops": 0}
    n = rk.synth_count(case["workload"], case["scale"], SYNTH_SEED)
    return {"bytes": 64 * n, "flops": 0}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        rec = _sort_input(case, seed)
        ids, at = torch.sort(rec.view(torch.int64)[:, 0])
        return {"ids": ids, "pos": rec.view(torch.float32)[at, 2:].double()}
    if kind == "potential":
        # every pair in 64 bits, softened as the call softens it; the tree
        # code's opening angle is the difference between the two
        po, cfg = _potential_input(case, seed)
        x = torch.from_numpy(po["pos"][:, :3].astype(np.float64)).cuda()
        pe = torch.empty(len(x), dtype=torch.float64, device="cuda")
        for i in range(0, len(x), 512):
            r = (x[i:i + 512, None, :] - x[None, :, :]).square_().sum(-1).sqrt_()
            inv = r.clamp_(min=cfg.force_res).reciprocal_()
            k = torch.arange(inv.shape[0], device="cuda")
            inv[k, i + k] = 0.0
            pe[i:i + 512] = inv.sum(1)
        return {"order": None, "pe": pe * cfg.particle_mass}
    return None  # the halo finder's decision chains have no short formula
