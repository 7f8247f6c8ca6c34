"""The work this framework is used for, as cases that can be timed and compared.

Three kinds of pass, each through public entry points:

* ``step``: one timestep of a loaded simulation and the per-grain statistics a program
  reads after it (``GrainHandler.step`` + ``GrainHandler.stats``: existence, volumes,
  surfaces, boxes, neighbour counts).  The state advances with every pass, as it does in a
  program's loop; the sizes are such that a hundred timesteps leave the structure much as
  it was.
* ``run``: a whole short simulation, for domains that change too quickly to be stepped for
  long: create, load, initial lists, ``loops`` timesteps, then what a program saves at the
  end (statistics, hull neighbours, the voxel container), and close.
* ``convolve``: the batched Gaussian convolution of boxes in the caller's device memory.

The microstructures are Voronoi (or Laguerre) tessellations of uniform random points made
on the GPU from the seed: the same distributions as ``gragles_3d_b200.microstructure``,
whose host generator takes too long to be called for every preparation.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gragles_3d_b200 as gg
from gragles_3d_b200 import microstructure as msgen

TIME_STEP = 0.2


def _case(name, kind, domain, grains, precision, **kw):
    case = {"name": name, "kind": kind, "domain": domain, "grains": grains, "precision": precision,
            "border": 10, "physics": "isotropic", "loops": 1}
    case.update(kw)
    return case


def listed():
    return [
        # a first try-out or a unit test of a coupled program: launches and host latency
        _case("run_32_20_fp64", "run", 32, 20, "fp64", border=5, loops=12),
        # the plain 64^3 / 200-grain configuration at its full length, on both paths' storage
        _case("run_64_200_mixed", "run", 64, 200, "mixed", loops=51),
        # grid coarsening with the interfacial elements kept, odd domain and border
        _case("run_45_200_coarsen_fp64", "run", 45, 200, "fp64", border=7, loops=40, physics="coarsening"),
        # the isotropic 128^3 / 2,000-grain workload, both precisions
        _case("step_128_2000_mixed", "step", 128, 2000, "mixed"),
        _case("step_128_2000_fp64", "step", 128, 2000, "fp64"),
        # anisotropic energies and mobilities with the correction, reference precision, odd domain
        _case("step_117_1900_aniso_fp64", "step", 117, 1900, "fp64", physics="anisotropic"),
        # stored energy with nuclei (recrystallisation), small and large boxes side by side
        _case("step_160_7200_stored_mixed", "step", 160, 7200, "mixed", physics="stored"),
        # lognormal Laguerre grains, isotropic, many small boxes
        _case("step_208_16800_laguerre_mixed", "step", 208, 16800, "mixed", physics="laguerre"),
        # late growth or a finely resolved sample: few grains, box sides above 64
        _case("step_120_30_coarse_mixed", "step", 120, 30, "mixed", physics="anisotropic"),
        # the flagship: 256^3 / 20,000 grains, anisotropic with the correction, both precisions
        _case("step_256_20000_aniso_mixed", "step", 256, 20000, "mixed", physics="anisotropic"),
        _case("step_192_8400_aniso_fp64", "step", 192, 8400, "fp64", physics="anisotropic"),
        # the convolution alone on a caller's boxes of mixed sides
        _case("convolve_48_mixed", "convolve", 128, 48, "mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "run", "convolve"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "convolve":
        return {"kind": kind, "domain": rng.randint(96, 160), "grains": rng.randint(20, 60), "precision": precision,
                "border": 10, "physics": "isotropic", "loops": 1}
    if kind == "run":
        domain = rng.randint(32, 66)
        return {"kind": kind, "domain": domain, "grains": max(12, int(domain ** 3 / rng.uniform(500, 1800))),
                "precision": precision, "border": rng.choice([5, 7, 10]), "loops": rng.randint(10, 50),
                "physics": rng.choice(["isotropic", "isotropic", "anisotropic", "coarsening"])}
    physics = rng.choice(["isotropic", "anisotropic", "anisotropic", "stored", "laguerre"])
    domain = _log_int(rng, 100, 200)
    # mean grain volume: 530 (finely grained) to 6,000 voxels; late growth (FP32 storage holds
    # its large boxes) up to 40,000
    lo, hi = (20000, 40000) if precision == "mixed" and rng.random() < 0.25 else (530, 6000)
    per_grain = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {"kind": kind, "domain": domain, "grains": max(24, int(domain ** 3 / per_grain)), "precision": precision,
            "border": 10, "physics": physics, "loops": 1}


# --- microstructures ---------------------------------------------------------------
def _label(N, pts, weights):
    """Label of every voxel: the point of least (power) distance to its centre, found
    among the points nearest to the centre of its 8^3 block."""
    dev = pts.device
    G = pts.shape[0]
    w = torch.zeros(G, device=dev) if weights is None else weights
    nb = (N + 7) // 8
    ax = torch.arange(nb, device=dev, dtype=torch.float32) * 8 + 4
    cz, cy, cx = torch.meshgrid(ax, ax, ax, indexing="ij")
    centres = torch.stack([cx.reshape(-1), cy.reshape(-1), cz.reshape(-1)], 1)
    o = torch.arange(8, device=dev, dtype=torch.float32) - 3.5
    oz, oy, ox = torch.meshgrid(o, o, o, indexing="ij")
    off = torch.stack([ox.reshape(-1), oy.reshape(-1), oz.reshape(-1)], 1)
    K = min(G, 96)
    out = torch.empty((nb * nb * nb, 512), dtype=torch.int32, device=dev)
    step = max(1, min(2048, 60_000_000 // G))
    for b in range(0, centres.shape[0], step):
        c = centres[b:b + step]
        d = sum((c[:, None, a] - pts[None, :, a]) ** 2 for a in range(3)) - w[None, :]
        near = d.topk(K, dim=1, largest=False).indices.sort(dim=1).values
        v = c[:, None, :] + off[None, :, :]
        p, pw = pts[near], w[near]
        dist = sum((v[:, :, None, a] - p[:, None, :, a]) ** 2 for a in range(3)) - pw[:, None, :]
        out[b:b + step] = torch.gather(near, 1, dist.argmin(dim=2)).to(torch.int32) + 1
    out = out.reshape(nb, nb, nb, 8, 8, 8).permute(0, 3, 1, 4, 2, 5).reshape(nb * 8, nb * 8, nb * 8)
    return out[:N, :N, :N].contiguous()


def _extents(labels, G):
    """Inclusive extents (G, 6) and voxel counts (G,) of the labels, as the mode-4 input has them."""
    dev, N = labels.device, labels.shape[0]
    lab = labels.reshape(-1).to(torch.int64)
    counts = torch.bincount(lab, minlength=G + 1)[1:]
    idx = torch.arange(N, device=dev, dtype=torch.int32)
    ext = torch.zeros((G, 6), dtype=torch.int32, device=dev)
    for axis in range(3):  # x, y, z
        shape = [1, 1, 1]
        shape[2 - axis] = N
        coord = idx.reshape(shape).expand(N, N, N).reshape(-1)
        lo = torch.full((G + 1,), N, dtype=torch.int32, device=dev).scatter_reduce(0, lab, coord, "amin")
        hi = torch.full((G + 1,), -1, dtype=torch.int32, device=dev).scatter_reduce(0, lab, coord, "amax")
        ext[:, 2 * axis], ext[:, 2 * axis + 1] = lo[1:], hi[1:]
    ext[counts == 0] = 0
    return ext.cpu().numpy(), counts.cpu().numpy().astype(np.int64)


def _euler(rng, G):
    """Uniformly random orientations as Bunge angles."""
    u = rng.random((G, 3))
    return np.stack([2 * np.pi * u[:, 0], np.arccos(2 * u[:, 1] - 1), 2 * np.pi * u[:, 2]], axis=1)


def _microstructure(case, seed):
    N, G = case["domain"], case["grains"]
    rng = np.random.default_rng([seed, N, G])
    pts = torch.from_numpy((rng.random((G, 3)) * N).astype(np.float32)).cuda()
    weights = None
    if case["physics"] == "laguerre":  # lognormal radii, mean cell volume N^3 / G
        r = np.exp(0.3 * rng.standard_normal(G))
        r *= (N ** 3 / G * 3 / (4 * np.pi)) ** (1 / 3) / r.mean()
        weights = torch.from_numpy((r * r).astype(np.float32)).cuda()
    labels = _label(N, pts, weights)
    torch.cuda.empty_cache()  # the library allocates its own device memory
    euler = _euler(rng, G)
    energy = None
    if case["physics"] == "stored":
        # lognormal stored energy in the parents, 5% nuclei of radius 2-3 voxels with none
        energy = 0.1 * np.exp(0.5 * rng.standard_normal(G)) * msgen.HAGB_ENERGY
        K = max(1, round(0.05 * G))
        centre = torch.from_numpy(rng.random((K, 3)) * N).cuda()
        radius = torch.from_numpy(2 + rng.random(K)).cuda()
        o = torch.arange(-4, 5, device="cuda")
        oz, oy, ox = torch.meshgrid(o, o, o, indexing="ij")
        v = centre.floor().long()[:, None, :] + torch.stack([ox.reshape(-1), oy.reshape(-1), oz.reshape(-1)], 1)[None]
        inside = ((v + 0.5 - centre[:, None, :]) ** 2).sum(2) <= (radius ** 2)[:, None]
        inside &= ((v >= 0) & (v < N)).all(2)
        ids = (G + 1 + torch.arange(K, device="cuda"))[:, None].expand(-1, v.shape[1])
        at = (v[..., 2] * N + v[..., 1]) * N + v[..., 0]
        flat = labels.reshape(-1).long()
        labels = flat.scatter_reduce(0, at[inside], ids[inside], "amax").to(torch.int32).reshape(N, N, N)
        G += K
        energy = np.concatenate([energy, np.zeros(K)])
        euler = np.concatenate([euler, _euler(rng, K)])
    ext, counts = _extents(labels, G)
    return {"labels": labels.cpu().numpy().astype(np.uint32), "extents": ext, "counts": counts, "euler": euler,
            "energy": energy, "grains": G}


def _start(case, ms):
    """A handler with the microstructure loaded and its lists built: what gg_run does before its loop."""
    physics = case["physics"]
    kw = {}
    if physics in ("anisotropic", "stored"):
        kw = {"correction": True, "unique_energies": False, "mobility_model": True,
              "stored_energy": physics == "stored"}
        if case["domain"] ** 3 < 1500 * case["grains"]:  # small grains: a few thousand triangles at most
            kw["hull_capacity"] = 6000
    elif physics == "coarsening":
        kw = {"grid_coarsening": True, "keep_elements": True}
    if case["domain"] >= 200:  # as the large workloads are run: room for the boxes' growth, not for twice their voxels
        e = ms["extents"].astype(np.int64)
        side = np.maximum.reduce([e[:, 1] - e[:, 0], e[:, 3] - e[:, 2], e[:, 5] - e[:, 4]]) + 1 + 2 * case["border"]
        kw["pool_voxels"] = int(1.4 * (side[ms["counts"] > 0] ** 3).sum())
    h = gg.GrainHandler(case["domain"], case["border"], TIME_STEP, ms["grains"],
                        precision=gg.PRECISION_FP64 if case["precision"] == "fp64" else gg.PRECISION_MIXED, **kw)
    h.load(ms["labels"], ms["extents"], ms["counts"])
    if kw.get("correction"):
        h.set_orientations(ms["euler"])
    if kw.get("stored_energy"):
        h.set_stored_energy(ms["energy"])
    h.rtree_lists()
    return h


# --- the three kinds of pass --------------------------------------------------------
def _boxes(case, seed):
    """Signed-distance-like FP boxes of a convolve case: side, offset and the packed fields."""
    n = case["grains"]
    rng = np.random.default_rng([n, case["domain"]])
    sides = np.clip(np.round(26 + 14 * np.exp(0.5 * rng.standard_normal(n))).astype(np.int32) - 6, 20, 64)
    offs = np.concatenate([[0], np.cumsum((sides.astype(np.int64) ** 3 + 31) // 32 * 32)])
    host = np.zeros(int(offs[-1]))
    h = 1.0 / case["domain"]
    delta = case["border"] * h
    rng = np.random.default_rng(seed)
    for b, s in enumerate(sides):
        ax = np.arange(s) - (s - 1) / 2 + rng.uniform(-1, 1)
        d = np.sqrt(ax[:, None, None] ** 2 + ax[None, :, None] ** 2 * rng.uniform(0.8, 1.2) + ax[None, None, :] ** 2)
        host[offs[b]:offs[b] + int(s) ** 3] = np.clip((s / 2 - case["border"] - d) * h, -delta, delta).ravel()
    if case["precision"] == "mixed":
        host = host.astype(np.float32)
    return sides, offs[:-1].copy(), host


def prepare(case, seed):
    if case["kind"] == "convolve":
        sides, offs, host = _boxes(case, seed)
        x = torch.from_numpy(host).cuda()
        return {"case": case, "sides": sides, "offs": offs, "in": x, "out": torch.zeros_like(x)}
    ms = _microstructure(case, seed)
    if case["kind"] == "step":
        return {"case": case, "handler": _start(case, ms)}
    return {"case": case, "ms": ms}


def _stats(h):
    s = h.stats()
    return {"exists": s.exists, "volume": s.volume, "surface": s.surface, "boxes": s.boxes, "n_neighbors": s.n_neighbors}


def run(state):
    case = state["case"]
    if case["kind"] == "convolve":
        fn = "gg_convolve_boxes_f64" if case["precision"] == "fp64" else "gg_convolve_boxes_mixed"
        p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        rc = getattr(gg.load_library(), fn)(ctypes.c_void_p(state["in"].data_ptr()),
                                            ctypes.c_void_p(state["out"].data_ptr()), p(state["sides"]),
                                            p(state["offs"]), len(state["sides"]), case["domain"], TIME_STEP)
        if rc < 0:
            raise gg.GGError(rc, fn)
        return state["out"]
    if case["kind"] == "step":
        h = state["handler"]
        report = h.step()
        return dict(_stats(h), grain_count=report["grain_count"], voxel_updates=report["voxel_updates"])
    with _start(case, state["ms"]) as h:
        reports = [h.step() for _ in range(case["loops"])]
        labels = h.voxel_container()  # smaller than the initial domain after a grid coarsening
        out = dict(_stats(h), container=np.zeros((case["domain"],) * 3, np.uint32))
        out["container"][:labels.shape[0], :labels.shape[1], :labels.shape[2]] = labels
        out["neighbors"] = np.zeros((len(out["exists"]), 256), np.int64)
        for g in np.flatnonzero(out["exists"]):
            ids = h.neighbors(int(g))
            out["neighbors"][g, :len(ids)] = ids
    for key in ("grain_count", "voxel_updates"):
        out[key] = np.array([r[key] for r in reports])
    return out


# --- the work a pass cannot do without ----------------------------------------------
def _box_voxels(case):
    """Voxels of all grain boxes: a Voronoi cell's extent is about 1.45 times the side of
    the cube of its volume, its box adds the border on both sides and stays in the grid."""
    N, G = case["domain"], case["grains"]
    side = min(1.45 * N / G ** (1 / 3) + 2 * case["border"], N + 2 * case["border"])
    return G * side ** 3, side


def work(case):
    fp64 = case["precision"] == "fp64"
    if case["kind"] == "convolve":
        sides, _, host = _boxes(case, 0)
        v, n = float((sides.astype(np.float64) ** 3).sum()), float(sides.max())
        return {"bytes": 2 * v * (8 if fp64 else 4), "flops": v * (15 * math.log2(n) + 1)}
    # per box voxel and timestep: convolution, comparison, contour and redistancing each read
    # the field once and all but the contour write it once, and the neighbour ID is written once
    v, side = _box_voxels(case)
    per = 7 * (8 if fp64 else 4) + 4
    flops = v * (15 * math.log2(side) + 24)
    return {"bytes": float(v * per * case["loops"]), "flops": float(flops * case["loops"])}


def exact(case, seed):
    """The convolution in 64 bits; a timestep is a chain of discrete choices with no such value."""
    if case["kind"] != "convolve":
        return None
    sides, offs, host = _boxes(case, seed)
    x = host.astype(np.float64)
    out = np.zeros_like(x)
    for s, o in zip(sides, offs):
        n = int(s)
        f = np.fft.rfftn(x[o:o + n ** 3].reshape(n, n, n))
        i = np.minimum(np.arange(n), n - np.arange(n)).astype(np.float64) ** 2
        k = np.arange(n // 2 + 1).astype(np.float64) ** 2
        S = i[:, None, None] + i[None, :, None] + k[None, None, :]
        f *= np.exp(-math.sqrt(2 / math.pi) * S * 4 * TIME_STEP / (n * n) * math.pi * math.pi)
        out[o:o + n ** 3] = np.fft.irfftn(f, s=(n, n, n), axes=(0, 1, 2)).ravel()
    return torch.from_numpy(out)
