"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" says which public entry point it goes through:
  scattering  models.frequency_domain.calculate_scattering, host arrays in and out, the scene's
              Tile_acceleration_structure kept by the caller (engine "cuda" or "numba", source-summed or per element)
  brute       propagation.pair_stage without a grid (Brute_Force structures, small meshes), device arrays
  network     beam_sweep.form_network: the per-pair network of an array, device arrays
  adjoint     adjoint.sink_field forward and backward
  sweep       beam_sweep.BeamSweep.run over a prepared network
  batched     batched.BatchedScattering.run: many uneven scenes x many frequencies in one launch
  paths       raycasting.numba_masks and empropagation.EMGPUFreqDomain: the numba engine's visibility sets and the
              products of a path list
Scenes are an array at the origin, an optional ground plane with random clutter triangles above it, scatter points
on the triangles and far-field sinks on an elevation-azimuth grid, as in the package's own scenes.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "lyceanem-python_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

C0 = 299792458.0
EXACT_TESTS = 3e10   # ray-triangle tests that exact() is ready to do in plain torch
EXACT_PAIRS = 2e7    # pairs whose field it is ready to form in 64 bits


def listed():
    return [
        # a small antenna behind clutter, one source-summed pattern at 5 degrees: a call of a design loop,
        # where host work and launches count
        _scat("direct_10ghz", side=8, n_el=37, n_az=72, radius=10.0, ground=0, clutter=1024, box=1.0, size=0.05,
              n_scat=0, freq=10e9, cell=0.0),
        # the same pattern by brute force on device arrays, with the visibility mask
        dict(_scat("brute_10ghz", side=8, n_el=37, n_az=72, radius=10.0, ground=0, clutter=1024, box=1.0, size=0.05,
                   n_scat=0, freq=10e9, cell=0.0), kind="brute"),
        # a small one-bounce scene (odd sizes): three stages of few thousand rays each
        _scat("bounce_small", side=5, n_el=37, n_az=73, radius=100.0, ground=31, clutter=1001, box=10.0, size=0.25,
              n_scat=501, freq=28e9, cell=0.5),
        # the default engine (cuda=False) on an ordinary scene, 2 degree sphere
        _scat("numba_bounce", side=16, n_el=91, n_az=181, radius=100.0, ground=100, clutter=10000, box=10.0,
              size=0.25, n_scat=5000, freq=28e9, cell=0.5, engine="numba"),
        # per-element fields of a small array with one bounce (what a beamforming tool asks for)
        _scat("elements_bounce", side=8, n_el=37, n_az=73, radius=100.0, ground=50, clutter=3000, box=10.0,
              size=0.25, n_scat=800, freq=28e9, cell=0.5, elements=True),
        # the 28 GHz direct + one-bounce scene of the package's benchmark
        _scat("bounce_28ghz", side=32, n_el=181, n_az=361, radius=100.0, ground=200, clutter=40000, box=10.0,
              size=0.25, n_scat=50000, freq=28e9, cell=0.5),
        # gradients of a pattern with respect to excitations, element and sink positions
        dict(_scat("adjoint_28ghz", side=16, n_el=181, n_az=181, radius=100.0, ground=200, clutter=40000, box=10.0,
                   size=0.25, n_scat=10000, freq=28e9, cell=0.5), kind="adjoint"),
        # the network of a 32 x 32 array at 2 degrees, formed once per design
        dict(_scat("network_28ghz", side=32, n_el=91, n_az=181, radius=100.0, ground=200, clutter=20000, box=10.0,
                   size=0.25, n_scat=0, freq=28e9, cell=0.5), kind="network"),
        # a full-resolution beam sweep of a 64 x 64 array, and a small one with odd sizes and FP16 halves
        dict(kind="sweep", name="sweep_28ghz", side=64, n_el=181, n_az=361, beams=2048, mode="bf16x3g", freq=28e9),
        dict(kind="sweep", name="sweep_small", side=31, n_el=37, n_az=73, beams=181, mode="fp16x3g", freq=28e9),
        # many uneven scenes at many frequencies in one launch
        dict(kind="batched", name="batched_8", scenes=8, elem_lo=16, elem_hi=4096, tri_lo=1000, tri_hi=100000,
             n_snk=4000, n_freq=16, max_scat=5000),
        # the numba engine's visibility sets, and the products of a list of direct and one-bounce paths
        dict(kind="paths", name="paths_one_bounce", n_src=16, n_snk=500, n_scat=200, clutter=2000, rows=300001,
             freq=2e9),
    ]


def _scat(name, side, n_el, n_az, radius, ground, clutter, box, size, n_scat, freq, cell, engine="cuda",
          elements=False):
    return dict(kind="scattering", name=name, side=side, n_el=n_el, n_az=n_az, radius=radius, ground=ground,
                clutter=clutter, box=box, size=size, n_scat=n_scat, freq=freq, cell=cell, engine=engine,
                elements=elements)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    c = _draw(rng)
    c.pop("name", None)
    return c


def _draw(rng):
    kind = rng.choice(["scattering", "scattering", "scattering", "brute", "network", "adjoint", "sweep", "batched",
                       "paths"])
    if kind == "sweep":
        mode = rng.choice(["bf16x3g", "fp16x3g"])
        n_el = _log(rng, 10, 181)
        return dict(kind=kind, side=_log(rng, 6, 64), n_el=n_el, n_az=2 * n_el - rng.randint(0, 2),
                    beams=_log(rng, 16, 2000), mode=mode, freq=28e9)
    if kind == "batched":
        return dict(kind=kind, scenes=rng.randint(2, 8), elem_lo=16, elem_hi=_log(rng, 64, 4096), tri_lo=1000,
                    tri_hi=_log(rng, 4000, 100000), n_snk=_log(rng, 500, 4000), n_freq=rng.randint(1, 16),
                    max_scat=_log(rng, 300, 5000))
    if kind == "paths":
        return dict(kind=kind, n_src=rng.randint(2, 16), n_snk=_log(rng, 30, 500), n_scat=_log(rng, 10, 200),
                    clutter=_log(rng, 100, 2000), rows=_log(rng, 1000, 300000), freq=2e9)
    n_el = _log(rng, 12, 181)
    n_az = 2 * n_el - rng.randint(-1, 3)
    if kind == "brute":
        n_el, n_az = _log(rng, 12, 91), _log(rng, 24, 181)
        return dict(_scat("d", side=rng.randint(3, 16), n_el=n_el, n_az=n_az, radius=10.0, ground=0,
                          clutter=_log(rng, 100, 4000), box=1.0, size=0.05, n_scat=0, freq=10e9, cell=0.0),
                    kind=kind)
    c = _scat("d", side=rng.randint(3, 32), n_el=n_el, n_az=n_az, radius=100.0, ground=_log(rng, 20, 200),
              clutter=_log(rng, 500, 40000), box=10.0, size=0.25, n_scat=_log(rng, 200, 50000), freq=28e9, cell=0.5,
              engine=rng.choice(["cuda", "cuda", "numba"]))
    if kind == "network":
        c.update(kind=kind, n_scat=0, side=rng.randint(3, 32), n_el=_log(rng, 12, 91), engine="cuda")
        c["n_az"] = 2 * c["n_el"] + rng.randint(-2, 2)
    elif kind == "adjoint":
        c.update(kind=kind, side=rng.randint(3, 16), n_scat=_log(rng, 100, 10000), engine="cuda")
    elif rng.random() < 0.25:  # per element: the networks travel to the host, so such calls are small
        c.update(elements=True, engine="cuda", side=rng.randint(2, 8), n_el=_log(rng, 12, 37),
                 n_scat=_log(rng, 100, 800))
        c["n_az"] = 2 * c["n_el"]
    return c


# ------------------------------------------------------------------ inputs

def _array(side, lam):
    p = (np.arange(side) - (side - 1) / 2.0) * lam / 2.0
    x, y = np.meshgrid(p, p, indexing="ij")
    pts = np.stack([x.ravel(), y.ravel(), np.zeros(side * side)], 1).astype(np.float32)
    return pts, np.tile(np.array([[0, 0, 1]], np.float32), (side * side, 1))


def _sphere(n_el, n_az, radius, closed):
    el = np.linspace(-np.pi / 2, np.pi / 2, n_el)
    az = np.linspace(-np.pi, np.pi, n_az, endpoint=closed)
    e, a = np.meshgrid(el, az, indexing="ij")
    d = np.stack([np.cos(e) * np.cos(a), np.cos(e) * np.sin(a), np.sin(e)], -1).reshape(-1, 3)
    return (radius * d).astype(np.float32), (-d).astype(np.float32)


def _mesh(rng, ground, clutter, box, size):
    """Clutter triangles in [-box, box]^2 x [0, box / 2] over a ground of ground^2 quads at -1 (box 1: clutter in
    [-1, 1]^2 x [0.5, 1.5], no ground)."""
    lo, hi = ((-box, -box, 0.0), (box, box, box / 2)) if box > 1.0 else ((-1, -1, 0.5), (1, 1, 1.5))
    c = np.asarray(lo) + (np.asarray(hi) - np.asarray(lo)) * rng.random((clutter, 3))
    v = (c[:, None] + rng.uniform(-size, size, (clutter, 3, 3))).reshape(-1, 3).astype(np.float32)
    f = np.arange(3 * clutter, dtype=np.int32).reshape(-1, 3)
    if ground:
        s = np.linspace(-box, box, ground + 1)
        x, y = np.meshgrid(s, s, indexing="ij")
        gv = np.stack([x.ravel(), y.ravel(), np.full(x.size, -1.0)], 1).astype(np.float32)
        i, j = np.meshgrid(np.arange(ground), np.arange(ground), indexing="ij")
        a, b = (i * (ground + 1) + j).ravel(), ((i + 1) * (ground + 1) + j).ravel()
        gf = np.concatenate([np.stack([a, b, b + 1], 1), np.stack([a, b + 1, a + 1], 1)]).astype(np.int32)
        v, f = np.concatenate([gv, v]), np.concatenate([gf, f + gv.shape[0]]).astype(np.int32)
    return v, f


def _scatter(rng, v, f, n):
    n = min(n, f.shape[0])
    t = v.astype(np.float64)[f[np.sort(rng.choice(f.shape[0], n, replace=False))]]
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-30)
    return (t.mean(1) + 1e-3 * nrm).astype(np.float32), nrm.astype(np.float32)


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    lam = C0 / case["freq"]
    s = {"lam": lam, "beta": 2 * np.pi / lam}
    s["src"], s["src_n"] = _array(case["side"], lam)
    s["snk"], s["snk_n"] = _sphere(case["n_el"], case["n_az"], case["radius"], case["box"] > 1.0)
    s["v"], s["f"] = _mesh(rng, case["ground"], case["clutter"], case["box"], case["size"])
    s["scat"], s["scat_n"] = _scatter(rng, s["v"], s["f"], case["n_scat"]) if case["n_scat"] else (None, None)
    n = s["src"].shape[0]
    s["w"] = np.exp(1j * rng.uniform(0, 2 * np.pi, n)).astype(np.complex64)  # a beam's unit-amplitude weights
    s["E"] = (s["w"][:, None] * np.array([[1, 0, 0]], np.complex64)).astype(np.complex64)
    s["g_rng"] = rng
    return s


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    # the sizes of the batch belong to the case, not to the seed
    srng = np.random.default_rng(case["scenes"] * 1000003 + case["tri_hi"] * 17 + case["n_snk"])
    lam = C0 / 27e9
    scenes = []
    for _ in range(case["scenes"]):
        ne = math.exp(srng.uniform(math.log(case["elem_lo"]), math.log(case["elem_hi"])))
        nt = int(math.exp(srng.uniform(math.log(case["tri_lo"]), math.log(case["tri_hi"]))))
        src, _ = _array(max(1, int(round(math.sqrt(ne)))), lam)
        g = max(1, int(math.sqrt(nt / 3.0)))
        v, f = _mesh(rng, g, max(1, nt - 2 * g * g), 10.0, 0.25)
        sc, sn = _scatter(rng, v, f, min(case["max_scat"], max(1, f.shape[0] // 10)))
        scenes.append(dict(src=src, verts=v, faces=f, scat=sc, scat_n=sn))
    i = np.arange(case["n_snk"]) + 0.5
    z = 1 - 2 * i / case["n_snk"]
    ph = np.pi * (3 - np.sqrt(5.0)) * i
    d = np.stack([np.sqrt(1 - z * z) * np.cos(ph), np.sqrt(1 - z * z) * np.sin(ph), z], 1)
    return scenes, (50 * d).astype(np.float32), (-d).astype(np.float32), np.linspace(24e9, 30e9, case["n_freq"])


def _path_scene(case, seed):
    rng = np.random.default_rng(seed)
    v, f = _mesh(rng, 0, case["clutter"], 2.0, 0.06)
    src = rng.uniform(-0.3, 0.3, (case["n_src"], 3)) + [0, 0, -1.0]
    snk = rng.uniform(-3, 3, (case["n_snk"], 3)) + [0, 0, 4.0]
    scat, scat_n = _scatter(rng, v, f, case["n_scat"])
    pos = np.concatenate([src, snk, scat]).astype(np.float32)
    nrm = rng.normal(size=(pos.shape[0], 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    nrm = nrm.astype(np.float32)
    nrm[-scat.shape[0]:] = scat_n
    w = np.ones((pos.shape[0], 3), np.complex64)
    n = case["n_src"]
    w[:n] = np.exp(1j * rng.uniform(0, 2 * np.pi, (n, 1))) * np.array([[1, 0.5, 0.25]])
    # path rows (1-based indices into sources, sinks, scatter points): a third direct, the others over one bounce
    m, ns, rows = case["n_snk"], scat.shape[0], case["rows"]
    idx = np.stack([rng.integers(0, n, rows) + 1, rng.integers(0, ns, rows) + n + m + 1,
                    rng.integers(0, m, rows) + n + 1], 1).astype(np.int32)
    idx[:rows // 3, 1], idx[:rows // 3, 2] = idx[:rows // 3, 2], 0
    return v, f, pos, nrm, w, ns, idx


def _network(case, seed):
    """Per-pair network of an array (plain torch): every second patch of sinks blocked, as behind clutter."""
    lam = C0 / case["freq"]
    src, _ = _array(case["side"], lam)
    snk, nrm = _sphere(case["n_el"], case["n_az"], 100.0, True)
    src, snk, nrm = (torch.from_numpy(a).cuda().double() for a in (src, snk, nrm))
    gen = torch.Generator("cuda").manual_seed(int(seed))
    patch = torch.rand((src.shape[0], (snk.shape[0] + 63) // 64), generator=gen, device="cuda") < 0.5
    out = torch.empty((src.shape[0], snk.shape[0], 3), dtype=torch.complex64, device="cuda")
    step = max(1, int(4e6 // snk.shape[0]))
    E = torch.tensor([1, 0, 0], dtype=torch.complex128, device="cuda")
    for a in range(0, src.shape[0], step):
        s = src[a:a + step]
        vis = patch[a:a + step].repeat_interleave(64, 1)[:, :snk.shape[0]]
        out[a:a + step] = _pair64(s, E.expand(s.shape[0], 3), snk, nrm, 0.0, 2 * np.pi / lam, vis).to(torch.complex64)
    W = torch.exp(1j * 2 * np.pi * torch.rand((case["beams"], src.shape[0]), generator=gen, device="cuda"))
    return out, W.to(torch.complex64)


def prepare(case, seed):
    from lyceanem_gb300 import batched, beam_sweep
    from lyceanem_gb300 import propagation as P
    from lyceanem_gb300.empropagation import scattering_point
    from lyceanem_gb300.geometry import Mesh
    from lyceanem_gb300.models.acceleration_structures import Tile_acceleration_structure
    kind = case["kind"]
    if kind == "sweep":
        net, W = _network(case, seed)
        return {"case": case, "sweep": beam_sweep.BeamSweep(net, mode=case["mode"]), "W": W}
    if kind == "batched":
        scenes, snk, snk_n, freqs = _batch(case, seed)
        return {"case": case, "batch": batched.BatchedScattering(scenes, snk, snk_n, freqs, cell_scale=1.5)}
    if kind == "paths":
        v, f, pos, nrm, w, ns, idx = _path_scene(case, seed)
        pts = np.zeros(pos.shape[0], scattering_point)
        for k, c in enumerate("xyz"):
            pts["p" + c], pts["n" + c], pts["e" + c] = pos[:, k], nrm[:, k], w[:, k]
        pts["Electric"] = True
        n, m = case["n_src"], case["n_snk"]
        return {"case": case, "env": (v, f), "pts": pts, "idx": idx, "src": pos[:n], "snk": pos[n:n + m], "scat": pos[n + m:]}
    s = _scene(case, seed)
    if kind == "scattering":
        solid = Mesh(s["v"], [("triangle", s["f"])])
        st = {"case": case, "solid": solid, "E": s["E"], "beta": s["beta"], "lam": s["lam"],
              "ap": Mesh(s["src"], point_data={"Normals": s["src_n"], "Area": np.ones(s["src"].shape[0], np.float32)}),
              "sk": Mesh(s["snk"], point_data={"Normals": s["snk_n"]}),
              "sc": None if s["scat"] is None else Mesh(s["scat"], point_data={"Normals": s["scat_n"]}),
              "acc": Tile_acceleration_structure(solid, 1, grid_cell=case["cell"] or None)}
        return st
    dev = {k: torch.from_numpy(s[k]).cuda() for k in ("src", "E", "snk", "snk_n", "w")}
    tris = P.pack_triangles(torch.from_numpy(s["v"]), torch.from_numpy(s["f"]))
    st = {"case": case, "beta": s["beta"], **dev}
    if kind == "brute":
        return {**st, "tris": tris}
    st["grid"] = P.UniformGrid(tris, cell=case["cell"] or None)
    if kind == "adjoint":
        st["scat"], st["scat_n"] = (torch.from_numpy(s[k]).cuda() for k in ("scat", "scat_n"))
        st["target"] = torch.from_numpy(_target(s)).cuda()
        st["pol"] = torch.tensor([1, 0, 0], dtype=torch.complex64, device="cuda")
    return st


def _target(s):
    """A seeded unit-amplitude pattern at the level of the array's field."""
    rng, m = s["g_rng"], s["snk"].shape[0]
    a = 0.1 * s["beta"] * s["src"].shape[0] ** 0.5 / 100.0
    return (a * np.exp(1j * rng.uniform(0, 2 * np.pi, (m, 3)))).astype(np.complex64)


# ------------------------------------------------------------------ one pass

def run(st):
    from lyceanem_gb300 import adjoint, beam_sweep, empropagation, raycasting
    from lyceanem_gb300 import propagation as P
    from lyceanem_gb300.models import frequency_domain as FD
    case = st["case"]
    kind = case["kind"]
    if kind == "scattering":
        return FD.calculate_scattering(st["ap"], st["sk"], st["solid"], st["E"], scatter_points=st["sc"],
                                       wavelength=st["lam"], scattering=int(st["sc"] is not None),
                                       elements=case["elements"], beta=st["beta"], cuda=case["engine"] == "cuda",
                                       acceleration_structure=st["acc"])
    if kind == "brute":
        r = P.pair_stage(st["src"], st["E"], st["snk"], st["snk_n"], beta=st["beta"], tris=st["tris"],
                         want_mask=True)
        return {"field": r.sink, "mask": r.mask()}
    if kind == "network":
        return beam_sweep.form_network(st["src"], st["E"], st["snk"], st["snk_n"], beta=st["beta"], grid=st["grid"])
    if kind == "adjoint":
        a, x, y = (st[k].clone().requires_grad_(True) for k in ("w", "src", "snk"))
        E = adjoint.sink_field(a, x, y, st["pol"], st["snk_n"], st["scat"], st["scat_n"], beta=st["beta"],
                               grid=st["grid"])
        d = E - st["target"]
        (d.real ** 2 + d.imag ** 2).sum().backward()
        return {"E": E.detach(), "a": a.grad, "x": x.grad, "y": y.grad}
    if kind == "sweep":
        return st["sweep"].fields(st["sweep"].run(st["W"]))
    if kind == "batched":
        return st["batch"].run()
    masks = raycasting.numba_masks(st["src"], st["snk"], st["scat"], st["env"])
    net = empropagation.EMGPUFreqDomain(case["n_src"], case["n_snk"], st["idx"], st["pts"], C0 / case["freq"], 0.0,
                                        2 * np.pi * case["freq"] / C0)
    return {"masks": masks[:3], "network": net}


def _sizes(case):
    if case["kind"] == "batched":
        scenes, snk, _, freqs = _batch(case, 0)
        return [(s["src"].shape[0], s["scat"].shape[0], snk.shape[0], s["faces"].shape[0]) for s in scenes]
    if case["kind"] == "paths":
        return [(case["n_src"], min(case["n_scat"], case["clutter"]), case["n_snk"], case["clutter"])]
    T = 2 * case["ground"] ** 2 + case["clutter"]
    return [(case["side"] ** 2, min(case["n_scat"], T), case["n_el"] * case["n_az"], T)]


def work(case):
    """Inputs read once and outputs written once; 30 flops (one ray-triangle test) per traced ray, 100 per pair of
    field (gradients twice that), 8 per complex multiply-add."""
    kind = case["kind"]
    if kind == "sweep":
        N, M, K = case["side"] ** 2, case["n_el"] * case["n_az"], case["beams"]
        return {"bytes": 24.0 * N * M + 8.0 * N * K + 24.0 * M * K, "flops": 24.0 * N * M * K}
    b = f = 0.0
    for N, Pn, M, T in _sizes(case):
        rays = N * M + N * Pn + Pn * M
        freqs = case.get("n_freq", 1)
        b += 48.0 * T + 36.0 * N + 24.0 * Pn + 24.0 * M + 24.0 * M * freqs
        f += rays * (30.0 + 100.0 * freqs)
        if kind == "network" or case.get("elements"):
            b += 24.0 * N * M
            f += 24.0 * N * Pn * M
        if kind == "adjoint":
            b += 20.0 * N + 12.0 * M
            f += rays * 200.0
        if kind == "paths":
            b += 48.0 * N * M + 12.0 * case["rows"] + N * M + N * Pn + Pn * M
            f += 200.0 * case["rows"] - 100.0 * rays
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64 bits

def _fma(a, b, c):
    """FP32 fma: the product of two FP32 values is exact in FP64."""
    return (a.double() * b.double() + c.double()).float()


def _visible(src, snk, v, f, culled, skip_same):
    """Visibility bool [N, M] by the ray-triangle test of the engines in its FP32 arithmetic (culling, 1e-6; or
    two-sided, 1e-7, FP64 after the determinant), brute force.  src, snk: float32 CUDA tensors."""
    eps = 1e-6 if culled else 1e-7
    t = torch.from_numpy(v).cuda()[torch.from_numpy(f).cuda().long()]
    v0, e1, e2 = t[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    N, M, T = src.shape[0], snk.shape[0], t.shape[0]
    out = torch.ones((N, M), dtype=torch.bool, device=src.device)
    step = max(1, int(3e7 // max(T, 1)))

    def cross(a, b):
        return [_fma(a[1], b[2], -(a[2] * b[1])), _fma(a[2], b[0], -(a[0] * b[2])), _fma(a[0], b[1], -(a[1] * b[0]))]

    def dot(a, b):
        return _fma(a[2], b[2], _fma(a[1], b[1], a[0] * b[0]))
    E1, E2 = [e1[None, :, k] for k in range(3)], [e2[None, :, k] for k in range(3)]
    for n in range(N):
        o = src[n]
        tv = [(o[k] - v0[:, k])[None] for k in range(3)]
        q = cross(tv, E1)
        w = dot(E2, q)
        for a in range(0, M, step):
            r = snk[a:a + step] - o
            if culled:
                ln = torch.sqrt(_fma(r[:, 2], r[:, 2], _fma(r[:, 1], r[:, 1], r[:, 0] * r[:, 0])))
            else:
                ln = torch.sqrt((r[:, 0] * r[:, 0] + r[:, 1] * r[:, 1]) + r[:, 2] * r[:, 2])
            d = [(r[:, k] / ln)[:, None] for k in range(3)]
            p = cross(d, E2)
            A = dot(E1, p)
            u, x = dot(tv, p), dot(d, q)
            if culled:
                ok, F = A >= eps, 1.0 / A
            else:
                ok, F = A.abs() >= eps, 1.0 / A.double()
            U, V, tt = F * u, F * x, F * w
            far = ln[:, None] - 2 * torch.tensor(eps, device=src.device) if culled else ln[:, None].double() - 2 * float(np.float32(eps))
            near = 2 * torch.tensor(eps, device=src.device) if culled else 2 * float(np.float32(eps))
            hit = ok & (U >= 0) & (U <= 1) & (V >= 0) & (U + V <= 1) & (tt > near) & (tt < far)
            out[n, a:a + step] = ~hit.any(1)
    if skip_same:
        k = min(N, M)
        out[torch.arange(k), torch.arange(k)] = True
    return out


def _pair64(src, E, snk, nrm, alpha, beta, vis):
    """Per-pair field complex128 [N, M, 3] of FP64 inputs (differentiable)."""
    rv = snk[None] - src[:, None]
    r = torch.sqrt((rv * rv).sum(-1))
    d = rv / r[..., None]
    loss = (alpha + 1 / r + 1j * beta) / (2 * np.pi) * torch.exp(-(alpha + 1j * beta) * r) / r
    loss = loss * (nrm[None] * d).sum(-1) * vis
    ed = (E[:, None] * d).sum(-1, keepdim=True)
    return (E[:, None] - ed * d) * loss[..., None]


def _project(v, n):
    u = n / torch.linalg.norm(n, dim=-1, keepdim=True)
    return v - (v * u).sum(-1, keepdim=True) * u


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        N, M, K = case["side"] ** 2, case["n_el"] * case["n_az"], case["beams"]
        if 24.0 * N * M * K > 2e12:
            return None
        net, W = _network(case, seed)
        Wd = W.to(torch.complex128)
        return torch.stack([(Wd @ net[:, :, c].to(torch.complex128)).T for c in range(3)], -1)
    if kind == "batched":
        return None  # visibility of every scene by brute force takes far too long
    if kind == "paths":
        return _exact_paths(case, seed)
    (N, Pn, M, T), = _sizes(case)
    rays = N * M + N * Pn + Pn * M
    if rays * T > EXACT_TESTS or rays > EXACT_PAIRS:
        return None
    s = _scene(case, seed)
    f32 = {k: torch.from_numpy(s[k]).cuda() for k in ("src", "snk", "snk_n", "scat", "scat_n") if s[k] is not None}
    d = {k: a.double() for k, a in f32.items()}
    numba = kind == "scattering" and case["engine"] == "numba"
    beta = float(np.float32(s["beta"])) if kind == "scattering" and not numba else s["beta"]
    same = not numba and kind != "network"
    E = torch.from_numpy(s["E"]).cuda().to(torch.complex128)
    if numba and Pn:  # that engine repeats the first row's real part
        E = E[0].real.expand(N, 3).to(torch.complex128)

    def vis(a, b):
        return _visible(f32[a], f32[b], s["v"], s["f"], not numba, same)

    def stage(a, e, b, m, W=None):
        """Source sum of W (.) S, chunked over the sources."""
        out = torch.zeros((d[b].shape[0], 3), dtype=torch.complex128, device="cuda")
        step = max(1, int(2e6 // d[b].shape[0]))
        for i in range(0, d[a].shape[0], step):
            S = _pair64(d[a][i:i + step], e[i:i + step], d[b], d[b + "_n"], 0.0, beta, m[i:i + step])
            out += (S if W is None else W[i:i + step, None] * S).sum(0)
        return out

    m0 = vis("src", "snk")
    if kind == "brute":
        return {"field": stage("src", E, "snk", m0), "mask": None}
    if kind == "network":
        return _pair64(d["src"], E, d["snk"], d["snk_n"], 0.0, beta, m0)
    if Pn:
        m1, m2 = vis("src", "scat"), vis("scat", "snk")
    if kind == "adjoint":
        a = torch.from_numpy(s["w"]).cuda().to(torch.complex128).requires_grad_(True)
        x, y = d["src"].clone().requires_grad_(True), d["snk"].clone().requires_grad_(True)
        pol = torch.tensor([1, 0, 0], dtype=torch.complex128, device="cuda")
        e = a[:, None] * pol
        field = _pair64(x, e, y, d["snk_n"], 0.0, beta, m0).sum(0)
        wp = _pair64(x, e, d["scat"], d["scat_n"], 0.0, beta, m1).sum(0)
        field = field + (wp[:, None] * _pair64(d["scat"], wp, y, d["snk_n"], 0.0, beta, m2)).sum(0)
        diff = field - torch.from_numpy(_target(s)).cuda()
        (diff.real ** 2 + diff.imag ** 2).sum().backward()
        return {"E": field.detach(), "a": a.grad, "x": x.grad, "y": y.grad}
    if case["elements"]:
        S = _pair64(d["src"], E, d["snk"], d["snk_n"], 0.0, beta, m0)
        if Pn:
            S1 = _pair64(d["src"], E, d["scat"], d["scat_n"], 0.0, beta, m1)
            S2 = _pair64(d["scat"], S1.sum(0), d["snk"], d["snk_n"], 0.0, beta, m2)
            S = S + torch.stack([S1[:, :, c] @ S2[:, :, c] for c in range(3)], -1)
        return tuple(S[:, :, c].contiguous() for c in range(3))
    out = stage("src", E, "snk", m0)
    if Pn:
        e_p = stage("src", E, "scat", m1)
        if numba:
            out = _project(out, d["snk_n"])
            out = out + stage("scat", _project(e_p, d["scat_n"]), "snk", m2)
        else:
            out = out + stage("scat", e_p, "snk", m2, e_p)
    return tuple(out[:, c].contiguous() for c in range(3))


def _exact_paths(case, seed):
    """The products of the listed paths summed per (source, sink): direct rows projected at the sink, one-bounce rows
    at the scatter point; a row's visibility is the caller's."""
    v, f, pos, nrm, w, ns, idx = _path_scene(case, seed)
    n, m, beta = case["n_src"], case["n_snk"], 2 * np.pi * case["freq"] / C0
    p, nr = torch.from_numpy(pos).cuda().double(), torch.from_numpy(nrm).cuda().double()
    w, idx = torch.from_numpy(w).cuda().to(torch.complex128), torch.from_numpy(idx).cuda().long() - 1

    def segment(a, b, e):
        r = torch.linalg.norm(p[b] - p[a], dim=1)
        d = (p[b] - p[a]) / r[:, None]
        loss = (1 / r + 1j * beta) / (2 * np.pi) * torch.exp(-1j * beta * r) / r * (nr[b] * d).sum(1)
        return (e - (e * d).sum(1, keepdim=True) * d) * loss[:, None]
    net = torch.zeros((n * m, 3), dtype=torch.complex128, device="cuda")
    k = case["rows"] // 3
    a, b = idx[:k, 0], idx[:k, 1]
    net.index_add_(0, a * m + b - n, _project(segment(a, b, w[a]), nr[b]))
    a, q, b = idx[k:, 0], idx[k:, 1], idx[k:, 2]
    net.index_add_(0, a * m + b - n, segment(q, b, _project(segment(a, q, w[a]), nr[q])))
    return {"masks": None, "network": net.reshape(n, m, 3)}
