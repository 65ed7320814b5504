"""GPU parity of the batched many-scene, many-frequency launch.

Against the FP64 oracle (per scene, per frequency, direct + one bounce of
calculate_scattering_cuda summed over sources) within 1e-5 max-normalised
relative error, with the visible-pair counters equal to the oracle's mask
counts; against the per-scene pair-stage path on a larger batch; every
frequency grouping agrees; the captured graph reproduces the eager launch bit
for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

from helpers import rel_err

pytestmark = pytest.mark.gpu

FIELD_TOL = 1e-5


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from lyceanem_gb300 import build
    build.build_native()


def _mods():
    from lyceanem_gb300 import batched as B
    from lyceanem_gb300 import propagation as P
    from lyceanem_gb300 import scenes as SC
    return B, P, SC


def _scene(SC, rng, side, n_clutter, n_ground, n_scat, lam):
    src, _ = SC.planar_array(side, side, lam)
    g = SC.ground_plane(20.0, n_ground, -1.0)
    cl = SC.random_triangles(rng, n_clutter, (-10, -10, 0.0), (10, 10, 5.0), 0.25)
    verts, faces = SC.merge(g, cl)
    E = (rng.normal(size=(src.shape[0], 3)) + 1j * rng.normal(size=(src.shape[0], 3))).astype(np.complex64)
    sc = SC.Scene(src=src, E=E, verts=verts, faces=faces)
    if n_scat:
        sc.scat, sc.scat_n = SC.scatter_points(rng, verts, faces, n_scat)
    else:
        sc.scat = np.zeros((0, 3), np.float32)
        sc.scat_n = np.zeros((0, 3), np.float32)
    return sc


def _small_batch(seed=11, n_snk=250):
    B, P, SC = _mods()
    rng = np.random.default_rng(seed)
    lam = B.C0 / 27e9
    scenes = [_scene(SC, rng, 4, 120, 6, 60, lam), _scene(SC, rng, 7, 300, 10, 150, lam),
              _scene(SC, rng, 3, 50, 2, 0, lam)]
    snk, snk_n = SC.fibonacci_sinks(50.0, n_snk)
    return scenes, snk, snk_n


def _oracle(scenes, snk, snk_n, betas):
    """complex128 [S, F, M, 3] and visible counts [S, 3] (sources->scatter, sources->sinks, scatter->sinks)."""
    out = np.zeros((len(scenes), len(betas), snk.shape[0], 3), np.complex128)
    counts = np.zeros((len(scenes), 3), np.int64)
    for s, sc in enumerate(scenes):
        t12 = O.pack_triangles(sc.verts, sc.faces)
        m0 = O.mask_brute(sc.src, snk, t12)
        counts[s, 1] = m0.sum()
        P_ = sc.scat.shape[0]
        if P_:
            m1 = O.mask_brute(sc.src, sc.scat, t12)
            m2 = O.mask_brute(sc.scat, snk, t12)
            counts[s, 0], counts[s, 2] = m1.sum(), m2.sum()
        for f, b in enumerate(betas):
            e = O.sink_field(sc.src, sc.E, snk, snk_n, 0.0, b, mask=m0)
            if P_:
                ep = O.sink_field(sc.src, sc.E, sc.scat, sc.scat_n, 0.0, b, mask=m1)
                e = e + O.sink_field(sc.scat, ep, snk, snk_n, 0.0, b, srcW=ep, mask=m2)
            out[s, f] = e
    return out, counts


def _check(field, ref):
    worst = 0.0
    for s in range(ref.shape[0]):
        for f in range(ref.shape[1]):
            worst = max(worst, rel_err(field[s, f], ref[s, f]))
    return worst


@pytest.fixture(scope="module")
def small():
    B, _, _ = _mods()
    scenes, snk, snk_n = _small_batch()
    freqs = np.linspace(24e9, 30e9, 8)
    betas = B.betas_of(freqs)
    ref, counts = _oracle(scenes, snk, snk_n, betas)
    return scenes, snk, snk_n, freqs, ref, counts


@pytest.mark.parametrize("config", [(1, 32, 0), (2, 64, 0), (4, 32, 0), (8, 64, 1)])
def test_batched_vs_oracle(small, config):
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, ref, counts = small
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs, config=config)
    field = bs.run().cpu().numpy()
    st, flags = P.device_errors()
    assert st == 0 and flags == 0, f"device error word {flags:#x}"
    err = _check(field, ref)
    assert err < FIELD_TOL, f"config {config}: field error {err:.3e}"
    assert np.array_equal(bs.counters.cpu().numpy()[:, :3], counts)


def test_nonuniform_frequencies(small):
    B, P, _ = _mods()
    scenes, snk, snk_n, _, _, _ = small
    freqs = np.array([24.0e9, 24.7e9, 26.1e9, 29.95e9, 27.3e9])
    with pytest.raises(ValueError):
        B.BatchedScattering(scenes, snk, snk_n, freqs, config=(4, 32, 0))
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs)
    assert bs.config[0] == 1
    ref, _ = _oracle(scenes, snk, snk_n, B.betas_of(freqs))
    err = _check(bs.run().cpu().numpy(), ref)
    assert err < FIELD_TOL, f"field error {err:.3e}"
    assert P.device_errors() == (0, 0)


def test_graph_replay_and_groupings_agree(small):
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, _, _ = small
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs, config=(4, 64, 0))
    eager = bs.run().clone()
    bs.capture()
    bs.field.zero_()
    for _ in range(3):
        replay = bs.run()
    torch.cuda.synchronize()
    assert torch.equal(replay, eager)  # each output element has one writer and a fixed summation order
    bs.configure((8, 32, 0))
    other = bs.run().clone()
    assert rel_err(other.cpu().numpy(), eager.cpu().numpy()) < 2e-6
    assert P.device_errors() == (0, 0)


def test_batched_vs_pair_stages():
    """A larger batch against the per-scene, per-frequency pair-stage path (FP64 phase)."""
    B, P, SC = _mods()
    rng = np.random.default_rng(5)
    lam = B.C0 / 27e9
    scenes = [_scene(SC, rng, 16, 1500, 20, 700, lam), _scene(SC, rng, 10, 4000, 30, 1200, lam)]
    snk, snk_n = SC.fibonacci_sinks(50.0, 3000)
    freqs = np.linspace(24e9, 30e9, 16)
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs, config=(8, 32, 0))
    field = bs.run().cpu().numpy()
    for s, sc in enumerate(scenes):
        d = bs.data[s]
        for f in (0, 7, 15):
            beta = float(bs.betas[f])
            kw = dict(grid=d.grid, alpha=0.0, beta=beta, self_to_self=False)
            scat = torch.from_numpy(sc.scat).cuda()
            scat_n = torch.from_numpy(sc.scat_n).cuda()
            out = P.pair_stage(sc.src, sc.E, snk, snk_n, **kw).sink
            ep = P.pair_stage(sc.src, sc.E, scat, scat_n, **kw).sink
            P.pair_stage(scat, ep, snk, snk_n, src_W=ep, sink_out=out, accumulate=True, **kw)
            err = rel_err(field[s, f], out.cpu().numpy())
            assert err < FIELD_TOL, f"scene {s} frequency {f}: {err:.3e}"
    assert P.device_errors() == (0, 0)


@pytest.mark.parametrize("config", [(4, 64, 8), (4, 32, 8), (4, 32, 3), (2, 32, 6), (1, 64, 8), (8, 64, 3)])
def test_register_capped_variants_vs_oracle(small, config):
    """The variants of the kernel that are capped for an occupancy give the oracle's field and visible pairs."""
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, ref, counts = small
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs, config=config)
    assert _check(bs.run().cpu().numpy(), ref) < FIELD_TOL
    assert np.array_equal(bs.counters.cpu().numpy()[:, :3], counts)
    assert P.device_errors() == (0, 0)


def test_autotune_picks_and_caches(small, tmp_path, monkeypatch):
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, ref, _ = small
    monkeypatch.setenv("LYEM_TUNE_CACHE", str(tmp_path / "tune.json"))
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs)
    proxy = B.BatchedScattering([scenes[i] for i in B.stratified_subset(scenes, snk.shape[0], every=2)], snk, snk_n,
                                freqs)
    cands = [(4, 32, 4), (2, 64, 0)]
    res = bs.autotune(candidates=cands, proxy=proxy)
    assert set(res) == set(cands) and bs.config == min(res, key=res.get)
    again = B.BatchedScattering(scenes, snk, snk_n, freqs)
    cached = again.autotune(candidates=cands)
    assert list(cached) == [bs.config] and again.config == bs.config
    assert _check(again.run().cpu().numpy(), ref) < FIELD_TOL
    assert P.device_errors() == (0, 0)


def test_autotune_cache_is_of_these_candidates_and_this_kernel(small, tmp_path, monkeypatch):
    """A choice that was made among other candidates, or timed on another revision of the kernel, is not taken."""
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, ref, _ = small
    monkeypatch.setenv("LYEM_TUNE_CACHE", str(tmp_path / "tune.json"))
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs)
    assert set(bs.autotune(candidates=[(2, 64, 8)])) == {(2, 64, 8)}
    assert set(bs.autotune(candidates=[(1, 32, 4), (4, 32, 4)])) == {(1, 32, 4), (4, 32, 4)}
    assert bs.config in ((1, 32, 4), (4, 32, 4))
    assert list(bs.autotune(candidates=[(4, 32, 4), (1, 32, 4)])) == [bs.config]  # the same ones: from the cache
    monkeypatch.setattr(B, "KERNEL_REVISION", B.KERNEL_REVISION + 1)
    assert len(bs.autotune(candidates=[(1, 32, 4), (4, 32, 4)])) == 2
    assert _check(bs.run().cpu().numpy(), ref) < FIELD_TOL
    assert P.device_errors() == (0, 0)


def test_density_cells_same_field(small, tmp_path, monkeypatch):
    """Density-scaled grids (one scale for the batch, a cell per scene) change only the traversal
    work: the same visible paths and fields as the oracle; the autotuner picks a scale."""
    B, P, _ = _mods()
    scenes, snk, snk_n, freqs, ref, counts = small
    tests = []
    for k in (0.6, 1.0, 1.7):
        bs = B.BatchedScattering(scenes, snk, snk_n, freqs, config=(2, 64, 0), cell_scale=k)
        cells = bs.grid_cells()
        assert len(set(round(c, 6) for c in cells)) > 1  # scenes of different density get different cells
        field = bs.run().cpu().numpy()
        assert _check(field, ref) < FIELD_TOL, f"scale {k}"
        cnt = bs.counters.cpu().numpy()
        assert np.array_equal(cnt[:, :3], counts), f"scale {k}"
        tests.append(int(cnt[:, 3].sum()))
    assert tests[0] != tests[2]
    monkeypatch.setenv("LYEM_TUNE_CACHE", str(tmp_path / "tune.json"))
    bs = B.BatchedScattering(scenes, snk, snk_n, freqs)
    res = bs.autotune(candidates=[(2, 64, 0), (4, 32, 4)], cell_scales=[0.8, 1.2])
    assert len(res) == 4 and all(len(k) == 4 for k in res)
    best = min(res, key=res.get)
    assert bs.config + (bs.cell_scale,) == best
    assert _check(bs.run().cpu().numpy(), ref) < FIELD_TOL
    again = B.BatchedScattering(scenes, snk, snk_n, freqs)
    cached = again.autotune(candidates=[(2, 64, 0), (4, 32, 4)], cell_scales=[0.8, 1.2])
    assert list(cached) == [best] and again.cell_scale == best[3] and again.grid_cells() == bs.grid_cells()
    assert P.device_errors() == (0, 0)


@pytest.mark.parametrize("copies", [1, 8, 30, 60])
@pytest.mark.parametrize("n_snk", [250, 2100])
def test_split_visibility_items(copies, n_snk):
    """Launches whose visibility items are split into 32, 4, 2 and no parts (the copies of one scene set how many
    items there are), with few sinks (every item turned) and more (scatter items in lockstep where not split): every
    copy gives the counts and the field of the per-scene pair stages."""
    B, P, SC = _mods()
    rng = np.random.default_rng(7)
    sc = _scene(SC, rng, 8, 200, 8, 150, B.C0 / 27e9)
    snk, snk_n = SC.fibonacci_sinks(50.0, n_snk)
    b = B.BatchedScattering([sc] * copies, snk, snk_n, [27e9], cell_scale=1.5, config=(4, 32, 3))
    field = b.run().cpu().numpy()
    counts = b.counters.cpu().numpy()
    beta = float(B.betas_of([27e9])[0])
    kw = dict(beta=beta, tris=P.pack_triangles(sc.verts, sc.faces))
    cnt = torch.zeros((3, 2), dtype=torch.int64, device="cuda")
    e_p = P.pair_stage(sc.src, sc.E, sc.scat, sc.scat_n, counters=cnt[0], **kw).sink
    out = P.pair_stage(sc.src, sc.E, snk, snk_n, counters=cnt[1], **kw).sink
    P.pair_stage(sc.scat, e_p, snk, snk_n, src_W=e_p, sink_out=out, accumulate=True, counters=cnt[2], **kw)
    assert (counts[:, :3] == cnt[:, 0].cpu().numpy()).all()
    for s in range(copies):
        assert rel_err(field[s, 0], out.cpu().numpy()) < 2e-6  # FP32 sums of up to 150 terms in two orders
    st, flags = P.device_errors()
    assert st == 0 and flags == 0


@pytest.mark.parametrize("fg,n_freq", [(1, 1), (1, 2), (1, 3), (1, 4), (1, 5), (1, 8), (1, 9), (1, 17), (1, 31), (1, 32),
                                       (1, 33), (1, 65), (2, 8), (2, 9), (2, 17), (2, 61), (4, 16), (4, 24), (8, 41)])
def test_shared_pair_setup(fg, n_freq):
    """Frequency groups on both sides of the line from which the lanes of a sink share its pairs' set-up instead of its
    sources, and that split a warp between slices or sinks unevenly: first, middle and last frequency against the
    per-scene pair stages."""
    B, P, SC = _mods()
    scenes, snk, snk_n = _small_batch(n_snk=83)
    freqs = np.linspace(25e9, 29e9, n_freq) if n_freq > 1 else np.array([27e9])
    b = B.BatchedScattering(scenes, snk, snk_n, freqs, cell_scale=1.5, config=(fg, 32, 4))
    field = b.run().cpu().numpy()
    betas = B.betas_of(freqs)
    for s, sc in enumerate(scenes):
        tris = P.pack_triangles(sc.verts, sc.faces)
        for f in sorted({0, n_freq // 2, n_freq - 1}):
            kw = dict(beta=float(betas[f]), tris=tris)
            out = P.pair_stage(sc.src, sc.E, snk, snk_n, **kw).sink
            if len(sc.scat):
                e_p = P.pair_stage(sc.src, sc.E, sc.scat, sc.scat_n, **kw).sink
                P.pair_stage(sc.scat, e_p, snk, snk_n, src_W=e_p, sink_out=out, accumulate=True, **kw)
            assert rel_err(field[s, f], out.cpu().numpy()) < 2e-6  # FP32 sums of up to 150 terms in two orders
    assert P.device_errors() == (0, 0)
