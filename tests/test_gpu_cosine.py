"""Greedy cosine on the GPU vs the oracle: bit-exact score, matches, overflow.

The oracle's float64 mode restates matchms CosineGreedy (the reference's
float64 target); its norms and score sums are taken in the same order as the
kernels', so all three outputs are compared bit for bit (which is stricter
than the 1e-5 score tolerance the specification asks for).
"""
import numpy as np
import pytest

from conftest import (assert_same, golden_cosine_cases, gpu_dense, gpu_plain, load_cosine_case)
from oracle import oracle

pytestmark = pytest.mark.gpu

CONFIGS = [None, {"mode": 2}, {"mode": 1, "tile_spectra": 32}, {"mode": 1, "tile_spectra": 4096},
           {"mode": 1, "bucket_width": 0.75}, {"mode": 1, "n_buckets": 1024},
           {"mode": 2, "pair_threads": 512}]


def P(tol, ml, n_max=1024, shift=0.0):
    return {"tolerance": tol, "shift": shift, "match_limit": ml, "n_max_peaks": n_max}


@pytest.mark.parametrize("name", golden_cosine_cases())
def test_fast_vs_oracle_golden(cuda_device, name):
    ref, qry, p, _ = load_cosine_case(name)
    want = oracle.cosine_greedy(ref, qry, p["tolerance"], p["shift"], p["match_limit"])
    for cfg in CONFIGS:
        assert_same(gpu_dense(ref, qry, p, cfg), want, f"{name} {cfg}")


@pytest.mark.parametrize("name", golden_cosine_cases())
def test_plain_vs_oracle_golden(cuda_device, name):
    ref, qry, p, _ = load_cosine_case(name)
    want = oracle.cosine_greedy(ref, qry, p["tolerance"], p["shift"], p["match_limit"])
    assert_same(gpu_plain(ref, qry, p), want, name)


def test_uniform_ragged_tiles(cuda_device):
    """1024x1024-config distribution at ragged sizes (tile edges, partial warps)."""
    from cudams import synthetic

    ref = synthetic.uniform_spectra(301, seed=1)
    qry = synthetic.uniform_spectra(257, seed=2)
    p = P(0.1, 2048)
    want = oracle.cosine_greedy(ref, qry, 0.1, 0.0, 2048)
    for cfg in CONFIGS:
        assert_same(gpu_dense(ref, qry, p, cfg), want, str(cfg))
    assert_same(gpu_plain(ref, qry, p), want, "plain")


def test_lognormal_heavy_tail(cuda_device):
    """100k-config distribution (heavy-tailed peak counts, tol 0.01), 1500 x 1200."""
    from cudams import synthetic

    ref = synthetic.lognormal_spectra(1500, seed=3)
    qry = synthetic.lognormal_spectra(1200, seed=4)
    p = P(0.01, 4096)
    want = oracle.cosine_greedy(ref, qry, 0.01, 0.0, 4096)
    assert_same(gpu_dense(ref, qry, p), want, "auto")
    assert_same(gpu_dense(ref, qry, p, {"mode": 1, "tile_spectra": 4096}), want, "tile4096")


def test_per_class_widths(cuda_device):
    """Per-length-class first sub-range widths (the tuner's per-bucket choice):
    narrow, odd and whole-tile widths for different classes, results
    bit-exact."""
    from cudams import synthetic

    ref = synthetic.lognormal_spectra(900, seed=13)
    qry = synthetic.lognormal_spectra(1100, seed=14)
    p = P(0.01, 4096)
    want = oracle.cosine_greedy(ref, qry, 0.01, 0.0, 4096)
    widths = [0] * 17
    widths[5], widths[6], widths[7], widths[8], widths[9], widths[10] = 32, 1, 96, 1024, 64, 7
    assert_same(gpu_dense(ref, qry, p, {"mode": 1, "tile_spectra": 1024,
                                        "width_by_class": widths}), want, "widths")


def test_measured_tuner_config(cuda_device, tmp_path):
    """Tuner.measure times tiles and per-bucket widths on the device, records
    them, and the chosen config computes the oracle's results."""
    from cudams import autotune, synthetic

    ref = synthetic.lognormal_spectra(3000, seed=15)
    qry = synthetic.lognormal_spectra(2500, seed=16)
    t = autotune.Tuner(str(tmp_path / "tune.json"))
    cfg, report = t.measure(ref, qry, 0.01, 0.0, 4096, device=cuda_device, sample_ref=1000,
                            tiles_per_trial=2)  # a torch.device, as bench.py passes it
    assert cfg["mode"] == 1 and len(cfg["width_by_class"]) == 17
    assert report["trials"] and report["buckets"]
    st = autotune.workload_stats(ref, qry, 0.01)
    assert t.lookup(st, "B200", qry.n, ref.n) == cfg
    want = oracle.cosine_greedy(ref, qry, 0.01, 0.0, 4096)
    assert_same(gpu_dense(ref, qry, P(0.01, 4096), cfg), want, "measured")


def test_clustered_overflow(cuda_device):
    """Overflow-stress distribution: ~all pairs reach match_limit; flags and counts exact."""
    from cudams import synthetic

    ref = synthetic.clustered_spectra(24, seed=5)
    qry = synthetic.clustered_spectra(20, seed=6)
    p = P(0.05, 1024, 2048)
    want = oracle.cosine_greedy(ref, qry, 0.05, 0.0, 1024)
    assert want[2].mean() > 0.9
    assert_same(gpu_dense(ref, qry, p, {"mode": 2}), want, "mode2")
    assert_same(gpu_dense(ref, qry, p, {"mode": 1, "tile_spectra": 32}), want, "mode1")
    assert_same(gpu_plain(ref, qry, p), want, "plain")


@pytest.mark.parametrize("ml, threads", [(512, 64), (1024, 128), (2048, 256), (4096, 512),
                                         (1000, 128), (700, 64)])
def test_pair_kernel_register_sort(cuda_device, ml, threads):
    """The pair kernel sorts in registers when a pair's padded candidate count
    is eight per thread (pairs that fill match_limit with threads = cap / 8),
    and in shared memory otherwise; both bit-exact.  Clustered spectra fill any
    of these limits; a few empty and short spectra give small pairs too."""
    from cudams import synthetic
    from cudams.packing import PackedSpectra

    ref = synthetic.clustered_spectra(18, seed=7, min_peaks=600, max_peaks=1500)
    qry = synthetic.clustered_spectra(14, seed=8, min_peaks=600, max_peaks=1500)
    # append a 3-peak and an empty query so that some pairs are tiny
    mz = np.concatenate([qry.mz, np.array([100.0, 200.0, 300.0], np.float32)])
    b = np.concatenate([qry.b, np.array([1.0, 0.5, 0.25])])
    a = None if qry.a is None else np.concatenate([qry.a, np.ones(3)])
    off = np.concatenate([qry.offsets, [qry.offsets[-1] + 3, qry.offsets[-1] + 3]])
    qry2 = PackedSpectra(mz, a, b, off.astype(np.int64), qry.mz_power, qry.intensity_power,
                         qry.n_max_peaks)
    p = P(0.05, ml, 2048)
    want = oracle.cosine_greedy(ref, qry2, 0.05, 0.0, ml)
    assert want[2].mean() > 0.5
    assert_same(gpu_dense(ref, qry2, p, {"mode": 2, "pair_threads": threads}), want,
                f"ml {ml} threads {threads}")
    assert_same(gpu_dense(ref, qry2, p, {"mode": 2}), want, f"ml {ml} auto threads")


def _block_spectra(n, seed, levels):
    """Spectra of 50 tight groups of 20 peaks (every peak of a group within
    0.01 of the others) with intensities drawn from `levels`: one intensity
    level gives all-equal keys, ordered by generation alone."""
    from cudams.packing import PackedSpectra

    rng = np.random.default_rng(seed)
    centres = 100.0 + 10.0 * np.arange(50)
    mz, b, off = [], [], [0]
    for _ in range(n):
        m = np.sort((np.repeat(centres, 20) + rng.uniform(-0.004, 0.004, 1000)).astype(np.float32))
        mz.append(m)
        b.append(rng.choice(np.asarray(levels, np.float64), m.shape[0]))
        off.append(off[-1] + m.shape[0])
    return PackedSpectra(np.concatenate(mz), None, np.concatenate(b),
                         np.asarray(off, np.int64), 0.0, 1.0, 2048)


@pytest.mark.parametrize("levels", [[1.0], [0.25, 0.5, 1.0], None])
@pytest.mark.parametrize("ml", [1024, 2048])
def test_pair_kernel_equal_keys(cuda_device, levels, ml):
    """Blocks of 20 x 20 candidates per peak group with all-equal keys (the
    order is generation alone), a few intensity levels (many ties broken by
    generation) or distinct keys (None): bit-exact through the whole-matrix
    pair kernel (register and shared-memory sorts) and through spills."""
    lv = levels if levels is not None else list(np.linspace(0.01, 1.0, 997))
    ref = _block_spectra(5, 30 + ml, lv)
    qry = _block_spectra(4, 40 + ml, lv)
    p = P(0.01, ml, 2048)
    want = oracle.cosine_greedy(ref, qry, 0.01, 0.0, ml)
    assert want[2].mean() > 0.5
    assert_same(gpu_dense(ref, qry, p, {"mode": 2}), want, f"mode2 {levels}")
    assert_same(gpu_dense(ref, qry, p, {"mode": 2, "pair_threads": 64}), want, f"64 {levels}")
    assert_same(gpu_dense(ref, qry, p, {"mode": 1, "tile_spectra": 32}), want, f"spill {levels}")


def test_self_similarity_spills(cuda_device):
    """Identical sets: diagonal pairs have one candidate per peak (long runs ->
    pair kernel), off-diagonal pairs few; both paths must agree."""
    from cudams import synthetic

    s = synthetic.uniform_spectra(200, seed=7)
    p = P(0.1, 2048)
    want = oracle.cosine_greedy(s, s, 0.1, 0.0, 2048)
    assert_same(gpu_dense(s, s, p), want, "auto")
    assert_same(gpu_dense(s, s, p, {"mode": 1, "tile_spectra": 4096}), want, "tile4096")
    d = np.diagonal(want[0])
    assert np.allclose(d, 1.0, atol=1e-6)


def test_pool_overflow_split(cuda_device):
    """Wide tolerance: ~50 candidates per pair, so a 4096-query tile overflows
    the 256-entry pool and the join must split the range down to single pairs."""
    from cudams import synthetic

    ref = synthetic.uniform_spectra(64, seed=8)
    qry = synthetic.uniform_spectra(300, seed=9)
    p = P(2.0, 2048)
    want = oracle.cosine_greedy(ref, qry, 2.0, 0.0, 2048)
    assert_same(gpu_dense(ref, qry, p, {"mode": 1, "tile_spectra": 4096}), want, "split")


def test_small_match_limit(cuda_device):
    """match_limit below typical candidate counts: runs >= limit go to the pair kernel."""
    from cudams import synthetic

    ref = synthetic.uniform_spectra(50, seed=10)
    qry = synthetic.uniform_spectra(40, seed=11)
    for ml in (1, 2, 3, 7):
        p = P(0.5, ml)
        want = oracle.cosine_greedy(ref, qry, 0.5, 0.0, ml)
        assert_same(gpu_dense(ref, qry, p), want, f"ml={ml}")
        assert_same(gpu_plain(ref, qry, p), want, f"plain ml={ml}")


def test_edge_spectra(cuda_device):
    """Empty spectra, single peaks, duplicate m/z, exact tolerance edges."""
    from cudams.packing import pack_spectra

    spectra = [
        (np.zeros(0), np.zeros(0)),
        (np.array([100.0]), np.array([1.0])),
        (np.array([100.0, 100.0, 100.0]), np.array([0.5, 1.0, 0.5])),
        (np.array([99.9, 100.1, 100.2]), np.array([1.0, 1.0, 1.0])),
        (np.array([50.0, 1000.0]), np.array([0.0, 1.0])),
    ]
    s = pack_spectra(spectra, 16)
    for tol in (0.0, 0.1, 0.2, 5.0):
        p = P(tol, 64, 16)
        want = oracle.cosine_greedy(s, s, tol, 0.0, 64)
        for cfg in CONFIGS:
            assert_same(gpu_dense(s, s, p, cfg), want, f"tol={tol} {cfg}")
        assert_same(gpu_plain(s, s, p), want, f"plain tol={tol}")


def test_powers_and_shift(cuda_device):
    from cudams import synthetic

    ref = synthetic.uniform_spectra(90, seed=12, mz_power=0.5, intensity_power=2.0)
    qry = synthetic.uniform_spectra(70, seed=13, mz_power=0.5, intensity_power=2.0)
    for shift in (0.0, 0.5, -1.25):
        p = P(0.3, 2048, shift=shift)
        want = oracle.cosine_greedy(ref, qry, 0.3, shift, 2048)
        for cfg in CONFIGS:
            assert_same(gpu_dense(ref, qry, p, cfg), want, f"shift={shift} {cfg}")


def test_long_spectra(cuda_device):
    """Spectra near the 16-bit peak-index limit."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(14)
    n = [65535, 3000, 7]
    mz = np.concatenate([np.sort(rng.uniform(50, 2000, k)) for k in n])
    it = rng.uniform(0.1, 1.0, mz.shape[0])
    off = np.concatenate([[0], np.cumsum(n)])
    s = pack_csr(mz, it, off, None)
    p = P(0.01, 4096, 65535)
    want = oracle.cosine_greedy(s, s, 0.01, 0.0, 4096)
    assert_same(gpu_dense(s, s, p), want, "auto")
    assert_same(gpu_dense(s, s, p, {"mode": 2}), want, "mode2")


def test_sparse_equals_dense_filtered(cuda_device):
    import torch

    from cudams import kernels, synthetic

    ref = synthetic.uniform_spectra(400, seed=15)
    qry = synthetic.uniform_spectra(350, seed=16)
    want = oracle.cosine_greedy(ref, qry, 0.1, 0.0, 2048)
    dev = torch.device("cuda", torch.cuda.current_device())
    for thr in (0.05, 0.2, 0.6):
        hits = kernels.cosine_greedy_sparse(ref.to_device(dev), qry.to_device(dev), 0.1, 0.0,
                                            2048, thr, capacity=16)  # forces a regrow
        r, q, s, m, o = hits.to_host()
        keep = want[0] >= thr
        rr, qq = np.nonzero(keep)
        np.testing.assert_array_equal(r, rr)
        np.testing.assert_array_equal(q, qq)
        np.testing.assert_array_equal(s.view(np.uint32), want[0][keep].view(np.uint32))
        np.testing.assert_array_equal(m, want[1][keep])
        np.testing.assert_array_equal(o, want[2][keep])


def test_bad_offsets_reported(cuda_device):
    """Non-monotone offsets: the validation kernel stops every later kernel and
    the call raises (no out-of-bounds access)."""
    import torch

    from cudams import kernels, synthetic
    from cudams._native import NativeError
    from cudams.packing import DeviceSpectra

    s = synthetic.uniform_spectra(10, seed=17)
    dev = torch.device("cuda", torch.cuda.current_device())
    d = s.to_device(dev)
    off = d.offsets.clone()
    off[3] = off[5] + 1
    bad = DeviceSpectra(d.mz, d.a, d.b, off, d.n, d.n_peaks)
    with pytest.raises(NativeError):
        kernels.cosine_greedy_dense(bad, d, 0.1, 0.0, 2048, check_errors=True)
    # the context stays usable
    want = oracle.cosine_greedy(s, s, 0.1, 0.0, 2048)
    assert_same(gpu_dense(s, s, P(0.1, 2048)), want, "after error")


def test_large_sampled(cuda_device):
    """12k x 12k heavy-tailed spectra: 40k sampled pairs bit-exact, and a
    second run bit-identical to the first (determinism)."""
    import torch

    from cudams import kernels, synthetic

    ref = synthetic.lognormal_spectra(12000, seed=18)
    qry = synthetic.lognormal_spectra(12000, seed=19)
    dev = torch.device("cuda", torch.cuda.current_device())
    rd, qd = ref.to_device(dev), qry.to_device(dev)
    a = kernels.cosine_greedy_dense(rd, qd, 0.01, 0.0, 4096, check_errors=True)
    a = [t.cpu().numpy() for t in a]
    b = kernels.cosine_greedy_dense(rd, qd, 0.01, 0.0, 4096, check_errors=True)
    b = [t.cpu().numpy() for t in b]
    assert_same(b, a, "determinism")
    rng = np.random.default_rng(0)
    pr = rng.integers(0, ref.n, 40000)
    pq = rng.integers(0, qry.n, 40000)
    # plus every pair that has a candidate in a band of rows
    band = np.nonzero(a[1][:200] != 0)
    pr = np.concatenate([pr, band[0]])
    pq = np.concatenate([pq, band[1]])
    s, m, o = oracle.cosine_greedy_pairs(ref, qry, pr, pq, 0.01, 0.0, 4096)
    np.testing.assert_array_equal(a[2][pr, pq], o)
    np.testing.assert_array_equal(a[1][pr, pq], m)
    np.testing.assert_array_equal(a[0][pr, pq].view(np.uint32), s.view(np.uint32))


@pytest.mark.parametrize("scale", ["plain", "ties", "wide", "tiny"])
def test_pair_pipeline_sort_paths(cuda_device, scale):
    """The pipelined pair kernel's sort through float32 words and what it falls back to:
    ordinary keys, many equal keys, keys that differ only below float32, keys below
    float32's range; truncated candidate lists of several sizes."""
    from cudams import synthetic
    from cudams.packing import PackedSpectra

    def weights(s, seed):
        rng = np.random.default_rng(seed)
        b = s.b.copy()
        if scale == "ties":
            b = np.round(rng.random(b.shape[0]) * 4 + 1)
        elif scale == "wide":
            b = 1.0 + rng.integers(0, 1 << 20, b.shape[0]) * 2.0 ** -45
        elif scale == "tiny":
            b = b * 2.0 ** -90
        return PackedSpectra(s.mz, None if scale != "plain" else s.a, b, s.offsets,
                             s.mz_power, s.intensity_power, s.n_max_peaks)

    ref = weights(synthetic.clustered_spectra(9, seed=91), 1)
    qry = weights(synthetic.clustered_spectra(11, seed=92), 2)
    for limit in (512, 1000, 1024, 2048):
        want = oracle.cosine_greedy(ref, qry, 0.05, 0.0, limit)
        assert_same(gpu_dense(ref, qry, P(0.05, limit, 2048), {"mode": 2}), want, f"{scale} {limit}")


def test_pair_pipeline_long_spectra(cuda_device):
    """Spectra with more peaks than the used-peak bitmaps of the pipelined kernel."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(93)
    def make(lens, seed):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([np.sort(rng.uniform(100.0, 130.0, k)) for k in lens])
        return pack_csr(mz.astype(np.float32), rng.random(off[-1]).astype(np.float32) + 0.01, off, None)
    ref, qry = make([8192, 8193, 20000, 3], 1), make([9000, 8192, 50], 2)
    for limit in (1024, 4096):
        want = oracle.cosine_greedy(ref, qry, 0.01, 0.0, limit)
        assert_same(gpu_dense(ref, qry, P(0.01, limit, 65535), {"mode": 2}), want, f"{limit}")


@pytest.mark.parametrize("weights", ["plain", "ties", "close"])
def test_run_lengths(cuda_device, weights):
    """Pairs with every number of candidates at which the join's way of resolving them changes
    (4/5, 8/9, 16/17, 32/33), all in one window or each peak with a few of its own; keys
    distinct, equal, and equal once rounded to float32."""
    from cudams.packing import PackedSpectra

    rng = np.random.default_rng(95)

    def make(lens, spacing):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([100.0 + spacing * np.arange(k) for k in lens]).astype(np.float32)
        b = {"plain": rng.random(off[-1]) + 0.01, "ties": np.round(rng.random(off[-1]) * 2 + 1),
             "close": 1.0 + rng.integers(0, 1 << 20, off[-1]) * 2.0 ** -45}[weights]
        return PackedSpectra(mz, None, b, off, 0.0, 1.0, 64)

    for spacing in (0.001, 0.03):
        ref = make(list(range(1, 9)) * 6 + [12], spacing)
        qry = make([1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 15, 16, 17, 31, 32, 33] * 5, spacing)
        want = oracle.cosine_greedy(ref, qry, 0.05, 0.0, 2048)
        for cfg in ({"mode": 1, "tile_spectra": 64}, {"mode": 1, "tile_spectra": 4096}):
            assert_same(gpu_dense(ref, qry, P(0.05, 2048), cfg), want, f"{spacing} {cfg}")
        want = oracle.cosine_greedy(qry, ref, 0.05, 0.0, 2048)
        assert_same(gpu_dense(qry, ref, P(0.05, 2048), {"mode": 1}), want, f"{spacing} swapped")


@pytest.mark.parametrize("n", [1, 2, 7])
def test_preparation_rounds(cuda_device, n):
    """Norms, weights and windows of spectra that end at, before and after a round of the
    preparation's loads, for one, two and an odd number of them a side."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(96)
    lens = np.array([129, 0, 128, 1, 127, 256, 1000])

    def make(lens):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([np.sort(rng.uniform(50.0, 150.0, k)) for k in lens])
        inten = rng.random(off[-1]) + 0.01
        return pack_csr(mz.astype(np.float32), inten.astype(np.float32), off, None, mz_power=1.0,
                        intensity_power=0.5)

    ref, qry = make(lens[:n]), make(np.roll(lens, 3)[:n])
    want = oracle.cosine_greedy(ref, qry, 0.02, 0.0, 4096)
    for cfg in ({"mode": 1, "tile_spectra": 32}, {"mode": 2}):
        assert_same(gpu_dense(ref, qry, P(0.02, 4096), cfg), want, f"{n} {cfg}")


@pytest.mark.parametrize("ml", [1, 40, 512, 520, 2048, 16384])
def test_spilled_pairs(cuda_device, ml):
    """Pairs the join leaves to the pair kernel, around the number of candidates up to which a
    warp takes one alone (512, or a share of small match limits), and with more peaks than its
    share of the used-peak bitmaps holds (2048)."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(97)

    def make(lens, spacing):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([100.0 + s * np.arange(k) for k, s in zip(lens, spacing)])
        inten = rng.integers(1, 50, off[-1])
        return pack_csr(mz.astype(np.float32), inten.astype(np.float32), off, None)

    ref = make([16, 5, 32, 2100, 33, 60], [0.001, 0.001, 0.001, 0.004, 0.001, 0.03])
    qry = make([31, 32, 33, 2047, 2049, 64, 7, 300], [0.001, 0.001, 0.001, 0.005, 0.005, 0.02, 0.001, 0.001])
    want = oracle.cosine_greedy(ref, qry, 0.05, 0.0, ml)
    for cfg in ({"mode": 1, "tile_spectra": 32}, {"mode": 1, "tile_spectra": 32, "pair_threads": 512},
                {"mode": 1, "tile_spectra": 32, "pair_threads": 96}):
        assert_same(gpu_dense(ref, qry, P(0.05, ml, 65535), cfg), want, f"{cfg}")


@pytest.mark.parametrize("pair_threads", [64, 128])
def test_pair_kernel_windows_as_defined(cuda_device, pair_threads):
    """m/z that are NaN (every window's last candidate) or next to zero under a shift that
    ends a window there: the candidates the float64 comparisons define."""
    from cudams.packing import pack_csr

    def pack(spectra):
        off = np.concatenate([[0], np.cumsum([len(s) for s in spectra])])
        mz = np.concatenate(spectra).astype(np.float32)
        inten = np.random.default_rng(len(spectra)).random(off[-1]).astype(np.float32) + 0.5
        return pack_csr(mz, inten, off, None, check=False)

    ref = pack([[100.0, 120.0, 300.0], [99.75, 100.0], [700.0]])
    qry = pack([[100.05, 119.95, np.nan], [299.95, np.nan, np.nan], [700.0], [np.nan]])
    cfg = {"mode": 2, "pair_threads": pair_threads}
    want = oracle.cosine_greedy(ref, qry, 0.1, 0.0, 64)
    assert want[1][0, 0] == 3 and want[1][0, 3] == 1
    assert_same(gpu_dense(ref, qry, P(0.1, 64), cfg), want, "nan")
    # lower end of the first peak's window one float64 step above zero
    near = pack([[0.0, 5e-15, 7.5e-15, 1e-14, 1.3e-14, 0.1, 0.2], [-1e-20, 1e-20]]
                + [[x] for x in (0.0, 5e-15, 7.5e-15, 1e-14, 1.3e-14)])
    for shift in (float(np.nextafter(100.0 - 0.1, 0.0)), 100.0 - 0.1, 100.0 + 0.1,
                  float(np.nextafter(100.0 + 0.1, 0.0))):
        want = oracle.cosine_greedy(ref, near, 0.1, shift, 64)
        assert_same(gpu_dense(ref, near, P(0.1, 64, shift=shift), cfg), want, f"{shift}")


def _one_candidate_a_peak(n, peaks, seed):
    from cudams.packing import pack_csr

    off = np.arange(n + 1) * peaks
    mz = np.tile(100.0 + 1500.0 / peaks * np.arange(peaks), n)
    inten = np.random.default_rng(seed).random(off[-1]) + 0.01
    return pack_csr(mz.astype(np.float32), inten.astype(np.float32), off, None)


@pytest.mark.parametrize("ml", [64, 4096, 16384])
def test_long_spectra_used_peaks(cuda_device, ml):
    """Spectra at and past the peaks whose bitmaps are in shared memory, with peaks
    shared by many candidates, through every launch of the pair kernels."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(98)

    def make(lens):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([np.sort(rng.uniform(100.0, 400.0, k)) for k in lens])
        return pack_csr(mz.astype(np.float32), rng.random(off[-1]).astype(np.float32) + 0.01, off,
                        None)

    ref, qry = make([8192, 8193, 20000, 40, 32767]), make([20000, 8193, 100, 8192])
    want = oracle.cosine_greedy(ref, qry, 0.03, 0.0, ml)
    for cfg in ({"mode": 2}, {"mode": 2, "pair_threads": 64}, {"mode": 1, "tile_spectra": 32}):
        assert_same(gpu_dense(ref, qry, P(0.03, ml, 65535), cfg), want, f"{cfg}")


@pytest.mark.parametrize("ml", [2048, 16384])
def test_long_spectra_cost(cuda_device, ml):
    """A pair's time grows with its peaks and candidates, not with their square: 2.5
    times the peaks (and at 16384 twice the candidates) within eight times the time."""
    import torch

    from cudams import kernels

    def seconds(peaks):
        a, b = (_one_candidate_a_peak(8, peaks, s).to_device(cuda_device) for s in (1, 2))
        best = float("inf")
        for _ in range(4):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            kernels.cosine_greedy_dense(a, b, 450.0 / peaks, 0.0, ml, config={"mode": 2})
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert seconds(20000) < 8 * seconds(8190)


@pytest.mark.parametrize("ml,peaks,pair_threads", [(1, 3, 128), (1, 3, 512), (600, 23, 512)])
def test_many_deferred_pairs(cuda_device, ml, peaks, pair_threads):
    """More light pairs than a CTA collects before it works them off, several times over,
    every one with more candidates than a warp's share of the buffer."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(101)
    n = 300 if ml == 1 else 200

    def make():
        off = np.arange(n + 1) * peaks
        mz = np.tile(100.0 + 0.001 * np.arange(peaks), n)
        return pack_csr(mz.astype(np.float32), rng.integers(1, 9, off[-1]).astype(np.float32), off,
                        None)

    ref, qry = make(), make()
    want = oracle.cosine_greedy(ref, qry, 0.05, 0.0, ml)
    cfg = {"mode": 1, "tile_spectra": 64, "pair_threads": pair_threads}
    for _ in range(2):
        assert_same(gpu_dense(ref, qry, P(0.05, ml), cfg), want, f"{cfg}")


@pytest.mark.parametrize("pair_threads", [96, 192, 224, 320, 416, 480])
def test_light_and_heavy_pairs(cuda_device, pair_threads):
    """Spilled pairs on both sides of the number of peaks a warp takes, with warps whose
    share of the used-peak bitmaps is an odd number of words."""
    from cudams.packing import pack_csr

    rng = np.random.default_rng(102)

    def make(lens):
        off = np.concatenate([[0], np.cumsum(lens)])
        mz = np.concatenate([np.sort(rng.uniform(100.0, 130.0, k)) for k in lens])
        return pack_csr(mz.astype(np.float32), rng.integers(1, 30, off[-1]).astype(np.float32), off,
                        None)

    ref, qry = make([255, 256, 257, 256, 300, 40]), make([256, 257, 255, 64, 256])
    for tol in (0.05, 0.2):
        want = oracle.cosine_greedy(ref, qry, tol, 0.0, 4096)
        cfg = {"mode": 1, "tile_spectra": 32, "pair_threads": pair_threads}
        assert_same(gpu_dense(ref, qry, P(tol, 4096), cfg), want, f"{tol} {cfg}")


def test_small_match_limit_cost(cuda_device):
    """Nearly every pair reaches a match limit of 16 and is left to the pair kernel, whose
    warps take such pairs: the call stays within 2.8 times that with a limit of 512."""
    import torch

    from cudams import kernels, synthetic

    a, b = (synthetic.uniform_spectra(1500, seed=s).to_device(cuda_device) for s in (1, 2))

    def seconds(ml):
        best = float("inf")
        for _ in range(4):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            kernels.cosine_greedy_dense(a, b, 0.5, 0.0, ml, config={"mode": 1, "tile_spectra": 64})
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert seconds(16) < 2.8 * seconds(512)


@pytest.mark.parametrize("cand", [0.05, 0.11, 0.6])
def test_automatic_tiles_agree(cuda_device, cand):
    """The library's own choice of tile is the one the Python estimate makes (the work
    items of a call, spectra times tiles, are counted by the trace)."""
    import torch

    from cudams import _native, autotune, kernels
    from cudams.packing import pack_csr

    n = 15000
    one = pack_csr(np.full(n, 100.0, np.float32), np.ones(n, np.float32), np.arange(n + 1), None)
    other = pack_csr(np.full(n, 200.0, np.float32), np.ones(n, np.float32), np.arange(n + 1), None)
    tile = autotune.heuristic_config(autotune.WorkloadStats(cand, 0.0, 1.0, 1.0), n, n)["tile_spectra"]
    rec = torch.zeros((1, 4), dtype=torch.int64, device=cuda_device)
    count = torch.zeros(1, dtype=torch.int64, device=cuda_device)
    ctx = _native.context(cuda_device.index)
    ctx.trace_enable(rec, count, 1)
    try:
        kernels.cosine_greedy_sparse(one.to_device(cuda_device), other.to_device(cuda_device), 0.1,
                                     0.0, 64, 0.5, config={"mode": 1, "cand_per_pair": cand})
    finally:
        ctx.trace_disable()
    assert int(count.item()) == n * -(-n // tile)
