"""Workloads of the pairwise spectrum-similarity path, for timing and for comparing results.

listed()             named cases, from one pair to billions of pairs
draw(rng)            one more case of the same ranges
prepare(case, seed)  inputs, outputs and plans on the GPU (or packed on the host, where the
                     entry point takes host spectra)
run(state)           one pass through the public entry points, and its outputs
work(case)           bytes and operations that one pass cannot do without
exact(case, seed)    the same outputs from plain torch in 64 bits (None where that is too long)

Kinds of case:
  pair         CudaCosineGreedy.pair on two spectra from the host: one comparison, as in a
               notebook or a scoring loop
  dense        all-vs-all greedy cosine of two device-resident sets into dense outputs; data
               "uniform" and "lognormal" are ordinary spectra, "clustered" the spectra whose
               pairs overflow match_limit; optional powers, shift and symmetric=1
  sparse       CudaCosineGreedy.matrix(array_type="sparse") on packed spectra: molecular
               networking and library matching, where only the good scores are kept
  search       SpectrumLibrary.search: a query batch against a resident library
  modified     all-vs-all modified cosine (analogue search)
  fingerprint  all-vs-all fingerprint similarity of bit-packed fingerprints
  mass         precursor m/z match (Dalton or ppm), the prefilter of the scores above
  intersect    m/z-set overlap
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "cosine-similarity_b200"))

from cudams import autotune, kernels  # noqa: E402
from cudams.packing import DeviceSpectra, PackedSpectra  # noqa: E402
from cudams.serving import SpectrumLibrary  # noqa: E402
from cudams.similarity import CudaCosineGreedy  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _dense(name, data, n_ref, n_q, tol, limit, mz_power=0.0, int_power=1.0, shift=0.0, sym=False):
    c = dict(kind="dense", data=data, n_ref=n_ref, n_q=n_q, tol=tol, limit=limit,
             mz_power=mz_power, int_power=int_power, shift=shift, sym=sym)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one pair of measured-size spectra: what a user's inner loop calls
        dict(name="pair", kind="pair", peaks_ref=120, peaks_q=85, tol=0.1, limit=2048,
             mz_power=0.0, int_power=1.0),
        # a batch against a batch, at the reference's default tolerance
        _dense("uniform_1k", "uniform", 1024, 1024, 0.1, 2048),
        # a spectral library against a data set, heavy-tailed peak counts
        _dense("lognormal_50k", "lognormal", 50000, 50000, 0.01, 4096),
        # a data set against itself for a network, weighted peaks, odd size
        _dense("symmetric_12k", "lognormal", 12345, 12345, 0.02, 2048, 1.0, 0.5, 0.0, True),
        # profile-like spectra of 1000 to 2000 peaks: nearly every pair reaches match_limit
        _dense("overflow_800", "clustered", 800, 907, 0.05, 1024, 3.0, 0.6),
        # the whole call from packed spectra to the kept scores
        dict(name="sparse_20k", kind="sparse", n_ref=20011, n_q=20000, tol=0.01, limit=2048,
             threshold=0.75),
        # a batch of queries against a resident library
        dict(name="search_1k", kind="search", n_ref=250000, n_q=1000, tol=0.01, limit=4096,
             threshold=0.7),
        # analogue search, odd sizes
        dict(name="modified_10k", kind="modified", n_ref=9001, n_q=11003, tol=0.1, limit=2048),
        # structures of a large library against each other, 2048-bit fingerprints
        dict(name="fingerprint_60k", kind="fingerprint", n_ref=60000, n_q=60000, bits=2048,
             measure="jaccard", missing=0.0, sym=False),
        # a small set of structures, some without a fingerprint
        dict(name="fingerprint_1k", kind="fingerprint", n_ref=1000, n_q=1501, bits=1024,
             measure="cosine", missing=0.02, sym=False),
        # precursor match in ppm over a whole data set
        dict(name="mass_ppm_40k", kind="mass", n_ref=40000, n_q=50000, tol=10.0, ppm=True),
        # shared m/z values of two sets
        dict(name="intersect_10k", kind="intersect", n_ref=10007, n_q=9000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "dense", "dense", "dense", "sparse", "search", "search", "modified",
                       "fingerprint", "fingerprint", "mass", "intersect"])
    powers = rng.choice([(0.0, 1.0), (0.0, 1.0), (0.0, 0.5), (1.0, 0.5), (3.0, 0.6)])
    if kind == "pair":
        return dict(kind=kind, peaks_ref=_log(rng, 5, 1000), peaks_q=_log(rng, 5, 1000),
                    tol=rng.choice([0.005, 0.01, 0.05, 0.1]), limit=2048, mz_power=powers[0],
                    int_power=powers[1])
    if kind == "dense":
        data = rng.choice(["uniform", "lognormal", "lognormal", "clustered"])
        if data == "clustered":
            return _dense(None, data, _log(rng, 60, 800), _log(rng, 60, 900), 0.05,
                          rng.choice([512, 1024, 2048]), *powers)
        tol = rng.choice([0.005, 0.01, 0.02, 0.1])
        top = 4000 if tol == 0.1 else 30000
        sym = rng.random() < 0.25
        n_ref = _log(rng, 30, top)
        n_q = n_ref if sym else _log(rng, 30, top)
        shift = 0.0 if sym else rng.choice([0.0, 0.0, 0.0, 14.01565, -0.9840])
        return _dense(None, data, n_ref, n_q, tol, rng.choice([1024, 2048, 4096]), *powers, shift,
                      sym)
    if kind == "sparse":
        return dict(kind=kind, n_ref=_log(rng, 100, 25000), n_q=_log(rng, 100, 25000),
                    tol=rng.choice([0.005, 0.01, 0.02]), limit=2048,
                    threshold=rng.choice([0.6, 0.7, 0.75, 0.9]))
    if kind == "search":
        return dict(kind=kind, n_ref=_log(rng, 20000, 250000), n_q=_log(rng, 1, 4096),
                    tol=rng.choice([0.005, 0.01, 0.02]), limit=4096,
                    threshold=rng.choice([0.6, 0.7, 0.8]))
    if kind == "modified":
        return dict(kind=kind, n_ref=_log(rng, 200, 12000), n_q=_log(rng, 200, 12000),
                    tol=rng.choice([0.01, 0.02, 0.1]), limit=2048)
    if kind == "fingerprint":
        sym = rng.random() < 0.2
        n_ref = _log(rng, 50, 50000)
        n_q = n_ref if sym else _log(rng, 50, 50000)
        if n_ref * n_q > 2_000_000:  # large results: rows of whole 128-byte lines
            n_q = (n_q + 31) // 32 * 32
            n_ref = n_q if sym else n_ref
        return dict(kind=kind, n_ref=n_ref, n_q=n_q,
                    bits=rng.choice([166, 512, 881, 1024, 2048, 4096]),
                    measure=rng.choice(["jaccard", "dice", "cosine"]),
                    missing=rng.choice([0.0, 0.0, 0.02]), sym=sym)
    if kind == "mass":
        ppm = rng.random() < 0.5
        return dict(kind=kind, n_ref=_log(rng, 100, 60000), n_q=_log(rng, 100, 60000),
                    tol=rng.choice([5.0, 10.0, 20.0]) if ppm else rng.choice([0.01, 0.1, 1.0]),
                    ppm=ppm)
    return dict(kind=kind, n_ref=_log(rng, 100, 12000), n_q=_log(rng, 100, 12000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Set:
    """A CSR spectrum set on the GPU: mz float32, intensity float32, offsets int64."""

    def __init__(self, mz, inten, off):
        self.mz, self.inten, self.off = mz, inten, off

    @property
    def n(self):
        return self.off.shape[0] - 1


def _gen(seed, salt):
    return torch.Generator(DEV).manual_seed(1000003 * int(seed) + salt)


def _offsets(lengths):
    off = torch.zeros(lengths.shape[0] + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(lengths, 0)
    return off


def _segments(lengths):
    return torch.repeat_interleave(torch.arange(lengths.shape[0], device=DEV), lengths)


def _sorted_set(seg, mz, inten, n):
    """Peaks (spectrum index, m/z, intensity) -> _Set, sorted by m/z inside each spectrum,
    intensities scaled to a maximum of 1."""
    mz = mz.to(torch.float32)
    # positive float32 values order as their bit patterns
    key = (seg << 32) | mz.view(torch.int32).to(torch.int64)
    key, order = torch.sort(key, stable=True)
    inten = inten[order]
    top = torch.full((n,), 1e-30, device=DEV, dtype=inten.dtype)
    top.scatter_reduce_(0, key >> 32, inten, "amax")
    inten = (inten / top[key >> 32]).to(torch.float32)
    lengths = torch.bincount(seg, minlength=n)
    return _Set((key & 0xFFFFFFFF).to(torch.int32).view(torch.float32), inten, _offsets(lengths))


def _lengths(data, n, g):
    if data == "uniform":
        return torch.randint(10, 201, (n,), generator=g, device=DEV)
    if data == "clustered":
        return torch.randint(1000, 2001, (n,), generator=g, device=DEV)
    z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
    return torch.exp(z + math.log(60.0)).round().clamp(5, 1000).to(torch.int64)


def _spectra(data, n, seed, salt):
    """uniform: 10-200 peaks, m/z U(50, 1000); lognormal: median 60 peaks (5-1000), m/z
    U(50, 2000), exponential intensities; clustered: 1000-2000 peaks around 200 centres."""
    g = _gen(seed, salt)
    lengths = _lengths(data, n, g)
    seg = _segments(lengths)
    p = seg.shape[0]
    u = torch.rand(p, generator=g, device=DEV, dtype=torch.float64)
    if data == "uniform":
        return _sorted_set(seg, 50.0 + 950.0 * u,
                           1.0 - torch.rand(p, generator=g, device=DEV), n)
    if data == "lognormal":
        return _sorted_set(seg, 50.0 + 1950.0 * u,
                           -torch.log1p(-torch.rand(p, generator=g, device=DEV)) + 1e-6, n)
    centres = 50.0 + 950.0 * torch.rand(200, generator=_gen(seed, 999), device=DEV,
                                        dtype=torch.float64)
    mz = centres[(u * 200).to(torch.int64).clamp(max=199)]
    mz = mz + 0.02 * torch.randn(p, generator=g, device=DEV, dtype=torch.float64)
    return _sorted_set(seg, mz, 1.0 - torch.rand(p, generator=g, device=DEV), n)


def _replicates(lib, n, seed, salt):
    """n query spectra: half re-measurements of library members (m/z jitter, a tenth of the
    peaks lost, intensities off by up to 30 %), half unrelated ones."""
    g = _gen(seed, salt)
    fresh = _spectra("lognormal", n, seed, salt + 1)
    pick = torch.randint(0, lib.n, (n,), generator=g, device=DEV)
    known = torch.arange(n, device=DEV) % 2 == 0
    len_lib = (lib.off[1:] - lib.off[:-1])[pick]
    len_new = fresh.off[1:] - fresh.off[:-1]
    lengths = torch.where(known, len_lib, len_new)
    seg = _segments(lengths)
    within = torch.arange(seg.shape[0], device=DEV) - _offsets(lengths)[seg]
    is_known = known[seg]
    at = torch.where(is_known, lib.off[pick][seg], fresh.off[:-1][seg]) + within
    at_lib = torch.where(is_known, at, 0)
    at_new = torch.where(is_known, 0, at)
    p = seg.shape[0]
    jitter = 0.002 * torch.randn(p, generator=g, device=DEV, dtype=torch.float64)
    gain = 0.7 + 0.6 * torch.rand(p, generator=g, device=DEV)
    mz = torch.where(is_known, lib.mz[at_lib].double() + jitter, fresh.mz[at_new].double())
    inten = torch.where(is_known, lib.inten[at_lib] * gain, fresh.inten[at_new])
    keep = ~is_known | (torch.rand(p, generator=g, device=DEV) >= 0.1)
    return _sorted_set(seg[keep], mz[keep], inten[keep], n)


def _analogues(n, seed, salt):
    """Families of eight analogues and their precursor m/z: members share the base spectrum's
    peaks, those above a cut move with the member's mass difference."""
    g = _gen(seed, salt)
    fam = (n + 7) // 8
    rand = lambda k: torch.rand(k, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    z = torch.randn(fam, generator=g, device=DEV, dtype=torch.float64)
    base_len = torch.exp(0.6 * z + math.log(60.0)).round().clamp(5, 600).to(torch.int64)
    base_prec = 300.0 + 1200.0 * rand(fam)
    base_off, base_seg = _offsets(base_len), _segments(base_len)
    base_mz = 50.0 + (base_prec[base_seg] - 55.0) * rand(base_seg.shape[0])
    base_int = -torch.log1p(-rand(base_seg.shape[0])) + 1e-6
    cut = (0.3 + 0.5 * rand(fam)) * base_prec
    member = torch.arange(n, device=DEV)
    f = member // 8
    diff = torch.where(rand(n) < 0.25, 0.0, 80.0 * rand(n) - 40.0)
    prec = base_prec[f] + diff
    lengths = base_len[f]
    seg = _segments(lengths)
    at = base_off[f][seg] + torch.arange(seg.shape[0], device=DEV) - _offsets(lengths)[seg]
    mz = base_mz[at] + torch.where(base_mz[at] > cut[f][seg], diff[seg], 0.0)
    mz = mz + 0.002 * torch.randn(seg.shape[0], generator=g, device=DEV, dtype=torch.float64)
    inten = base_int[at] * (0.7 + 0.6 * rand(seg.shape[0]))
    keep = rand(seg.shape[0]) >= 0.1
    return _sorted_set(seg[keep], mz[keep].clamp(min=1.0), inten[keep], n), prec


def _weights(s, mz_power, int_power):
    """Peak weights in float64 as the packer makes them: (m/z ** p or None, intensity ** q)."""
    a = None if mz_power == 0 else s.mz.double() ** mz_power
    return a, (s.inten.double() if int_power == 1 else s.inten.double() ** int_power)


def _device(s, mz_power=0.0, int_power=1.0):
    a, b = _weights(s, mz_power, int_power)
    return DeviceSpectra(s.mz, a, b, s.off, s.n, int(s.mz.shape[0]))


def _packed(s, mz_power=0.0, int_power=1.0):
    """The set as packed host spectra."""
    a, b = _weights(s, mz_power, int_power)
    return PackedSpectra(s.mz.cpu().numpy(), None if a is None else a.cpu().numpy(),
                         b.cpu().numpy(), s.off.cpu().numpy(), float(mz_power), float(int_power),
                         1024, _b32=s.inten.cpu().numpy() if int_power == 1 else None)


def _plan(ref, qry, tol, shift):
    """The framework's own plan for two sets, from the first spectra of large ones."""
    def part(s):
        k = min(s.n, 20000)
        p = int(s.off[k])
        return _packed(_Set(s.mz[:p], s.inten[:p], s.off[:k + 1]))

    r, q = part(ref), part(qry)
    stats = autotune.workload_stats(r, q, tol, shift, n_pairs=64)
    return autotune.heuristic_config(stats, qry.n, ref.n)


def _outputs(n_ref, n_q):
    return tuple(torch.empty((n_ref, n_q), dtype=t, device=DEV)
                 for t in (torch.float32, torch.int32, torch.uint8))


def _fingerprints(n, bits, missing, seed, salt):
    """(words int32 [n, ceil(bits / 32)], valid uint8 [n], 0/1 matrix uint8 [n, bits]);
    5-15 % of the bits of a row are set."""
    g = _gen(seed, salt)
    dens = 0.05 + 0.10 * torch.rand(n, generator=g, device=DEV)
    dense = (torch.rand((n, bits), generator=g, device=DEV) < dens[:, None]).to(torch.uint8)
    valid = torch.rand(n, generator=g, device=DEV) >= missing
    valid[0] = True
    dense *= valid[:, None].to(torch.uint8)
    n_words = (bits + 31) // 32
    words = torch.zeros((n, n_words * 32), dtype=torch.uint8, device=DEV)
    words[:, :bits] = dense
    words = words.view(n, n_words, 32)
    packed = torch.zeros((n, n_words), dtype=torch.int64, device=DEV)
    for k in range(32):
        packed |= words[:, :, k].to(torch.int64) << k
    packed = torch.where(packed >= 1 << 31, packed - (1 << 32), packed)
    return packed.to(torch.int32), valid.to(torch.uint8), dense


def _masses(n, seed, salt):
    """Precursor m/z: half drawn freely, half near one of a few hundred compounds."""
    g = _gen(seed, salt)
    rand = lambda k: torch.rand(k, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    known = 100.0 + 1100.0 * torch.rand(400, generator=_gen(seed, 7), device=DEV,
                                        dtype=torch.float64)
    m = known[(rand(n) * 400).to(torch.int64).clamp(max=399)] * (1.0 + 4e-5 * (rand(n) - 0.5))
    return torch.where(rand(n) < 0.5, m, 100.0 + 1100.0 * rand(n))


def _rounded_mz(n, seed, salt):
    """(m/z float64 rounded to two decimals, offsets) of lognormal spectra."""
    s = _spectra("lognormal", n, seed, salt)
    return torch.round(s.mz.double() * 100.0) / 100.0, s.off


def _pair_spectra(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in (case["peaks_ref"], case["peaks_q"]):
        mz = np.sort(rng.uniform(50.0, 1000.0, k)).astype(np.float32)
        inten = (1.0 - rng.uniform(0.0, 1.0, k)).astype(np.float32)
        out.append([mz, (inten / inten.max()).astype(np.float32)])
    # a few fragments in common, as between related compounds
    (mr, _), (mq, _) = out
    k = min(len(mr), len(mq)) // 3
    shared = rng.choice(len(mr), k, replace=False)
    mq[rng.choice(len(mq), k, replace=False)] = mr[shared] + rng.normal(0, 0.002, k).astype("f4")
    out[1][0] = np.sort(mq)
    return [tuple(s) for s in out]


def _two_sets(case, seed):
    kind = case["kind"]
    if kind == "dense":
        ref = _spectra(case["data"], case["n_ref"], seed, 11)
        return ref, ref if case["sym"] else _spectra(case["data"], case["n_q"], seed, 12)
    ref = _spectra("lognormal", case["n_ref"], seed, 13)
    return ref, _replicates(ref, case["n_q"], seed, 14)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pair":
        ref, qry = _pair_spectra(case, seed)
        cg = CudaCosineGreedy(tolerance=case["tol"], mz_power=case["mz_power"],
                              intensity_power=case["int_power"], match_limit=case["limit"])
        return dict(kind=kind, cg=cg, ref=ref, qry=qry)
    if kind == "dense":
        ref, qry = _two_sets(case, seed)
        cfg = _plan(ref, qry, case["tol"], case["shift"])
        if case["sym"]:
            cfg["symmetric"] = 1
        rd = _device(ref, case["mz_power"], case["int_power"])
        qd = rd if case["sym"] else _device(qry, case["mz_power"], case["int_power"])
        return dict(kind=kind, ref=rd, qry=qd, cfg=cfg, tol=case["tol"], shift=case["shift"],
                    limit=case["limit"], out=_outputs(ref.n, qry.n))
    if kind == "sparse":
        ref, qry = _two_sets(case, seed)
        cg = CudaCosineGreedy(tolerance=case["tol"], match_limit=case["limit"],
                              sparse_threshold=case["threshold"])
        return dict(kind=kind, cg=cg, ref=_packed(ref), qry=_packed(qry), rows=_rows(case))
    if kind == "search":
        ref, qry = _two_sets(case, seed)
        lib = SpectrumLibrary(_packed(ref), tolerance=case["tol"], match_limit=case["limit"])
        return dict(kind=kind, lib=lib, qry=_packed(qry), threshold=case["threshold"],
                    rows=_rows(case))
    if kind == "modified":
        ref, rp = _analogues(case["n_ref"], seed, 15)
        qry, qp = _analogues(case["n_q"], seed, 15 if case["n_q"] == case["n_ref"] else 16)
        cfg = _plan(ref, qry, case["tol"], 0.0)
        if cfg.get("cand_per_pair"):  # two passes: twice the candidates, half the tile
            cfg["cand_per_pair"] *= 2.0
            cfg["tile_spectra"] = max(32, (cfg["tile_spectra"] // 2 + 31) // 32 * 32)
        return dict(kind=kind, ref=_device(ref), rp=rp, qry=_device(qry), qp=qp, cfg=cfg,
                    tol=case["tol"], limit=case["limit"], out=_outputs(ref.n, qry.n))
    if kind == "fingerprint":
        r, rv, _ = _fingerprints(case["n_ref"], case["bits"], case["missing"], seed, 17)
        if case["sym"]:
            q, qv = r, rv
        else:
            q, qv, _ = _fingerprints(case["n_q"], case["bits"], case["missing"], seed, 18)
        return dict(kind=kind, measure=case["measure"], r=r, rv=rv, q=q, qv=qv, sym=case["sym"],
                    out=torch.empty((case["n_ref"], case["n_q"]), device=DEV))
    if kind == "mass":
        return dict(kind=kind, r=_masses(case["n_ref"], seed, 19), q=_masses(case["n_q"], seed, 20),
                    tol=case["tol"], ppm=case["ppm"],
                    out=torch.empty((case["n_ref"], case["n_q"]), dtype=torch.uint8, device=DEV))
    rm, ro = _rounded_mz(case["n_ref"], seed, 21)
    qm, qo = _rounded_mz(case["n_q"], seed, 22)
    return dict(kind=kind, rm=rm, ro=ro, qm=qm, qo=qo,
                out=torch.empty((case["n_ref"], case["n_q"]), dtype=torch.float64, device=DEV))


def _rows(case):
    """Rows of the table that a search's hits are kept in: far more than there are hits."""
    return 8 * case["n_q"] + case["n_ref"] // 4 + 256


def _table(rows, **columns):
    """The hits as columns of one length, and their number."""
    n = len(columns["row"])
    if n > rows:
        raise ValueError(f"{n} hits in a table of {rows} rows")
    out = {"hits": n}
    for name, x in columns.items():
        out[name] = np.zeros(rows, dtype=x.dtype)
        out[name][:n] = x
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "pair":
        r = s["cg"].pair(s["ref"], s["qry"])
        return {f: r[f] for f in ("score", "matches", "overflow")}
    if kind == "dense":
        return kernels.cosine_greedy_dense(s["ref"], s["qry"], s["tol"], s["shift"], s["limit"],
                                           out=s["out"], config=s["cfg"])
    if kind == "sparse":
        sp = s["cg"].matrix(s["ref"], s["qry"], array_type="sparse")
        d = sp.data
        return _table(s["rows"], row=sp.row, col=sp.col, score=d["sparse_score"],
                      matches=d["sparse_matches"], overflow=d["sparse_overflow"])
    if kind == "search":
        r = s["lib"].search(s["qry"], threshold=s["threshold"])
        return _table(s["rows"], row=r.ref, col=r.query, score=r.score, matches=r.matches,
                      overflow=r.overflow)
    if kind == "modified":
        return kernels.modified_cosine_dense(s["ref"], s["rp"], s["qry"], s["qp"], s["tol"],
                                             s["limit"], out=s["out"], config=s["cfg"])
    if kind == "fingerprint":
        return kernels.fingerprint_matrix(s["measure"], s["r"], s["rv"], s["q"], s["qv"],
                                          int(s["r"].shape[1]), float("nan"), out=s["out"],
                                          symmetric=s["sym"])
    if kind == "mass":
        return kernels.mass_match_matrix(s["r"], s["q"], s["tol"], s["ppm"], out=s["out"])
    return kernels.intersect_mz_matrix(s["rm"], s["ro"], s["qm"], s["qo"], out=s["out"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_MEAN_PEAKS = {"uniform": 105.0, "lognormal": 94.0, "clustered": 1500.0}


def work(case):
    kind = case["kind"]
    if kind == "pair":
        return {"bytes": 12.0 * (case["peaks_ref"] + case["peaks_q"]) + 9,
                "flops": 3.0 * (case["peaks_ref"] + case["peaks_q"])}
    n_r, n_q = float(case["n_ref"]), float(case["n_q"])
    pairs = n_r * n_q
    if kind == "dense":
        peaks = _MEAN_PEAKS[case["data"]] * (n_r if case["sym"] else n_r + n_q)
        per = 12.0 if case["mz_power"] == 0 else 20.0
        return {"bytes": per * peaks + 9.0 * pairs, "flops": 3.0 * peaks}
    if kind in ("sparse", "search"):
        peaks = _MEAN_PEAKS["lognormal"] * (n_r + n_q)
        return {"bytes": 12.0 * peaks + 17.0 * n_q / 2, "flops": 3.0 * peaks}
    if kind == "modified":
        peaks = 64.0 * (n_r + n_q)
        return {"bytes": 12.0 * peaks + 8 * (n_r + n_q) + 9.0 * pairs, "flops": 3.0 * peaks}
    if kind == "fingerprint":
        row = 4.0 * ((case["bits"] + 31) // 32) + 1
        return {"bytes": row * (n_r if case["sym"] else n_r + n_q) + 4.0 * pairs,
                "flops": 2.0 * case["bits"] * pairs}
    if kind == "mass":
        return {"bytes": 8.0 * (n_r + n_q) + pairs, "flops": (5.0 if case["ppm"] else 2.0) * pairs}
    return {"bytes": 8.0 * 94.0 * (n_r + n_q) + 8.0 * pairs, "flops": 2.0 * pairs}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _expand(lo, hi):
    """(owner, position) of every position in [lo[i], hi[i]), owners ascending."""
    cnt = (hi - lo).clamp(min=0)
    own = torch.repeat_interleave(torch.arange(lo.shape[0], device=DEV), cnt)
    start = torch.cumsum(cnt, 0) - cnt
    return own, lo[own] + torch.arange(own.shape[0], device=DEV) - start[own]


def _greedy_rows(ref, a_r, b_r, qry, a_q, b_q, rows, tol, shift, limit, prec=None):
    """Scores float64 [rows, n_q] of references rows[0]..rows[1] - 1: candidates in generation
    order, cut at `limit`, sorted by product (ties: the later one first), then accepted best
    first; every round accepts the best remaining candidate of every pair at once."""
    r0, r1 = rows
    n_q = qry.n
    p0, p1 = int(ref.off[r0]), int(ref.off[r1])
    seg_r = _segments(ref.off[r0 + 1:r1 + 1] - ref.off[r0:r1])
    mz_r = ref.mz[p0:p1].double()
    seg_q = _segments(qry.off[1:] - qry.off[:-1])
    mz_q = qry.mz.double()
    found = []
    for second in ((False, True) if prec is not None else (False,)):
        if second:
            prec_r, prec_q = prec
            val_q, val_r, margin = mz_q - prec_q[seg_q], mz_r - prec_r[r0:r1][seg_r], 1e-6
        else:
            val_q, val_r, margin = mz_q + shift, mz_r, 0.0
        val_q, order = torch.sort(val_q, stable=True)
        lo = torch.searchsorted(val_q, val_r - tol - margin, right=False)
        hi = torch.searchsorted(val_q, val_r + tol + margin, right=True)
        own, at = _expand(lo, hi)
        at = order[at]
        if second:
            y = mz_q[at] + (prec_r[r0:r1][seg_r[own]] - prec_q[seg_q[at]])
            ok = ~(y > mz_r[own] + tol) & ~(y < mz_r[own] - tol)
            own, at = own[ok], at[ok]
        found.append((own, at))
    own = torch.cat([f[0] for f in found])
    at = torch.cat([f[1] for f in found])
    pair = seg_r[own] * n_q + seg_q[at]
    # generation order inside a pair: pass, reference peak, query peak
    pair, order = torch.sort(pair, stable=True)
    own, at = own[order], at[order]
    n = pair.shape[0]
    first = torch.ones(n, dtype=torch.bool, device=DEV)
    first[1:] = pair[1:] != pair[:-1]
    start = torch.cummax(torch.where(first, torch.arange(n, device=DEV), 0), 0).values
    keep = torch.arange(n, device=DEV) - start < limit
    pair, own, at = pair[keep], own[keep], at[keep]
    w = b_r[p0:p1] if a_r is None else a_r[p0:p1] * b_r[p0:p1]
    key = w[own] * b_q[at] if a_q is None else w[own] * a_q[at] * b_q[at]
    for k in (lambda: torch.arange(pair.shape[0] - 1, -1, -1, device=DEV),
              lambda: torch.sort(key, descending=True, stable=True).indices,
              lambda: torch.sort(pair, stable=True).indices):
        o = k()
        pair, own, at, key = pair[o], own[o], at[o], key[o]
    score = torch.zeros((r1 - r0) * n_q, dtype=torch.float64, device=DEV)
    while pair.shape[0]:
        first = torch.ones(pair.shape[0], dtype=torch.bool, device=DEV)
        first[1:] = pair[1:] != pair[:-1]
        lead = torch.nonzero(first).squeeze(1)
        score[pair[lead]] += key[lead]
        mine = lead[torch.cumsum(first, 0) - 1]
        live = (own != own[mine]) & (at != at[mine])
        pair, own, at, key = pair[live], own[live], at[live], key[live]

    def norm(s, a, b):
        w2 = (b if a is None else a * b) ** 2
        total = torch.zeros(s.n, dtype=torch.float64, device=DEV)
        return total.index_add_(0, _segments(s.off[1:] - s.off[:-1]), w2).sqrt()
    denom = norm(ref, a_r, b_r)[r0:r1, None] * norm(qry, a_q, b_q)[None, :]
    score = score.view(r1 - r0, n_q)
    return torch.where(score > 0, score / denom, 0.0)


def _candidates(ref, qry, tol, shift):
    """About how many candidates all pairs have."""
    step = max(1, qry.mz.shape[0] // 200000)
    y = torch.sort(qry.mz[::step].double() + shift).values
    x = ref.mz[::max(1, ref.mz.shape[0] // 200000)].double()
    hits = (torch.searchsorted(y, x + tol, right=True) - torch.searchsorted(y, x - tol)).sum()
    return float(hits) / (x.shape[0] * y.shape[0]) * ref.mz.shape[0] * qry.mz.shape[0]


def _greedy(ref, qry, mz_power, int_power, tol, shift, limit, prec=None, sink=None):
    """Scores of all pairs in row blocks; sink(r0, block) or the whole matrix."""
    a_r, b_r = _weights(ref, mz_power, int_power)
    a_q, b_q = _weights(qry, mz_power, int_power)
    total = _candidates(ref, qry, tol, shift) * (2 if prec is not None else 1)
    if total > 4e8:
        return None
    rows = max(1, min(ref.n, int(ref.n * 3e7 / max(total, 1.0)), int(3e8 / max(1, qry.n))))
    whole = None if sink else torch.empty((ref.n, qry.n), dtype=torch.float64, device=DEV)
    for r0 in range(0, ref.n, rows):
        r1 = min(ref.n, r0 + rows)
        block = _greedy_rows(ref, a_r, b_r, qry, a_q, b_q, (r0, r1), tol, shift, limit, prec)
        if sink:
            sink(r0, block)
        else:
            whole[r0:r1] = block
    return whole if whole is not None else True


def exact(case, seed):
    kind = case["kind"]
    if kind == "pair":
        sets = []
        for mz, inten in _pair_spectra(case, seed):
            sets.append(_Set(torch.from_numpy(mz).to(DEV), torch.from_numpy(inten).to(DEV),
                             torch.tensor([0, len(mz)], device=DEV)))
        s = _greedy(*sets, case["mz_power"], case["int_power"], case["tol"], 0.0, case["limit"])
        return {"score": s.reshape(()), "matches": None, "overflow": None}
    if kind == "dense":
        if case["data"] == "clustered":
            return None  # about 1000 rounds over hundreds of millions of candidates
        ref, qry = _two_sets(case, seed)
        s = _greedy(ref, qry, case["mz_power"], case["int_power"], case["tol"], case["shift"],
                    case["limit"])
        if s is None:
            return None
        if case["sym"]:
            s = torch.triu(s) + torch.triu(s, 1).T
        return s, None, None
    if kind in ("sparse", "search"):
        ref, qry = _two_sets(case, seed)
        hits = []

        def sink(r0, block):
            at = torch.nonzero(block.float() >= np.float32(case["threshold"]).item())
            hits.append((at[:, 0] + r0, at[:, 1], block[at[:, 0], at[:, 1]]))

        if _greedy(ref, qry, 0.0, 1.0, case["tol"], 0.0, case["limit"], sink=sink) is None:
            return None
        r, q, s = (torch.cat([h[k] for h in hits]) for k in range(3))
        if kind == "search":  # sorted by query, then library spectrum
            s = s[torch.argsort(q * ref.n + r)]
        score = torch.zeros(_rows(case), dtype=torch.float64, device=DEV)
        score[:s.shape[0]] = s
        return {"hits": None, "row": None, "col": None, "score": score, "matches": None,
                "overflow": None}
    if kind == "modified":
        ref, rp = _analogues(case["n_ref"], seed, 15)
        qry, qp = _analogues(case["n_q"], seed, 15 if case["n_q"] == case["n_ref"] else 16)
        s = _greedy(ref, qry, 0.0, 1.0, case["tol"], 0.0, case["limit"], prec=(rp, qp))
        return None if s is None else (s, None, None)
    if kind == "fingerprint":
        r, rv, rd = _fingerprints(case["n_ref"], case["bits"], case["missing"], seed, 17)
        if case["sym"]:
            rd2, qv = rd, rv
        else:
            _, qv, rd2 = _fingerprints(case["n_q"], case["bits"], case["missing"], seed, 18)
        out = torch.empty((case["n_ref"], case["n_q"]), dtype=torch.float64, device=DEV)
        b = rd2.double().sum(1)
        qt = rd2.half().T.contiguous()  # counts of at most 4096 are exact in float32 sums
        for k in range(0, case["n_ref"], 4096):
            part = rd[k:k + 4096]
            a = part.double().sum(1)[:, None]
            inter = _counts(part.half(), qt)
            if case["measure"] == "jaccard":
                v = inter / (a + b - inter)
            elif case["measure"] == "dice":
                v = 2.0 * inter / (a + b)
            else:
                v = inter / torch.sqrt(a * b)
            out[k:k + 4096] = torch.nan_to_num(v)
        out[rv == 0] = float("nan")
        out[:, qv == 0] = float("nan")
        return out
    if kind == "mass":
        return None  # bytes, compared as they are
    rm, ro = _rounded_mz(case["n_ref"], seed, 21)
    qm, qo = _rounded_mz(case["n_q"], seed, 22)

    def distinct(mz, off):
        seg = _segments(off[1:] - off[:-1])
        first = torch.ones(mz.shape[0], dtype=torch.bool, device=DEV)
        first[1:] = (mz[1:] != mz[:-1]) | (seg[1:] != seg[:-1])
        return mz[first], seg[first]

    (vr, sr), (vq, sq) = distinct(rm, ro), distinct(qm, qo)
    vq, order = torch.sort(vq, stable=True)
    own, at = _expand(torch.searchsorted(vq, vr), torch.searchsorted(vq, vr, right=True))
    inter = torch.bincount(sr[own] * case["n_q"] + sq[order][at],
                           minlength=case["n_ref"] * case["n_q"])
    inter = inter.view(case["n_ref"], case["n_q"]).double()
    union = (torch.bincount(sr, minlength=case["n_ref"])[:, None]
             + torch.bincount(sq, minlength=case["n_q"])[None, :]) - inter
    return torch.where(union > 0, inter / union, 0.0)


def _counts(part, qt):
    """Intersection counts in float64: 2048 bits at a time, exact in half-precision products
    accumulated in float32 and rounded to the nearest half below 2049."""
    out = None
    for k in range(0, part.shape[1], 2048):
        c = (part[:, k:k + 2048] @ qt[k:k + 2048]).double()
        out = c if out is None else out + c
    return out
