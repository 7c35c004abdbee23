// Tiled greedy cosine for sm_100a: cms_cosine_greedy / cms_cosine_greedy_sparse.
//
// Replaces the reference's per-pair Numba kernel (cudams/similarity/
// spectrum_similarity_functions.py:39-262) and the batch loop around it
// (cudams/similarity/CudaCosineGreedy.py:138-226).  Results are identical to
// the plain kernel and to the oracle; only the way candidates are found and
// ordered differs.
//
// Pipeline of one call (all on one stream, no host synchronisation):
//   1. prep_kernel       both sets in one launch: offsets sane, spectra <= CMS_MAX_PEAKS
//                        (else every later kernel exits at once and the error
//                        word is set); sqrt(sum (a*b)^2) per spectrum,
//                        sequential float64; the reference spectra's length
//                        classes and the query peaks' bucket counts;
//      probe_kernel      per reference peak its window and buckets
//   2. order_scatter     reference spectra ordered by peak count, largest
//                        first (log2 length classes), for load balance
//   3. index kernels     query spectra are cut into tiles of tile_spectra;
//                        each tile's peaks are bucketed by m/z (bucket width
//                        tol by default, buckets hashed modulo n_buckets;
//                        two-launch scan of the counts, then scatter) into a
//                        CSR "tile stream" of (m/z, query<<16 | peak, weight)
//   4. join_kernel       persistent warps; one work item = (reference
//                        spectrum, query tile).  Lanes take reference peaks,
//                        jump through the bucket table to the tile-stream
//                        entries inside the tolerance window (the
//                        two-pointer sweep of the reference, with the second
//                        pointer advanced by the index instead of one step at
//                        a time), test them with exact float32 window bounds
//                        and push candidates into a per-warp pool (shared
//                        memory, extended in global memory).  Each query's
//                        run is then resolved greedily: 1-4 candidates in
//                        closed form by one lane, 5-8 by an 8-lane segment,
//                        9-16 by half a warp, 17-32 by the warp.
//                        The sweep is load-balanced: a chunk's window entries
//                        are expanded 32 at a time over the warp, and each
//                        query's candidates are chained through a per-warp
//                        head table (tagged by an epoch, so it is rarely
//                        cleared) instead of being counting-sorted.
//                        The dense row segment is zeroed with coalesced
//                        stores just before, and each run stores its result
//                        over its zeros.  Pairs with longer runs (or >=
//                        match_limit candidates) go to a spill list.
//   5. pair_kernel       a CTA per heavy spilled pair (or per pair of the whole
//                        matrix in mode 2), a warp per light one: exact generation-order sweep with
//                        match_limit truncation, bitonic sort of (key, gen)
//                        (in registers when there are eight candidates a
//                        thread, else in shared memory), warp greedy with
//                        used-peak bitmasks and conflict masks over the live
//                        candidates.
//   6. mirror_kernel     (symmetric dense calls, csrc/mirror.cu) lower
//                        triangle copied from the upper one.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "cms_internal.cuh"

namespace cms {
namespace {

constexpr int kJoinWarps = 8;
constexpr int kJoinThreads = kJoinWarps * 32;
constexpr int kMidRun = 8;        // runs up to this length are resolved four per warp step
constexpr int kMaxTile = 4096;    // max query spectra per tile
constexpr int kOrderClasses = 17; // log2 length classes (0..16)
// Length classes (512 peaks and more) whose spectra the join takes first,
// against every tile: one of them against the last tile, begun when the other
// warps are nearly done, would be waited for (12345 symmetric: 1.90 ms tile by
// tile, 1.70 ms with them first; 1000 queries against a library 1.78 and 1.67).
// Not for modified cosine, whose few large spectra are slower when they all
// run together (8.8 ms tile by tile, 9.5 with them first).
constexpr int kLargeClass = 10;
constexpr int kModifiedMaxPeaks = 32767;  // modified cosine: reference peak index in 15 bits

__device__ __forceinline__ double peak_a(const double* a, int64_t i) { return a ? a[i] : 1.0; }

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// ---------------------------------------------------------------------------
// tile index over the query side
// ---------------------------------------------------------------------------
// tile-stream entry: m/z (also in the neutral-loss index), (query within tile
// << 16 | peak), intensity weight b
struct __align__(16) Entry {
    float mz;
    uint32_t id;
    double b;
};

struct IndexGeom {
    int tile;        // query spectra per tile
    int n_tiles;
    int nb;          // buckets per tile (power of two)
    double inv_w;    // 1 / bucket width
};

// Bucket of an m/z value: floor(mz / width), hashed modulo nb by the caller.
// Monotone non-decreasing in mz (one float64 multiply, then round down), so
// every entry inside [L, H] falls in a bucket of [bucket_of(L), bucket_of(H)].
// (float64 keeps one bucket per width even when mz / width exceeds 2^24.)
__device__ __forceinline__ long long bucket_of(float x, double inv_w) {
    return __double2ll_rd(__dmul_rn((double)x, inv_w));
}

// The value the neutral-loss index of modified cosine buckets a peak by: its
// m/z minus its spectrum's precursor m/z, computed in float64 and rounded to
// float32 (the windows are widened by a margin that covers this rounding, and
// the join confirms each candidate exactly).
__device__ __forceinline__ float loss_value(float mz, double prec) {
    return __double2float_rn(__dsub_rn((double)mz, prec));
}
// Neutral-loss window of modified cosine's shifted pass: entries whose
// m/z - precursor lies within tol of the sweeping peak's, widened by twice
// the float32 spacing there (the indexed values are rounded to float32) and a
// float64 rounding allowance, rounded outwards; every entry of its buckets is
// then tested exactly against the shifted window.
__device__ __forceinline__ bool nl_window(float mz, double prec, double tol, float& L, float& H) {
    const double zr = __dsub_rn((double)mz, prec);
    const float mag = __double2float_ru(fabs(zr) + tol + 1.0);
    const double m = 2.0 * (double)(nextafterf(mag, INFINITY) - mag) +
                     1e-9 * (fabs((double)mz) + fabs(prec) + 1.0);
    L = __double2float_rd(__dsub_rn(__dsub_rn(zr, tol), m));
    H = __double2float_ru(__dadd_rn(__dadd_rn(zr, tol), m));
    return isfinite(L) && isfinite(H);
}

// Exact float32 window of one sweeping peak.
//
// The float64 test of the reference (query peak y matches reference peak x iff
// !(y+shift > x+tol) && !(y+shift < x-tol)) is, for a fixed sweeping peak, a
// conjunction of a predicate non-decreasing in the indexed peak's m/z and one
// non-increasing in it.  So the float32 values it accepts form one interval
// [L, H] of float32 numbers.  It is found once per sweeping peak by rounding
// an estimate and stepping with nextafterf until the float64 predicates flip;
// each entry is then tested with two float32 compares, with exactly the same
// outcome as the float64 test.  The estimate is within an ulp or two; the
// step loops are capped, and a peak that does not converge (non-finite input)
// gets an empty window and an error flag.
template <bool A_IS_REF, bool NOSHIFT>
struct Window {
    // A_IS_REF: x = sweeping reference peak; lo/hi = x -+ tol
    // else:     c = sweeping query peak + shift
    __device__ __forceinline__ static bool not_below(float y, double lo, double c, double tol,
                                                     double shift) {
        if (A_IS_REF) return !(__dadd_rn((double)y, shift) < lo);
        return !(c > __dadd_rn((double)y, tol));
    }
    __device__ __forceinline__ static bool not_above(float y, double hi, double c, double tol,
                                                     double shift) {
        if (A_IS_REF) return !(__dadd_rn((double)y, shift) > hi);
        return !(c < __dsub_rn((double)y, tol));
    }
    __device__ static bool bounds(float mzA, double tol, double shift, float& L, float& H) {
        const double x = (double)mzA;
        if (A_IS_REF && NOSHIFT) {
            // y (float32, exact in float64) is accepted iff lo <= y <= hi: the
            // interval ends are lo rounded up and hi rounded down to float32
            L = __double2float_ru(__dsub_rn(x, tol));
            H = __double2float_rd(__dadd_rn(x, tol));
            return isfinite(L) && isfinite(H);
        }
        double lo = 0.0, hi = 0.0, c = 0.0, el, eh;
        if (A_IS_REF) {
            lo = __dsub_rn(x, tol);
            hi = __dadd_rn(x, tol);
            el = __dsub_rn(lo, shift);
            eh = __dsub_rn(hi, shift);
        } else {
            c = __dadd_rn(x, shift);
            el = __dsub_rn(c, tol);
            eh = __dadd_rn(c, tol);
        }
        float l = __double2float_rd(el), h = __double2float_ru(eh);
        int k = 0;
        for (; k < 16 && !not_below(l, lo, c, tol, shift); ++k) l = nextafterf(l, INFINITY);
        for (; k < 32 && not_below(nextafterf(l, -INFINITY), lo, c, tol, shift); ++k)
            l = nextafterf(l, -INFINITY);
        for (; k < 48 && !not_above(h, hi, c, tol, shift); ++k) h = nextafterf(h, -INFINITY);
        for (; k < 64 && not_above(nextafterf(h, INFINITY), hi, c, tol, shift); ++k)
            h = nextafterf(h, INFINITY);
        const bool ok = k < 64 && isfinite(l) && isfinite(h) && not_below(l, lo, c, tol, shift) &&
                        not_above(h, hi, c, tol, shift);
        L = l;
        H = h;
        return ok;
    }
};

// What the join needs to know of a sweeping peak, computed once per call: its
// window [lo, hi] in the indexed side's float32 m/z and the window's first and
// last bucket (first > last: the range wraps around the hashed table;
// kNoBucket: no entry can match).
struct __align__(16) Probe {
    float lo, hi;
    uint32_t bl, bh;
};
constexpr uint32_t kNoBucket = 0xffffffffu;

__device__ __forceinline__ uint2 bucket_range(float L, float H, const IndexGeom& g) {
    if (!(L <= H)) return make_uint2(kNoBucket, 0u);
    const long long blo = bucket_of(L, g.inv_w), bhi = bucket_of(H, g.inv_w);
    if (bhi - blo + 1 >= g.nb) return make_uint2(0u, (unsigned)g.nb - 1u);
    const unsigned mask = (unsigned)(g.nb - 1);
    return make_uint2((unsigned)blo & mask, (unsigned)bhi & mask);
}

// A sweeping spectrum in the order the join takes them.
struct __align__(16) SweepItem {
    int64_t a0;   // its first peak
    int32_t a;    // its index
    int32_t na;   // its peaks
    double rn;    // 1 / norm (recip_norm)
    double pad;
};

// 1 / norm for the join's division-free score, NaN (which sends the score to
// the division) for norms whose products with it could leave the normal range
__device__ __forceinline__ double recip_norm(double sn) {
    return sn >= 1e-100 && sn <= 1e100 ? __drcp_rn(sn) : __longlong_as_double(0x7ff8000000000000ll);
}

// ---------------------------------------------------------------------------
// 1. preparation of a spectrum set: validation, norms, length classes and
//    bucket counts in one launch
// ---------------------------------------------------------------------------
__device__ __forceinline__ int length_class(int64_t len) {
    return len <= 0 ? 0 : min(kOrderClasses - 1, 64 - __clzll((unsigned long long)len));
}

struct PrepSide {
    SpecSet S;
    double* sn;           // sqrt(sum_k (a_k * b_k)^2), summed in peak order
    double* rn;           // recip_norm(sn) (null: not wanted)
    uint32_t* cls_count;  // spectra per length class (null: not wanted)
    uint32_t* cnt;        // peaks per (tile, bucket) of the m/z index (null: not wanted)
    uint32_t* cnt2;       // the same of the neutral-loss index (null: not wanted)
    double* w;            // per peak a * b (null: not wanted)
};

// The sides of a call in one launch: its first blocks0 blocks take side 0.
struct PrepSides {
    PrepSide side[2];
    int blocks0;
    uint32_t* any_long;  // set to 1 by a spectrum of more than kLongPeaks peaks (null: not wanted)
};
constexpr int kLongPeaks = 8192;  // longer spectra have no used-peak bitmaps in shared memory

struct ProbeArgs {
    SpecSet S;          // the sweeping side
    Probe* probe;       // per peak
    uint2* probe2;      // per peak, its shifted window's buckets (null: not wanted)
    double tol, shift;  // of the windows
    int is_ref;         // the sweeping side is the reference side
};

// The windows and buckets of every sweeping peak, a thread a peak.  In a launch
// of its own: warps of the kernel below, a few spectra each, took 20 us for
// them at 1024 spectra and 25 at 20000 (4 and 10 here).
constexpr int kProbeThreads = 256;
__global__ void __launch_bounds__(kProbeThreads)
probe_kernel(ProbeArgs P, IndexGeom g, const uint32_t* bad, uint32_t* err) {
    if (*bad) return;
    const int64_t first = P.S.off[0], last = P.S.off[P.S.n];
    const int64_t step = (int64_t)gridDim.x * kProbeThreads;
    for (int64_t k = first + (int64_t)blockIdx.x * kProbeThreads + threadIdx.x; k < last; k += step) {
        const float mz = P.S.mz[k];
        Probe p{1.0f, 0.0f, kNoBucket, 0u};
        float L, H;
        const bool ok = !P.is_ref        ? Window<false, false>::bounds(mz, P.tol, P.shift, L, H)
                        : P.shift == 0.0 ? Window<true, true>::bounds(mz, P.tol, P.shift, L, H)
                                         : Window<true, false>::bounds(mz, P.tol, P.shift, L, H);
        if (ok) {
            const uint2 b = bucket_range(L, H, g);
            p = Probe{L, H, b.x, b.y};
        } else {
            atomicOr(err, kErrBadOffsets);
        }
        *reinterpret_cast<uint4*>(&P.probe[k]) =
            make_uint4(__float_as_uint(p.lo), __float_as_uint(p.hi), p.bl, p.bh);
        if (P.probe2) {
            int64_t s = 0, e = P.S.n;  // the spectrum: off[s] <= k < off[e]
            while (e - s > 1) {
                const int64_t m = s + (e - s) / 2;
                if (P.S.off[m] <= k)
                    s = m;
                else
                    e = m;
            }
            uint2 b = make_uint2(kNoBucket, 0u);
            if (nl_window(mz, P.S.prec[s], P.tol, L, H))
                b = bucket_range(L, H, g);
            else
                atomicOr(err, kErrBadOffsets);
            P.probe2[k] = b;
        }
    }
}

// cnt / cnt2 have geometry g.  Offsets out of order or range and spectra above
// max_peaks raise the error word and *bad, which stops every later kernel of
// the call; such a spectrum is skipped here.
//
// A norm is one float64 sum in peak order, a serial chain, so a warp takes
// kPrepSpectra spectra at once: their peaks come 32 * kPrepPeaks at a time with
// coalesced loads through a shared-memory tile, and lane j adds up spectrum j
// while the next peaks of each are in flight.  One thread a spectrum, reading
// its peaks one after the other, took 24 us for 1024 spectra of up to 200
// peaks, 84 us for 50000 of up to 1000 and 445 us for 900 of up to 2000.  What
// is left is the time of a round of loads, and how many rounds a long spectrum
// has: both sides of 1024 uniform spectra 9 us, of 12288 lognormal ones 49 us,
// with the bucket counts; eight spectra of 32 peaks a round 18 and 66, four of
// 128 12 and 62, one of 256 8 and 62.
constexpr int kPrepSpectra = 2;
constexpr int kPrepPeaks = 4;  // of a spectrum, per lane and round
constexpr int kPrepThreads = 128;
__global__ void __launch_bounds__(kPrepThreads)
prep_kernel(const __grid_constant__ PrepSides sides, IndexGeom g, uint32_t* bad, uint32_t* err,
            int max_peaks) {
    const bool second = (int)blockIdx.x >= sides.blocks0;
    const PrepSide& P = sides.side[second];
    const int block = (int)blockIdx.x - (second ? sides.blocks0 : 0);
    const int blocks = second ? (int)gridDim.x - sides.blocks0 : sides.blocks0;
    __shared__ double s_tile[kPrepThreads / 32][kPrepSpectra][32 * kPrepPeaks + 1];
    __shared__ uint32_t s_cls[kOrderClasses];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned full = 0xffffffffu;
    double(*tile)[32 * kPrepPeaks + 1] = s_tile[wid];
    if (threadIdx.x < kOrderClasses) s_cls[threadIdx.x] = 0u;
    __syncthreads();
    const unsigned mask = (unsigned)(g.nb - 1);
    const int64_t warps = (int64_t)blocks * (kPrepThreads / 32);
    const int64_t n = P.S.n;
    for (int64_t s0 = ((int64_t)block * (kPrepThreads / 32) + wid) * kPrepSpectra; s0 < n;
         s0 += warps * kPrepSpectra) {
        int64_t lo = 0;
        int len = 0;
        if (lane < kPrepSpectra && s0 + lane < n) {
            lo = P.S.off[s0 + lane];
            const int64_t hi = P.S.off[s0 + lane + 1];
            uint32_t e = 0;
            if (lo < 0 || hi < lo || hi > P.S.n_peaks) e |= kErrBadOffsets;
            if (hi - lo > max_peaks) e |= kErrSpectrumTooLong;
            if (e) {
                atomicOr(err, e);
                atomicOr(bad, 1u);
                lo = 0;
            } else {
                len = (int)(hi - lo);
                if (P.cls_count) atomicAdd(&s_cls[length_class(len)], 1u);
                if (sides.any_long && len > kLongPeaks) *sides.any_long = 1u;
            }
        }
        const int longest = __reduce_max_sync(full, len);
        // the loads of all spectra are issued before the first is used
        constexpr int kRound = 32 * kPrepPeaks, kAll = kPrepSpectra * kPrepPeaks;
        double v[kAll], w[kAll];
        float z[kAll];
        auto each = [&](int c, auto&& f) {  // (index, spectrum, offset in it, in it?)
#pragma unroll
            for (int i = 0; i < kAll; ++i) {
                const int j = i / kPrepPeaks, o = c + 32 * (i % kPrepPeaks) + lane;
                f(i, j, o, o < __shfl_sync(full, len, j));
            }
        };
        auto load = [&](int c) {
            each(c, [&](int i, int j, int o, bool in) {
                const int64_t k = __shfl_sync(full, lo, j) + o;
                v[i] = in ? P.S.b[k] : 0.0;
                w[i] = (in && P.S.a) ? P.S.a[k] : 1.0;
                z[i] = (in && P.cnt) ? P.S.mz[k] : 0.f;
            });
        };
        auto weights = [&](int c) {
            if (!P.w) return;
            each(c, [&](int i, int j, int o, bool in) {
                const int64_t k = __shfl_sync(full, lo, j) + o;
                if (in) P.w[k] = __dmul_rn(w[i], v[i]);
            });
        };
        auto count = [&](int c) {
            if (!P.cnt) return;
            each(c, [&](int i, int j, int, bool in) {
                if (!in) return;
                const int64_t t = (s0 + j) / g.tile * (int64_t)g.nb;
                atomicAdd(&P.cnt[t + ((unsigned)bucket_of(z[i], g.inv_w) & mask)], 1u);
                if (P.cnt2) {
                    const float d = loss_value(z[i], P.S.prec[s0 + j]);
                    atomicAdd(&P.cnt2[t + ((unsigned)bucket_of(d, g.inv_w) & mask)], 1u);
                }
            });
        };
        double acc = 0.0;
        load(0);
        for (int c = 0; c < longest; c += kRound) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kAll; ++i) {
                const double x = __dmul_rn(w[i], v[i]);
                tile[i / kPrepPeaks][32 * (i % kPrepPeaks) + lane] = __dmul_rn(x, x);
            }
            count(c);
            weights(c);
            __syncwarp();
            if (c + kRound < longest) load(c + kRound);
            // past a spectrum's end the tile holds +0.0, which leaves the sum as it is
            if (lane < kPrepSpectra) {
#pragma unroll 16
                for (int k = 0; k < kRound; ++k) acc = __dadd_rn(acc, tile[lane][k]);
            }
        }
        if (lane < kPrepSpectra && s0 + lane < n) {
            const double sn = sqrt(acc);
            P.sn[s0 + lane] = sn;
            if (P.rn) P.rn[s0 + lane] = recip_norm(sn);
        }
        __syncwarp();
    }
    __syncthreads();
    if (P.cls_count && threadIdx.x < kOrderClasses && s_cls[threadIdx.x])
        atomicAdd(&P.cls_count[threadIdx.x], s_cls[threadIdx.x]);
}

// Exclusive scan of the bucket counts into tab[t][0..nb], and the counters to
// the bucket starts (scatter cursors), in two launches of one CTA per chunk of
// kScanChunk buckets: the chunks' sums, then each chunk's own scan on top of
// the sums of its tile's earlier chunks.  Coalesced both ways: 25 us for 25
// tiles of 2^18 buckets (one CTA a tile, each thread walking its own run of
// buckets: 636 us).
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanChunk = kScanThreads * kScanPer;
__host__ __device__ constexpr int scan_chunks(int nb) { return (nb + kScanChunk - 1) / kScanChunk; }

__device__ __forceinline__ uint32_t block_sum(uint32_t x, uint32_t* s_warp) {
    x = __reduce_add_sync(0xffffffffu, x);
    __syncthreads();  // s_warp free from an earlier use
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) total += s_warp[w];
    return total;
}

__global__ void __launch_bounds__(kScanThreads)
index_sums_kernel(IndexGeom g, const uint32_t* cnt, uint32_t* sums, const uint32_t* bad) {
    if (*bad) return;
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const int per_tile = scan_chunks(g.nb);
    const int t = (int)blockIdx.x / per_tile, ch = (int)blockIdx.x % per_tile;
    const uint32_t* c = cnt + (int64_t)t * g.nb + (int64_t)ch * kScanChunk;
    const int m = min(kScanChunk, g.nb - ch * kScanChunk);
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        const int k = i * kScanThreads + (int)threadIdx.x;
        if (k < m) x += c[k];
    }
    x = block_sum(x, s_warp);
    if (threadIdx.x == 0) sums[blockIdx.x] = x;
}

__global__ void __launch_bounds__(kScanThreads)
index_scan_kernel(IndexGeom g, uint32_t* cnt_cur, uint32_t* tab, const uint32_t* sums,
                  const uint32_t* bad) {
    if (*bad) return;
    __shared__ uint32_t s_val[kScanChunk + kScanChunk / kScanPer];
    __shared__ uint32_t s_warp[kScanThreads / 32], s_incl[kScanThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per_tile = scan_chunks(g.nb);
    const int t = (int)blockIdx.x / per_tile, ch = (int)blockIdx.x % per_tile;
    uint32_t* c = cnt_cur + (int64_t)t * g.nb + (int64_t)ch * kScanChunk;
    uint32_t* out = tab + (int64_t)t * (g.nb + 1) + (int64_t)ch * kScanChunk;
    const int m = min(kScanChunk, g.nb - ch * kScanChunk);
    // coalesced in, kScanPer consecutive buckets a thread out of shared memory
    // (one word of padding per kScanPer, so that neither side has conflicts)
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        const int k = i * kScanThreads + tid;
        s_val[k + k / kScanPer] = k < m ? c[k] : 0u;
    }
    uint32_t prev = 0;  // the tile's earlier chunks
    for (int i = tid; i < ch; i += kScanThreads) prev += sums[t * per_tile + i];
    prev = block_sum(prev, s_warp);
    uint32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) sum += s_val[tid * (kScanPer + 1) + i];
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) s_incl[wid] = incl;
    __syncthreads();
    uint32_t run = prev + incl - sum;
    for (int w = 0; w < wid; ++w) run += s_incl[w];
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        const uint32_t v = s_val[tid * (kScanPer + 1) + i];
        s_val[tid * (kScanPer + 1) + i] = run;
        run += v;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        const int k = i * kScanThreads + tid;
        if (k < m) {
            const uint32_t v = s_val[k + k / kScanPer];
            out[k] = v;
            c[k] = v;
        }
    }
    if (ch == per_tile - 1 && tid == kScanThreads - 1) out[m] = run;
}

// Warp per spectrum: its peaks (value, q_local<<16 | peak) into the tile
// stream, four chunks of 32 with their cursor atomics in flight at a time
// (4.7 M peaks: 110 us; one chunk at a time 135 us).
template <bool NL>
__global__ void index_scatter_kernel(SpecSet B, IndexGeom g, uint32_t* cur, Entry* ent,
                                     double* ent_a, const uint32_t* bad) {
    if (*bad) return;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned mask = (unsigned)(g.nb - 1);
    constexpr int kU = 4;
    for (int64_t s = warp; s < B.n; s += nwarps) {
        const int64_t t = s / g.tile;
        const int64_t base = B.off[t * g.tile];
        const uint32_t ql = (uint32_t)(s - t * g.tile);
        const int64_t lo = B.off[s], hi = B.off[s + 1];
        uint32_t* c = cur + t * (int64_t)g.nb;
        for (int64_t k0 = lo + lane; k0 < hi; k0 += 32 * kU) {
            float v[kU], mz[kU];
            double b[kU], a[kU];
            uint32_t pos[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int64_t k = k0 + 32 * u;
                if (k < hi) {
                    mz[u] = B.mz[k];
                    v[u] = NL ? loss_value(mz[u], B.prec[s]) : mz[u];
                    b[u] = B.b[k];
                    if (ent_a) a[u] = B.a[k];
                }
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (k0 + 32 * u < hi)
                    pos[u] = atomicAdd(&c[(unsigned)bucket_of(v[u], g.inv_w) & mask], 1u);
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int64_t k = k0 + 32 * u;
                if (k < hi) {
                    Entry en;
                    en.mz = mz[u];
                    en.id = (ql << 16) | (uint32_t)(k - lo);
                    en.b = b[u];
                    ent[base + pos[u]] = en;
                    if (ent_a) ent_a[base + pos[u]] = a[u];
                }
            }
        }
    }
}

// Sweeping-side order (largest length class first); a block's spectra are
// ranked per class in shared memory, so that the 17 cursors get one atomic a
// block and class.
constexpr int kOrderThreads = 256;
__global__ void __launch_bounds__(kOrderThreads)
order_scatter_kernel(SpecSet S, const double* sn, const uint32_t* cls_count, uint32_t* cls_cursor,
                     SweepItem* items, const uint32_t* bad) {
    if (*bad) return;
    __shared__ uint32_t s_cnt[kOrderClasses], s_base[kOrderClasses];
    const int tid = threadIdx.x;
    for (int64_t s0 = (int64_t)blockIdx.x * kOrderThreads; s0 < S.n;
         s0 += (int64_t)gridDim.x * kOrderThreads) {
        if (tid < kOrderClasses) s_cnt[tid] = 0u;
        __syncthreads();
        const int64_t s = s0 + tid;
        int c = 0;
        uint32_t rank = 0;
        SweepItem it{};
        if (s < S.n) {
            it.a0 = S.off[s];
            it.na = (int32_t)(S.off[s + 1] - it.a0);
            it.a = (int32_t)s;
            it.rn = recip_norm(sn[s]);
            c = length_class(it.na);
            rank = atomicAdd(&s_cnt[c], 1u);
        }
        __syncthreads();
        if (tid < kOrderClasses && s_cnt[tid]) {
            uint32_t base = 0;
            for (int k = kOrderClasses - 1; k > tid; --k) base += cls_count[k];
            s_base[tid] = base + atomicAdd(&cls_cursor[tid], s_cnt[tid]);
        }
        __syncthreads();
        if (s < S.n) items[s_base[c] + rank] = it;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// shared helpers for greedy resolution
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long order_key(double k) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(k);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double key_from_order(unsigned long long o) {
    const unsigned long long u = (o >> 63) ? (o & 0x7fffffffffffffffull) : ~o;
    return __longlong_as_double((long long)u);
}
// (key, gen) strictly precedes (key', gen') in the greedy order
__device__ __forceinline__ bool before(double k1, uint32_t g1, double k2, uint32_t g2) {
    return k1 > k2 || (k1 == k2 && g1 > g2);
}

__device__ __forceinline__ void emit_hit(const SparseOut& o, int r, int q, float sc, int mt,
                                         uint8_t ovf) {
    const bool both = o.mirror && r != q;
    const unsigned long long pos = atomicAdd(o.count, both ? 2ull : 1ull);
    if (pos < (unsigned long long)o.capacity) {
        o.r[pos] = r;
        o.q[pos] = q;
        o.score[pos] = sc;
        o.matches[pos] = mt;
        o.overflow[pos] = ovf;
    }
    if (both && pos + 1 < (unsigned long long)o.capacity) {
        o.r[pos + 1] = q;
        o.q[pos + 1] = r;
        o.score[pos + 1] = sc;
        o.matches[pos + 1] = mt;
        o.overflow[pos + 1] = ovf;
    }
}

// Optional per-work-item timing records (cms_trace_enable): 4 words each --
// tag | smid << 32, item index, %globaltimer at its start and end (ns).
struct TraceOut {
    unsigned long long* rec;
    unsigned long long* count;
    long long cap;
    unsigned int tag;
};

// Pairs for the pair kernel, which works on them by size: heavy ones from the
// front of the list, light ones from its back.
// A pair with a longer spectrum than this is heavy: a warp alone would be the last
// one running.  (128, 256, 512 and 1024 peaks: 209, 180, 211 and 285 us for 12345
// symmetric spectra, 124, 113, 174 and 270 for sparse 20000 x 20000, 340, 297, 243
// and 223 for modified cosine of 9001 x 11003.)
constexpr int kHeavyPeaks = 256;
struct SpillList {
    int2* pairs;                // (reference, query)
    unsigned long long* count;  // heavy pairs | light pairs << 32
    unsigned int cap;
};

__device__ __forceinline__ void spill_push(const SpillList& sl, int r, int q, int64_t longest,
                                           uint32_t* err) {
    const bool heavy = longest > kHeavyPeaks;
    const unsigned long long n = atomicAdd(sl.count, heavy ? 1ull : 1ull << 32);
    const unsigned int front = (unsigned int)n, back = (unsigned int)(n >> 32);
    if ((unsigned long long)front + back < sl.cap)
        sl.pairs[heavy ? front : sl.cap - 1 - back] = make_int2(r, q);
    else
        atomicOr(err, kErrSpillOverrun);
}

// ---------------------------------------------------------------------------
// 4. join kernel
// ---------------------------------------------------------------------------
struct JoinParams {
    SpecSet A;  // sweeping side (one spectrum per work item)
    SpecSet B;  // indexed side (tiles)
    const SweepItem* items;  // sweeping spectra, largest length class first
    const uint32_t* cls_count;  // their number per length class
    const Probe* probe;      // per sweeping peak: window and buckets
    const uint2* probe2;     // modified cosine: buckets of the shifted window
    const double* w;         // per sweeping peak: its weight in the key
    const double* snA;
    const double* snB;
    const double* rnB;
    const uint32_t* tab;
    const Entry* ent;
    const double* ent_a;   // m/z weight a of each tile-stream entry (null: 1.0)
    const uint32_t* tab2;  // modified cosine: neutral-loss index (m/z - precursor)
    const Entry* ent2;
    const double* ent2_a;
    IndexGeom g;
    double tol;
    int match_limit;
    float init_width_scale;  // first sub-range width = scale / n_A_peaks (0: whole tile)
    // first sub-range width per length class of the sweeping spectrum (the
    // tuner's measured candidate-pool split); 0: init_width_scale decides
    int width_by_class[kOrderClasses];
    int warp_smem_bytes;     // per-warp slice of dynamic shared memory
    int pool_smem;           // candidates of the pool in shared memory (join_pool)
    int pool_max;            // candidates a sweep may hold: kPoolMax, or pool_smem without gpool
    int max_fetch;           // work items per warp before it exits (0: no limit)
    unsigned char* gpool;    // global pool extension, kGPool * 16 bytes per warp (or null)
    // bounded launches: a CTA claims one of n_slots global-pool slices (a bit
    // of `slots`) for its lifetime instead of using slice blockIdx.x (null:
    // slice blockIdx.x, persistent launches)
    unsigned int* slots;
    int n_slots;
    TraceOut trace;          // per-item timing records (rec null: off)
    unsigned long long* work;
    SpillList spill;
    DenseOut dense;
    int vec_rows;            // dense arrays 16 / 16 / 4-byte aligned: vector zeros
    SparseOut sparse;
    uint32_t* err;
    const uint32_t* bad;
    int sym;  // only pairs (reference i, query j) with i <= j
};

// Pool slots a lane has in flight when owners are looked up (one: 1 to 3% slower).
constexpr int kIlpR = 2;
constexpr int kSearchWaves = 4;            // waves of short-lived CTAs per library search
constexpr int kSlotWords = 64;             // slot bitmap words of a bounded join launch
constexpr int kPoolMax = 4096;             // candidates per sweep: smem pool + global extension
constexpr int kPoolMin = 128;              // of them at least in shared memory (join_pool)
constexpr int kGPool = kPoolMax - kPoolMin;  // global extension entries per warp
static_assert(kPoolMax <= 4096, "pool slots are packed into 12 bits");
static_assert(kMaxTile <= 4096, "query indices within a range are packed into 12 bits");

// One candidate: key, generation word and a metadata word, which holds the
// query's index within the swept range (bits 0-11) and the slot of the
// previous candidate of the same query (bits 12-23, present when kHasNext is
// set).  A query's candidates form a chain that starts at the slot its head
// names (the candidate pushed last).
struct __align__(16) PoolEntry {
    double key;
    uint32_t gen;
    uint32_t meta;
};
constexpr uint32_t kHasNext = 1u << 24;
__device__ __forceinline__ int meta_query(uint32_t m) { return (int)(m & 0xFFFu); }
__device__ __forceinline__ int meta_next(uint32_t m) { return (int)((m >> 12) & 0xFFFu); }

// A warp's candidate pool: the first n_smem entries live in shared memory, the
// rest in a per-warp slice of global scratch (L2-resident), so that a large
// reference spectrum is swept once even when it has thousands of candidates
// in a tile.  Slots are indices into the concatenation; an access is one
// 16-byte generic load or store (gbase points n_smem entries before the slice).
struct Pool {
    PoolEntry* sbase;
    PoolEntry* gbase;
    int n_smem;
    __device__ __forceinline__ PoolEntry* at(int i) const { return (i < n_smem ? sbase : gbase) + i; }
    __device__ __forceinline__ PoolEntry get(int i) const {
        const uint4 v = *reinterpret_cast<const uint4*>(at(i));
        return PoolEntry{__hiloint2double((int)v.y, (int)v.x), v.z, v.w};
    }
    __device__ __forceinline__ uint32_t meta(int i) const { return at(i)->meta; }
    __device__ __forceinline__ void put(int i, double k, uint32_t g, uint32_t m) const {
        *reinterpret_cast<uint4*>(at(i)) =
            make_uint4((unsigned)__double2loint(k), (unsigned)__double2hiint(k), g, m);
    }
};

// Per-warp shared-memory slice (offsets in bytes; the head table's length
// depends on the tile size, so the slice size is computed at launch).
//   rec   uint4 [32]         sweep: the chunk's peaks with window entries, in order:
//                            stream offset, window, lane.  Resolution: uint16 queue
//                            of chain heads with two or more candidates
//   wa    double [32]        per-lane sweeping-peak weight of the current chunk
//                            Resolution: accepted keys of a long run in order
//   runs  uint32 [kLongRuns] runs of five or more candidates queued for the warp:
//                            slot of the chain head | length << 12; runs of at
//                            most kMidRun from the front, longer ones from the back
//   lists uint16 [kLists]    slots of the long runs being resolved: 32 of up to
//                            8 candidates or 8 of up to 32
//   t0    uint64             %globaltimer at the current item's start (trace only)
//   head  uint16 [tile]      one per query of the range: (epoch << 12) | slot of
//                            its last candidate; a head of another epoch means
//                            "no candidate yet"
//   pool  PoolEntry [join_pool(tile)]
constexpr int kLongRuns = 64;
constexpr int kLists = 256;
constexpr int kQueue = 256;
__host__ __device__ constexpr int head_bytes(int tile) { return (2 * tile + 15) & ~15; }
constexpr int kSliceFixed = 16 * 32 + 8 * 32 + 4 * kLongRuns + 2 * kLists + 16;
// Pool entries in shared memory, between kPoolMin and kPoolMost: as many as
// leave the L1 cache its share when three CTAs are resident.  Above kSliceTarget
// bytes a warp the next larger carve-out of shared memory is taken, which
// costs about 32 KB of L1, where the bucket table's and the tile stream's
// sectors hit: 50000 x 50000 lognormal spectra in tiles of 1792 take 9.6 ms
// with 8208 bytes a warp, 8.9 ms with 8112 (186 entries) and 8.95 ms with 7800.
// More than 256 entries gain nothing where the tiles are small.
constexpr int kPoolMost = 256;
constexpr int kSliceTarget = 8112;
__host__ __device__ constexpr int join_pool(int tile) {
    const int fit = (kSliceTarget - kSliceFixed - head_bytes(tile)) / 16;
    return fit < kPoolMin ? kPoolMin : fit > kPoolMost ? kPoolMost : fit;
}
__host__ __device__ constexpr int warp_slice_bytes(int tile) {
    return kSliceFixed + head_bytes(tile) + 16 * join_pool(tile);
}

// Reference peak of a candidate's generation word.  Modified cosine marks
// candidates of its second (precursor-shifted) pass in bit 31, which makes
// them later in generation order than every unshifted one (the order of
// matchms' concatenation) and limits its spectra to 32767 peaks.
template <bool MODIFIED>
__device__ __forceinline__ uint32_t gen_p1(uint32_t g) {
    return MODIFIED ? ((g >> 16) & 0x7FFFu) : (g >> 16);
}

// Kept out of line: the division's code would be in the join several times.
__device__ __noinline__ float cosine_exact(double score, const double* nr, const double* nq) {
    return (float)__ddiv_rn(score, __dmul_rn(*nr, *nq));
}

// float32 of score / (nr * nq) with both operations rounded in float64, as the
// reference order has it, mostly without the division: rr and rq are the
// norms' reciprocals (NaN when a norm is out of [1e-100, 1e100]), so
// (score * rr) * rq is within 3 * 2^-52 of the quotient, and when the float32
// values of both ends of a band of 2^-49 around it agree, the quotient rounds
// to that value too.  Otherwise (about one in 10^7, zero norms and scores
// below 1e-30) the quotient itself.
__device__ __forceinline__ float cosine_of(double score, double rr, double rq, const double* nr,
                                           const double* nq) {
    const double x = __dmul_rn(__dmul_rn(score, rr), rq);
    const float lo = (float)__dmul_rn(x, 1.0 - 0x1p-49), hi = (float)__dmul_rn(x, 1.0 + 0x1p-49);
    if (lo == hi && lo > 1e-30f) return lo;
    return cosine_exact(score, nr, nq);
}

// Bound by instruction issue and latency together (about 13 cycles between a
// warp's instructions at six warps a scheduler), not by memory: 50000 x 50000
// lognormal spectra, dense, move 11.5 B a pair at half the copy rate.
// So what counts is the length of an item's instruction chain: windows and
// buckets come ready-made per sweeping peak, item descriptors in order, a
// pool entry is one 16-byte access, and owners of one candidate do not wait
// for the code of longer runs (50000 x 50000: 11.45 ms with all of that done
// per item, 9.6 ms after; 8.5 ms with the L1 cache that join_pool leaves).
// The code is kept short, 45 KB instead of 126 KB: modified cosine 13.2 -> 8.8 ms and 1024 x 1024 328 -> 272 us together with
// the comparison instead of the sorting of long runs.  Four CTAs at 64
// registers spill: 1024 x 1024 +13%, search of 1000 +10%, modified +6%.
// Three CTAs (24 warps) per SM: up to 80 registers a thread.
template <bool A_IS_REF, bool SPARSE, bool MODIFIED>
__global__ void __launch_bounds__(kJoinThreads, 3)
join_kernel(JoinParams P) {
    if (*P.bad) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int hb = head_bytes(P.g.tile);
    unsigned char* slice = smem_raw + (size_t)(threadIdx.x >> 5) * P.warp_smem_bytes;
    uint4* s_rec = reinterpret_cast<uint4*>(slice);
    uint16_t* queue = reinterpret_cast<uint16_t*>(s_rec);
    double* s_wa = reinterpret_cast<double*>(slice + 16 * 32);
    uint32_t* long_runs = reinterpret_cast<uint32_t*>(slice + 24 * 32);
    uint16_t* lists = reinterpret_cast<uint16_t*>(long_runs + kLongRuns);
    unsigned long long* s_t0 = reinterpret_cast<unsigned long long*>(lists + kLists);
    uint16_t* head = reinterpret_cast<uint16_t*>(slice + kSliceFixed);
    // Global-pool slice of this CTA: blockIdx.x, or under bounded launches a
    // slice claimed from the slot bitmap (at most n_slots CTAs are resident at
    // once, so one is free; if a release has not landed yet the CTA runs with
    // the shared-memory pool only).  Every search is bounded by 2 passes over
    // the words and 32 attempts per word.
    __shared__ int s_slot;
    int pslot = (int)blockIdx.x;
    if (P.slots) {
        if (threadIdx.x == 0) {
            int got = -1;
            const int words = (P.n_slots + 31) >> 5;
            for (int i = 0; i < 2 * words && got < 0; ++i) {
                const int w = (int)((blockIdx.x + (unsigned)i) % (unsigned)words);
                const int nb = min(32, P.n_slots - 32 * w);
                const unsigned valid = nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u);
                unsigned cur = atomicOr(&P.slots[w], 0u);
                for (int k = 0; k < 32 && got < 0; ++k) {
                    const unsigned freeb = ~cur & valid;
                    if (!freeb) break;
                    const unsigned bit = freeb & (0u - freeb);
                    const unsigned old = atomicOr(&P.slots[w], bit);
                    if (!(old & bit))
                        got = 32 * w + (__ffs(bit) - 1);
                    else
                        cur = old | bit;
                }
            }
            s_slot = got;
        }
        __syncthreads();
        pslot = s_slot;
    }
    const int pool_max = (P.gpool && pslot >= 0) ? P.pool_max : P.pool_smem;
    Pool pool;
    pool.n_smem = P.pool_smem;
    pool.sbase = reinterpret_cast<PoolEntry*>(slice + kSliceFixed + hb);
    pool.gbase = pool.sbase;
    if (P.gpool && pslot >= 0)
        pool.gbase = reinterpret_cast<PoolEntry*>(P.gpool) +
                     ((size_t)pslot * kJoinWarps + (threadIdx.x >> 5)) * (size_t)kGPool - P.pool_smem;

    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const unsigned below = (1u << lane) - 1u;
    const unsigned upto = below | (1u << lane);
    const int64_t nA = P.A.n;
    const int64_t n_items = nA * (int64_t)P.g.n_tiles;
    // epoch of the head table (1..15): every swept range takes the next one,
    // so heads left by earlier ranges read as empty without clearing the
    // table; it is cleared once per 15 ranges (and before the first)
    unsigned epoch = 15;

    int64_t n_large = 0;
    if (!MODIFIED)
        for (int c = kLargeClass; c < kOrderClasses; ++c) n_large += P.cls_count[c];
    // the next item's index is fetched while the current one is processed
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(P.work, 1ull);
    for (int fetches = 0; P.max_fetch == 0 || fetches < P.max_fetch; ++fetches) {
        const unsigned long long item = __shfl_sync(full, next, 0);
        if ((int64_t)item >= n_items) break;
        if (lane == 0 && (P.max_fetch == 0 || fetches + 1 < P.max_fetch))
            next = atomicAdd(P.work, 1ull);
        int t;
        SweepItem A;
        {
            // large spectra over all tiles, then the others tile by tile
            const bool small = (int64_t)item >= n_large * P.g.n_tiles;
            const int64_t j = small ? (int64_t)item - n_large * P.g.n_tiles : (int64_t)item;
            const int64_t m = small ? nA - n_large : n_large;
            int64_t ai;
            if (n_items <= 0xffffffffll) {
                t = (int)((unsigned)j / (unsigned)m);
                ai = (unsigned)j - (unsigned)t * (unsigned)m;
            } else {
                t = (int)(j / m);
                ai = j - (int64_t)t * m;
            }
            const int4* it = reinterpret_cast<const int4*>(P.items + ai + (small ? n_large : 0));
            const int4 x = __ldg(it);
            A.a0 = ((int64_t)x.y << 32) | (unsigned)x.x;
            A.a = x.z;
            A.na = x.w;
            A.rn = __ldg(reinterpret_cast<const double*>(it + 1));
        }
        if (P.trace.rec && lane == 0) *s_t0 = global_ns();
        const int a = A.a, na = A.na;
        const int b_begin = t * P.g.tile;
        const int tn = (int)min((int64_t)P.g.tile, P.B.n - b_begin);
        const int64_t tbase = P.B.off[b_begin];
        const uint32_t* T = P.tab + (int64_t)t * (P.g.nb + 1);
        const uint32_t* T2 = MODIFIED ? P.tab2 + (int64_t)t * (P.g.nb + 1) : nullptr;
        // dense position of (this spectrum, query b_begin); the join's dense
        // output always has the sweeping spectrum as its row
        auto row = [&]() { return SPARSE ? 0 : (int64_t)a * P.dense.ld + b_begin; };
        // a resolved run's score and count, for query q of the tile
        auto store_result = [&](int q, double score, int mt, double rnB) {
            const float sc = cosine_of(score, A.rn, rnB, P.snA + a, P.snB + b_begin + q);
            if (SPARSE) {
                if (sc >= P.sparse.threshold)
                    emit_hit(P.sparse, A_IS_REF ? a : b_begin + q, A_IS_REF ? b_begin + q : a, sc,
                             mt, 0);
            } else {
                __stcs(P.dense.score + row() + q, sc);
                __stcs(P.dense.matches + row() + q, mt);
            }
        };
        // a run for the pair kernel (its dense cells marked until then)
        auto spill_run = [&](int q) {
            const int64_t nq = P.B.off[b_begin + q + 1] - P.B.off[b_begin + q];
            spill_push(P.spill, A_IS_REF ? a : b_begin + q, A_IS_REF ? b_begin + q : a,
                       max((int64_t)na, nq), P.err);
            if (!SPARSE) {
                __stcs(P.dense.score + row() + q, __int_as_float(0x7fc00000));
                __stcs(P.dense.matches + row() + q, -1);
            }
        };

        int width = tn;
        const int wc = P.width_by_class[length_class(na)];
        if (wc > 0)
            width = max(1, min(tn, wc));
        else if (P.init_width_scale > 0.f && na > 0)  // multiples of 32 keep row writes aligned
            width = max(32, min(tn, (int)(P.init_width_scale / (float)na) & ~31));
        // queries of this item: the whole tile, or under `sym` those on or
        // above the diagonal (reference index <= query index)
        int range_lo = 0, q_end = tn;
        if (P.sym) {
            if (A_IS_REF)
                range_lo = max(0, min(tn, a - b_begin));
            else
                q_end = max(0, min(tn, a - b_begin + 1));
        }
        while (range_lo < q_end) {
            const int range_hi = min(range_lo + width, q_end);
            const int rw = range_hi - range_lo;
            epoch = epoch == 15 ? 1u : epoch + 1u;
            if (epoch == 1u)
                for (int w = lane; w < hb / 16; w += 32)
                    reinterpret_cast<uint4*>(head)[w] = make_uint4(0u, 0u, 0u, 0u);
            __syncwarp();
            // ---- sweep: candidates of (a, queries [range_lo, range_hi)) ----
            // Each lane takes one sweeping peak of a 32-peak chunk and finds
            // the tile-stream entries of its window's buckets (one run, or two
            // when the hashed bucket range wraps: then the chunk takes a second
            // turn for the wrapped parts).  The chunk's entries are processed
            // 32 at a time, flat entry k by lane k % 32, so that every lane
            // tests an entry in every round, however unevenly the entries fall
            // among the peaks.  The peaks that have entries leave a record each,
            // in order; a round's first entries of peaks are or-ed into a mask
            // over its 32 positions, so the owner of an entry is the count of
            // mask bits up to its position (one reduction, one population count
            // and one shared-memory read; a binary search by shuffles over the
            // entry counts took five dependent shuffles).
            // Latency is hidden by running ahead: a step's bucket-table loads
            // are issued one step early (steps are chunks, or chunk x pass
            // for modified cosine), the probes they need one chunk early.
            int n = 0;  // candidates found (warp-uniform)
            constexpr int kPasses = MODIFIED ? 2 : 1;
            const int n_steps = ((na + 31) >> 5) * kPasses;
            // this step's probe (pr) and the next chunk's (pn)
            Probe pr, pn;
            uint2 pr2 = make_uint2(kNoBucket, 0u), pn2 = pr2;  // shifted pass: buckets, m/z
            float mz_c = 0.f, mz_n = 0.f;
            double w_c = 0.0, w_n = 0.0;
            auto load_peak = [&](int pp, Probe& x, uint2& x2, float& mz, double& w) {
                x = Probe{1.0f, 0.0f, kNoBucket, 0u};
                if (MODIFIED) x2 = make_uint2(kNoBucket, 0u);
                if (pp < na) {
                    const int4 v = __ldg(reinterpret_cast<const int4*>(P.probe + A.a0 + pp));
                    x = Probe{__int_as_float(v.x), __int_as_float(v.y), (uint32_t)v.z, (uint32_t)v.w};
                    w = __ldg(P.w + A.a0 + pp);
                    if (MODIFIED) {
                        x2 = __ldg(P.probe2 + A.a0 + pp);
                        mz = __ldg(P.A.mz + A.a0 + pp);
                    }
                }
            };
            // raw bucket-table values: entries [t0, t1), and [0, t2) when wrapped
            auto table = [&](const uint32_t* TT, uint32_t bl, uint32_t bh, uint32_t& t0,
                             uint32_t& t1, uint32_t& t2) {
                const bool some = bl != kNoBucket, wraps = some && bl > bh;
                t0 = some ? __ldg(TT + bl) : 0u;
                t1 = some ? __ldg(TT + (wraps ? (uint32_t)P.g.nb : bh + 1u)) : 0u;
                t2 = wraps ? __ldg(TT + bh + 1u) : 0u;
            };
            load_peak(lane, pr, pr2, mz_c, w_c);
            load_peak(32 + lane, pn, pn2, mz_n, w_n);
            uint32_t t0, t1, t2;
            table(T, pr.bl, pr.bh, t0, t1, t2);
            for (int st = 0; st < n_steps; ++st) {
                const int pass = MODIFIED ? (st & 1) : 0;
                const int pc = (MODIFIED ? (st >> 1) : st) * 32;
                const uint32_t r0 = t0, c0 = t1 - t0, c1 = t2;
                // window of the record; the shifted pass tests with the peak's m/z
                const float x0 = (MODIFIED && pass) ? mz_c : pr.lo, x1 = pr.hi;
                if (pass == 0) s_wa[lane] = w_c;
                // the next step's table values, in flight during this step's rounds
                if (MODIFIED && pass == 0) {
                    table(T2, pr2.x, pr2.y, t0, t1, t2);
                } else {
                    pr = pn;
                    w_c = w_n;
                    if (MODIFIED) {
                        pr2 = pn2;
                        mz_c = mz_n;
                    }
                    table(T, pr.bl, pr.bh, t0, t1, t2);
                    load_peak(pc + 64 + lane, pn, pn2, mz_n, w_n);
                }
                const Entry* EE = ((MODIFIED && pass) ? P.ent2 : P.ent) + tbase;
                const double* EA = (MODIFIED && pass) ? P.ent2_a : P.ent_a;
                const int turns = __any_sync(full, c1 != 0u) ? 2 : 1;
                for (int turn = 0; turn < turns; ++turn) {
                    const uint32_t c = turn ? c1 : c0;
                    uint32_t incl = c;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t v = __shfl_up_sync(full, incl, d);
                        if (lane >= d) incl += v;
                    }
                    const uint32_t excl = incl - c;
                    const uint32_t E = __shfl_sync(full, incl, 31);
                    const unsigned some = __ballot_sync(full, c != 0u);
                    if (c != 0u)
                        s_rec[__popc(some & below)] =
                            make_uint4((turn ? 0u : r0) - excl, __float_as_uint(x0),
                                       __float_as_uint(x1), (unsigned)lane);
                    __syncwarp();
                    int started = -1;  // records whose first entry lies before the round, minus 1
#pragma unroll 1
                    for (uint32_t kb = 0; kb < E; kb += 32) {
                        const uint32_t d = excl - kb, k = kb + (uint32_t)lane;
                        const unsigned first =
                            __reduce_or_sync(full, (c != 0u && d < 32u) ? 1u << d : 0u);
                        const int ri = started + __popc(first & upto);
                        started += __popc(first);
                        uint4 rec = make_uint4(0u, 0u, 0u, 0u);
                        int4 v = make_int4(0, 0, 0, 0);
                        if (k < E) {
                            rec = s_rec[ri];
                            v = __ldg(reinterpret_cast<const int4*>(EE + (rec.x + k)));
                        }
                        const int bq = (int)((unsigned)v.y >> 16), qr = bq - range_lo;
                        const float mz = __int_as_float(v.x);
                        bool cand = k < E && bq >= range_lo && bq < range_hi;
                        if (MODIFIED && pass) {
                            // the shifted window exactly as matchms tests it:
                            // mz2 = mz_q + (prec_ref - prec_q) against mz_ref -+ tol
                            if (cand) {
                                const double mz2 = __dadd_rn(
                                    (double)mz, __dsub_rn(P.A.prec[a], P.B.prec[b_begin + bq]));
                                const double x = (double)__uint_as_float(rec.y);
                                cand = !(mz2 > __dadd_rn(x, P.tol)) && !(mz2 < __dsub_rn(x, P.tol));
                            }
                        } else {
                            cand = cand && mz >= __uint_as_float(rec.y) && mz <= __uint_as_float(rec.z);
                        }
                        double ea = 1.0;
                        if (EA && cand) ea = __ldg(EA + tbase + (rec.x + k));
                        const unsigned bal = __ballot_sync(full, cand);
                        const int slot = n + __popc(bal & below);
                        n += __popc(bal);
                        cand = cand && slot < pool_max;
                        // push onto the queries' chains: the slot is written into its
                        // query's 16-bit head and read back; where several lanes wrote
                        // the same head, those that do not find their slot go again,
                        // behind the one that got in.  The head read first, if of this
                        // epoch, is the chain's next element.  (A match_any of the
                        // queries instead: 6 to 13% slower.)
                        const unsigned claim = (epoch << 12) | (unsigned)slot;
                        unsigned ph = 0u;
                        if (cand) ph = head[qr];
                        __syncwarp();
                        if (cand) head[qr] = (uint16_t)claim;
                        __syncwarp();
                        bool lost = cand && head[qr] != claim;
                        while (__any_sync(full, lost)) {
                            if (lost) ph = head[qr];
                            __syncwarp();
                            if (lost) head[qr] = (uint16_t)claim;
                            __syncwarp();
                            lost = lost && head[qr] != claim;
                        }
                        if (cand) {
                            const int pB = v.y & 0xFFFF, pa = pc + (int)rec.w;
                            const double eb = __hiloint2double(v.w, v.z), wa = s_wa[rec.w];
                            double key;
                            uint32_t gen;
                            if (A_IS_REF) {
                                key = EA ? __dmul_rn(__dmul_rn(wa, ea), eb) : __dmul_rn(wa, eb);
                                gen = ((uint32_t)pa << 16) | (uint32_t)pB;
                                if (MODIFIED) gen |= (uint32_t)pass << 31;
                            } else {
                                key = EA ? __dmul_rn(ea, eb) : eb;
                                if (P.A.a) key = __dmul_rn(key, P.A.a[A.a0 + pa]);
                                key = __dmul_rn(key, wa);
                                gen = ((uint32_t)pB << 16) | (uint32_t)pa;
                            }
                            uint32_t m = (uint32_t)qr;
                            if ((ph >> 12) == epoch) m |= ((ph & 0xFFFu) << 12) | kHasNext;
                            pool.put(slot, key, gen, m);
                        }
                        if (n > pool_max) break;
                    }
                    __syncwarp();  // s_rec / s_wa are rewritten by the next turn or step
                    if (n > pool_max) break;
                }
                if (n > pool_max) break;
            }
            __syncwarp();
            if (n > pool_max) {
                if (rw > 1) {
                    // too many candidates for one pool: retry a narrower range
                    width = max(1, (int)((long long)rw * pool_max / (2LL * n)));
                    width = min(width, rw / 2 > 0 ? rw / 2 : 1);
                    continue;
                }
                // a single pair has more candidates than the pool: pair kernel
                if (lane == 0) {
                    spill_run(range_lo);
                    if (!SPARSE) P.dense.overflow[row() + range_lo] = 0;
                }
                __syncwarp();
                range_lo = range_hi;
                width = max(32, width);
                continue;
            }

            // ---- zeros for the dense row segment of the range: queries without
            // a candidate keep them; the runs' results, stored by this warp
            // after the __syncwarp below, overwrite theirs (a spilled pair's
            // overflow flag is rewritten by the pair kernel).  Written just
            // before the runs are resolved, so that the lines are still in L2
            // when the results land in them (zeroing before the sweep let L2
            // evict ~1/3 of them first: +40% DRAM traffic).  Four queries per
            // lane and 16-byte streaming stores from the first aligned query on,
            // whatever the row's own alignment.
            if (!SPARSE) {
                const int64_t r = row() + range_lo;
                auto zero1 = [&](int64_t o) {
                    __stcs(P.dense.score + o, 0.f);
                    __stcs(P.dense.matches + o, 0);
                    __stcs(P.dense.overflow + o, (unsigned char)0);
                };
                if (P.vec_rows) {
                    const int pre = min(rw, (int)(-r & 3));
                    const int nv = (rw - pre) >> 2;
                    if (lane < pre) zero1(r + lane);
                    for (int v = lane; v < nv; v += 32) {
                        const int64_t o = r + pre + 4 * v;
                        __stcs(reinterpret_cast<float4*>(P.dense.score + o),
                               make_float4(0.f, 0.f, 0.f, 0.f));
                        __stcs(reinterpret_cast<int4*>(P.dense.matches + o), make_int4(0, 0, 0, 0));
                        __stcs(reinterpret_cast<uchar4*>(P.dense.overflow + o),
                               make_uchar4(0, 0, 0, 0));
                    }
                    if (lane < ((rw - pre) & 3)) zero1(r + pre + 4 * nv + lane);
                } else {
                    for (int qr = lane; qr < rw; qr += 32) zero1(r + qr);
                }
            }
            __syncwarp();

            // ---- resolve each query's run ----
            // Slot s owns its query's run when the query's head names it (it
            // was pushed last).  Runs of one candidate, most of them, are
            // stored at once; the owners of longer runs are queued and taken 32
            // at a time, a lane walking its run's chain: 2 to 4 candidates are
            // resolved there in closed form (the queue keeps the lanes of that
            // code busy: an owner loop that did both ran it for a few lanes in
            // every step), 5..32 go to a second queue resolved by the warp, and
            // longer runs (or runs reaching match_limit) to the pair kernel.
            int n_mid = 0, n_big = 0, n_queue = 0;
            // Every queue is worked off at one place in the code, when it may not
            // take another step's slots or nothing is left to come: copies of it
            // wherever it is needed made three quarters of the kernel's code.
#pragma unroll 1
            for (int c = 0;; c += 32 * kIlpR) {
                const bool last = c >= n;
                if (!last) {
                    // kIlpR slots a lane, their loads in flight together
                    PoolEntry x[kIlpR];
                    double rnB[kIlpR];
                    bool own[kIlpR], more[kIlpR];
#pragma unroll
                    for (int u = 0; u < kIlpR; ++u) {
                        const int sl = c + 32 * u + lane;
                        own[u] = sl < n;
                        x[u] = PoolEntry{0.0, 0u, 0u};
                        if (own[u]) x[u] = pool.get(sl);
                    }
#pragma unroll
                    for (int u = 0; u < kIlpR; ++u) {
                        const int qr = meta_query(x[u].meta);
                        own[u] = own[u] && (head[qr] & 0xFFFu) == (unsigned)(c + 32 * u + lane);
                        more[u] = own[u] && ((x[u].meta & kHasNext) || P.match_limit <= 1);
                        rnB[u] = 0.0;
                        if (own[u] && !more[u]) rnB[u] = __ldg(P.rnB + b_begin + range_lo + qr);
                    }
#pragma unroll
                    for (int u = 0; u < kIlpR; ++u) {
                        if (own[u] && !more[u])
                            store_result(range_lo + meta_query(x[u].meta), x[u].key, 1, rnB[u]);
                        const unsigned mb = __ballot_sync(full, more[u]);
                        if (more[u])
                            queue[n_queue + __popc(mb & below)] = (uint16_t)(c + 32 * u + lane);
                        n_queue += __popc(mb);
                    }
                }
                if (!last && n_queue <= kQueue - 32 * kIlpR) continue;
                __syncwarp();
#pragma unroll 1
                for (int qc = 0;; qc += 32) {
                    const bool qlast = qc >= n_queue;
                    if (!qlast) {
                        int L = 0, q = 0, s = 0;
                        double rnB = 0.0;
                        double k0 = 0.0, k1 = 0.0, k2 = -INFINITY, k3 = -INFINITY;
                        uint32_t g0 = 0, g1 = 0, g2 = 0, g3 = 0;
                        if (qc + lane < n_queue) {
                            s = queue[qc + lane];
                            PoolEntry x = pool.get(s);
                            q = range_lo + meta_query(x.meta);
                            rnB = __ldg(P.rnB + b_begin + q);
                            k0 = x.key;
                            g0 = x.gen;
                            L = 1;
                            if (x.meta & kHasNext) {
                                x = pool.get(meta_next(x.meta));
                                k1 = x.key;
                                g1 = x.gen;
                                L = 2;
                                if (x.meta & kHasNext) {
                                    x = pool.get(meta_next(x.meta));
                                    k2 = x.key;
                                    g2 = x.gen;
                                    L = 3;
                                    if (x.meta & kHasNext) {
                                        x = pool.get(meta_next(x.meta));
                                        k3 = x.key;
                                        g3 = x.gen;
                                        L = 4;
                                        // longer runs: count on to kMidRun + 1
                                        uint32_t m = x.meta;
#pragma unroll 1
                                        while ((m & kHasNext) && L <= kMidRun) {
                                            m = pool.meta(meta_next(m));
                                            ++L;
                                        }
                                    }
                                }
                            }
                        }
                        __syncwarp();
                        const bool to_pair = L >= P.match_limit;
                        const bool is_long = L > 4 && !to_pair;
                        const bool is_mid = is_long && L <= kMidRun;
                        const unsigned mb = __ballot_sync(full, is_mid);
                        const unsigned bb = __ballot_sync(full, is_long && !is_mid);
                        const unsigned run = (unsigned)s | ((unsigned)L << 12);
                        if (is_mid)
                            long_runs[n_mid + __popc(mb & below)] = run;
                        else if (is_long)
                            long_runs[kLongRuns - 1 - (n_big + __popc(bb & below))] = run;
                        n_mid += __popc(mb);
                        n_big += __popc(bb);
                        if (to_pair) spill_run(q);
                        if (L != 0 && !is_long && !to_pair) {
                            // two to four candidates: sorting network (absent ones hold
                            // -infinity and stay last), then greedy
                            auto order = [](double& ka, uint32_t& ga, double& kb, uint32_t& gb) {
                                if (before(kb, gb, ka, ga)) {
                                    const double tk = ka;
                                    ka = kb;
                                    kb = tk;
                                    const uint32_t tg = ga;
                                    ga = gb;
                                    gb = tg;
                                }
                            };
                            auto clash = [](uint32_t ga, uint32_t gb) {
                                return gen_p1<MODIFIED>(ga) == gen_p1<MODIFIED>(gb) || ((ga ^ gb) & 0xFFFFu) == 0u;
                            };
                            order(k0, g0, k1, g1);
                            if (L > 2) {
                                order(k2, g2, k3, g3);
                                order(k0, g0, k2, g2);
                                order(k1, g1, k3, g3);
                                order(k1, g1, k2, g2);
                            }
                            double score = k0;
                            int mt = 1;
                            const bool take1 = !clash(g0, g1);
                            if (take1) {
                                score = __dadd_rn(score, k1);
                                mt = 2;
                            }
                            if (L > 2) {
                                const bool take2 = !clash(g0, g2) && !(take1 && clash(g1, g2));
                                if (take2) {
                                    score = __dadd_rn(score, k2);
                                    ++mt;
                                }
                                if (L > 3 && !clash(g0, g3) && !(take1 && clash(g1, g3)) && !(take2 && clash(g2, g3))) {
                                    score = __dadd_rn(score, k3);
                                    ++mt;
                                }
                            }
                            store_result(q, score, mt, rnB);
                        }
                    }
                    if (n_mid + n_big > kLongRuns - 32 || (qlast && last)) {
                        __syncwarp();
                        // Runs of 5..8 candidates are resolved four at a time on 8-lane segments,
                        // of 9..16 two at a time, longer ones by the whole warp; more than 32
                        // candidates, or match_limit, go to the pair kernel.  Their chains are
                        // walked first, a lane a run and 32 (8 longer) runs at a time, which leaves
                        // the slots of run i at lists[i + stride * j].  A walk per resolved run was
                        // a chain of up to 32 dependent reads each, and all pairs of a run were
                        // compared as float64 keys with their generation words: 8.83 -> 6.32 ms
                        // (9001 x 11003 modified cosine), 274 -> 237 us (1024 x 1024 uniform),
                        // 1.67 -> 1.48 ms (12288 symmetric).
#pragma unroll 1
                        for (int r0 = 0; r0 < n_mid + n_big;) {
                            const bool mid = r0 < n_mid;
                            const int stride = mid ? kLists / kMidRun : kLists / 32;
                            const int cnt = min(stride, (mid ? n_mid : n_mid + n_big) - r0);
                            int Lw = 0;  // length of the run this lane walked
                            if (lane < cnt) {
                                const unsigned e =
                                    long_runs[mid ? r0 + lane : kLongRuns - 1 - (r0 - n_mid + lane)];
                                int at = (int)(e & 0xFFFu);
                                uint32_t m;
#pragma unroll 1
                                do {
                                    lists[lane + stride * Lw] = (uint16_t)at;
                                    m = pool.meta(at);
                                    at = meta_next(m);
                                    ++Lw;
                                } while ((m & kHasNext) && Lw < 32);
                                if ((m & kHasNext) || Lw >= P.match_limit) {
                                    spill_run(range_lo + meta_query(m));
                                    Lw = 0;
                                }
                            }
                            __syncwarp();
                            const unsigned lt17 = __ballot_sync(full, Lw <= 16 && Lw != 0);
                            unsigned left = __ballot_sync(full, Lw != 0);
#pragma unroll 1
                            while (left) {
                                // the next runs: four of up to 8, two of up to 16, or one
                                int seg, run, most;
                                if (mid) {
                                    seg = 8;
                                    most = 8;
                                    const int f = (__ffs(left) - 1) & ~3;
                                    run = f + (lane >> 3);
                                    left &= 0xfffffff0u << f;
                                } else if (left & lt17) {
                                    seg = 16;
                                    most = 16;
                                    const unsigned two = left & lt17, rest = two & (two - 1u);
                                    run = __ffs(lane < 16 || !rest ? two : rest) - 1;
                                    if (lane >= 16 && !rest) run = 31;
                                    left &= ~(two ^ (rest & (rest - 1u)));
                                } else {
                                    seg = 32;
                                    most = 32;
                                    run = __ffs(left) - 1;
                                    left &= left - 1u;
                                }
                                const int tq = lane & (seg - 1), sb = lane - tq;
                                const int L = __shfl_sync(full, Lw, run);
                                double k = -INFINITY, rnB = 0.0;
                                uint32_t g = 0;
                                int q = 0;
                                const bool mine = tq < L;
                                if (mine) {
                                    const PoolEntry x = pool.get(lists[run + stride * tq]);
                                    k = x.key;
                                    g = x.gen;
                                    q = range_lo + meta_query(x.meta);
                                    rnB = __ldg(P.rnB + b_begin + q);
                                }
                                // The candidates that precede a lane's own in greedy order, as a mask
                                // of segment positions: by the key rounded to float32, which decides
                                // unless two round alike (then not all ranks occur), else exactly.
                                const float w = __double2float_rn(k);
                                unsigned prec = 0u;
#pragma unroll 1
                                for (int j = 0; j < most; j += 8) {
#pragma unroll
                                    for (int u = 0; u < 8; ++u)
                                        if (__shfl_sync(full, w, j + u, seg) > w) prec |= (1u << u) << j;
                                }
                                const unsigned here = __ballot_sync(full, mine);
                                const unsigned ranks =
                                    __reduce_or_sync(full, mine ? (1u << sb) << __popc(prec) : 0u);
                                if (ranks != here) {
                                    prec = 0u;
#pragma unroll 1
                                    for (int j = 0; j < most; ++j) {
                                        const double ok = __shfl_sync(full, k, j, seg);
                                        const uint32_t og = __shfl_sync(full, g, j, seg);
                                        if (j < L && before(ok, og, k, g)) prec |= 1u << j;
                                    }
                                }
                                prec <<= sb;
                                // the preceding lanes that share a peak with this one's (as two
                                // more comparisons per position: modified cosine 4% slower)
                                const unsigned clash =
                                    prec & (__match_any_sync(full, gen_p1<MODIFIED>(g)) |
                                            __match_any_sync(full, g & 0xFFFFu));
                                // A lane decides as soon as every preceding clashing lane has (the
                                // first always can), usually in two or three rounds.
                                unsigned dec = ~here, acc = 0u;
#pragma unroll 1
                                while (dec != full) {
                                    bool my_dec = (dec >> lane) & 1u, my_acc = (acc >> lane) & 1u;
                                    if (!my_dec && (clash & ~dec) == 0u) {
                                        my_dec = true;
                                        my_acc = (clash & acc) == 0u;
                                    }
                                    dec = __ballot_sync(full, my_dec);
                                    acc = __ballot_sync(full, my_acc);
                                }
                                // accepted keys are added in greedy order through s_wa
                                if ((acc >> lane) & 1u) s_wa[sb + __popc(prec & acc)] = k;
                                __syncwarp();
                                if (L && tq == 0) {
                                    const int mt = __popc(acc & here & (seg == 32 ? full : ((1u << seg) - 1u) << sb));
                                    double score = 0.0;
#pragma unroll 1
                                    for (int i = 0; i < mt; ++i) score = __dadd_rn(score, s_wa[sb + i]);
                                    store_result(q, score, mt, rnB);
                                }
                                __syncwarp();
                            }
                            r0 += cnt;
                        }
                        n_mid = 0;
                        n_big = 0;
                    }
                    if (qlast) break;
                }
                n_queue = 0;
                __syncwarp();
                if (last) break;
            }
            range_lo = range_hi;
            if (n < pool_max / 4) width = min(tn, width * 2);
        }
        __syncwarp();
        if (P.trace.rec && lane == 0) {
            const unsigned long long k = atomicAdd(P.trace.count, 1ull);
            if ((long long)k < P.trace.cap) {
                unsigned int smid;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
                unsigned long long* r = P.trace.rec + 4 * k;
                r[0] = (unsigned long long)P.trace.tag | ((unsigned long long)smid << 32);
                r[1] = item;
                r[2] = *s_t0;
                r[3] = global_ns();
            }
        }
    }
    if (P.slots) {  // give the global-pool slice back
        __syncthreads();
        if (threadIdx.x == 0 && pslot >= 0) {
            atomicAnd(&P.slots[pslot >> 5], ~(1u << (pslot & 31)));
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// 5. pair kernel: a CTA or a warp per pair
// ---------------------------------------------------------------------------
struct PairParams {
    SpecSet R;
    SpecSet Q;
    const double* snR;
    const double* snQ;
    double tol;
    double shift;
    int match_limit;
    int cap;  // candidates a buffer holds: a power of two >= match_limit, or list_cap
    int cache;  // pair_kernel: query m/z values kept in shared memory (pair_cache)
    int used_words;       // pair_kernel: words of each used-peak bitmap in shared memory
    uint32_t* long_bits;  // bitmaps of pairs with more peaks, kLongWords a greedy warp (or null)
    // launches for either kind of call (null: always run): the kernel returns
    // unless *gate == gate_value
    const uint32_t* gate;
    uint32_t gate_value;
    // work: either the spill list (pairs != nullptr) or every pair of R x Q
    const int2* pairs;
    const unsigned long long* n_pairs;  // SpillList::count
    unsigned int pairs_cap;
    unsigned long long* work;
    DenseOut dense;
    SparseOut sparse;
    uint32_t* err;
    const uint32_t* bad;
    int sym;  // only pairs (reference i, query j) with i <= j
    // test hook (CMS_TEST_STALL=pair): the pipelined kernel's greedy warp
    // leaves at once, so the producers' bounded waits run out
    int test_stall;
};

// Register-blocked bitonic sort of m = 8 * blockDim.x candidates, descending by
// (order key, gen), for the pair kernel: each thread holds the 8 consecutive
// elements 8t..8t+7 in registers.  Exchange distance j < 8: inside the
// thread; 8 <= j < 256: with lane t ^ (j / 8) of the same warp by shuffle;
// j >= 256: with thread t ^ (j / 8) of another warp through shared memory
// (element-major staging, so those accesses have no bank conflicts).  The
// network and the result are those of the plain shared-memory bitonic sort.
struct Cand {
    unsigned long long k;
    uint32_t g;
};
__device__ __forceinline__ bool cand_gt(const Cand& a, const Cand& b) {
    return a.k > b.k || (a.k == b.k && a.g > b.g);
}
// keep the larger of the pair (i, i ^ j) at the lower index when the block
// of kk elements containing i sorts descending
template <int J>
__device__ __forceinline__ void sort8_local(Cand (&c)[8], int base, int kk) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if (e & J) continue;
        const int f = e | J;
        const bool desc = ((base + e) & kk) == 0;
        const bool gt = cand_gt(c[e], c[f]);
        if (desc ? !gt : gt) {
            const Cand t = c[e];
            c[e] = c[f];
            c[f] = t;
        }
    }
}
// Barriers of the threads that generate and sort a pair's candidates: the
// whole block, or (pipelined pair kernel) the producer warps only, on named
// barrier 1.
struct BlockSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
struct WarpSync {
    __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
struct GroupSync {
    int n;  // participating threads (a multiple of 32)
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
    }
};

// nt threads (tid 0..nt-1) sort okey/cgen[0, m), m = 8 * nt, in registers.
template <typename Sync>
__device__ void sort8_block(unsigned long long* okey, uint32_t* cgen, int m, int nt, int tid,
                            Sync sync) {
    const int base = 8 * tid;
    const unsigned full = 0xffffffffu;
    Cand c[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        c[e].k = okey[base + e];
        c[e].g = cgen[base + e];
    }
    for (int kk = 2; kk <= m; kk <<= 1) {
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (j >= 8) {
                const int pt = tid ^ (j >> 3);
                const bool lower = (base & j) == 0;
                const bool desc = (base & kk) == 0;  // kk >= 16: the same for all e
                Cand o[8];
                if (j >= 256) {
                    sync();
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        okey[e * nt + tid] = c[e].k;
                        cgen[e * nt + tid] = c[e].g;
                    }
                    sync();
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        o[e].k = okey[e * nt + pt];
                        o[e].g = cgen[e * nt + pt];
                    }
                } else {
                    const int d = j >> 3;
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        o[e].k = __shfl_xor_sync(full, c[e].k, d);
                        o[e].g = __shfl_xor_sync(full, c[e].g, d);
                    }
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const bool gt = cand_gt(c[e], o[e]);
                    if ((lower == desc) ? !gt : gt) c[e] = o[e];
                }
            } else if (j == 4) {
                sort8_local<4>(c, base, kk);
            } else if (j == 2) {
                sort8_local<2>(c, base, kk);
            } else {
                sort8_local<1>(c, base, kk);
            }
        }
    }
    sync();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        okey[base + e] = c[e].k;
        cgen[base + e] = c[e].g;
    }
    sync();
}

constexpr int kGenPeaks = 2;  // reference peaks a thread takes per chunk
constexpr int kGenIlp = 4;    // candidates a thread has in flight while their keys are made

// Shared scratch of gen_pair: its chunk's reference peak weights, and (cache > 0)
// the query's first `cache` m/z values.
struct GenScratch {
    double* w;     // [kGenPeaks * threads]
    float* qmz;    // [cache]
    int cache;
};
__host__ __device__ constexpr size_t gen_scratch_bytes(int threads, int cache) {
    return (size_t)threads * 8 * kGenPeaks + (size_t)cache * 4;
}
__device__ __forceinline__ GenScratch gen_scratch(void* p, int threads, int cache) {
    GenScratch g;
    g.w = reinterpret_cast<double*>(p);
    g.qmz = reinterpret_cast<float*>(g.w + kGenPeaks * threads);
    g.cache = cache;
    return g;
}

// Candidates of pair (ri, qi) in generation order, truncated at `limit`,
// into okey/cgen, by nt threads (tid 0..nt-1, whole warps) with barrier
// `sync`; s_scan holds one int per warp.  Returns the number generated
// before truncation stopped it (>= limit: there may be more).
//
// A thread takes a reference peak and finds its window by binary search, in a
// shared-memory copy of the query's m/z where it fits (eleven dependent reads:
// from L2 they were most of the time).  It writes its candidates' generation
// words; the keys are then made one rank a thread, so that the weight loads are
// independent and no thread waits for one with more candidates.
template <bool MODIFIED, bool ONE, typename Sync>
__device__ int gen_pair(const PairParams& P, int64_t ri, int64_t qi, unsigned long long* okey,
                        uint32_t* cgen, int limit, int nt, int tid, int* s_scan,
                        const GenScratch& G, Sync sync) {
    const int lane = tid & 31, wid = tid >> 5, nwarps = nt >> 5;
    const unsigned full = 0xffffffffu;
    const int64_t r0 = P.R.off[ri], q0 = P.Q.off[qi];
    const int nr = (int)(P.R.off[ri + 1] - r0), nq = (int)(P.Q.off[qi + 1] - q0);
    const float* qmz = P.Q.mz + q0;
    if (nr == 0 || nq == 0) return 0;
    if (nq <= G.cache) {
        for (int i = tid; i < nq; i += nt) G.qmz[i] = qmz[i];
        qmz = G.qmz;
        sync();
    }
    int total = 0;
    bool overflow = false;
    // modified cosine generates twice: at shift 0, then at the pair's
    // precursor difference, continuing the same candidate list
#pragma unroll 1
    for (int pass = 0; pass < (MODIFIED ? 2 : 1) && !overflow; ++pass) {
        const double shift = (MODIFIED && pass) ? __dsub_rn(P.R.prec[ri], P.Q.prec[qi]) : P.shift;
#pragma unroll 1
        for (int pc = 0; pc < nr && !overflow; pc += kGenPeaks * nt) {
            // kGenPeaks consecutive peaks a thread (a pair that overflows is usually
            // done after one chunk of 256), or (ONE) one where that is enough: a
            // thread's peaks are searched for one after the other (300 x 301 uniform
            // spectra, the whole matrix at match_limit 2048: 1250 us with two, 1070
            // with one; spilled pairs: 183 us with two, 192 with one for 12345
            // symmetric spectra, 193 and 189 for modified cosine)
            const bool one = ONE && nr - pc <= nt;
            auto peak = [&](int u) { return (one ? tid : kGenPeaks * tid) + u; };  // in the chunk
            int start[kGenPeaks], cnt[kGenPeaks], mine = 0;
            float mz[kGenPeaks];
#pragma unroll
            for (int u = 0; u < kGenPeaks; ++u) {
                const int p1 = pc + peak(u);
                mz[u] = p1 < nr ? P.R.mz[r0 + p1] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < kGenPeaks; ++u) {
                const int p1 = pc + peak(u);
                start[u] = cnt[u] = 0;
                if (p1 < nr && (u == 0 || !one)) {
                    const double mz1 = (double)mz[u];
                    // the window as float32 bounds of the query's m/z (exact, see
                    // Window): first p2 at or above, then on to the last one inside.
                    // (With a shift the search for the lower bound may end early next
                    // to zero, where float32 is finer than the float64 sums.)
                    float wl, wh;
                    const bool ok =
                        shift == 0.0
                            ? Window<true, true>::bounds(mz[u], P.tol, shift, wl, wh)
                            : Window<true, false>::bounds(mz[u], P.tol, shift, wl, wh) &&
                                  !Window<true, false>::not_below(nextafterf(wl, -INFINITY),
                                                                  __dsub_rn(mz1, P.tol), 0.0, P.tol,
                                                                  shift);
                    int L = 0, H = nq;
                    if (ok) {
                        while (L < H) {
                            const int M = (L + H) >> 1;
                            if (qmz[M] < wl)
                                L = M + 1;
                            else
                                H = M;
                        }
                        start[u] = L;
                        while (L < nq && !(qmz[L] > wh)) ++L;
                    } else {  // no such bounds: as the definition tests it
                        const double lo = __dsub_rn(mz1, P.tol), hi = __dadd_rn(mz1, P.tol);
                        while (L < H) {
                            const int M = (L + H) >> 1;
                            if (__dadd_rn((double)qmz[M], shift) < lo)
                                L = M + 1;
                            else
                                H = M;
                        }
                        start[u] = L;
                        while (L < nq && !(__dadd_rn((double)qmz[L], shift) > hi)) ++L;
                    }
                    cnt[u] = L - start[u];
                    if (cnt[u])
                        G.w[peak(u)] = __dmul_rn(peak_a(P.R.a, r0 + p1), P.R.b[r0 + p1]);
                }
                mine += cnt[u];
            }
            // exclusive scan of the counts over the nt threads
            int incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(full, incl, d);
                if (lane >= d) incl += v;
            }
            if (lane == 31) s_scan[wid] = incl;
            sync();
            int chunk_total = 0, first = incl - mine;
            for (int w = 0; w < nwarps; ++w) {
                const int x = s_scan[w];
                if (w < wid) first += x;
                chunk_total += x;
            }
            const int take = min(chunk_total, limit - total);
#pragma unroll
            for (int u = 0; u < kGenPeaks; ++u) {
                uint32_t gen = ((uint32_t)pass << 31) |
                               ((uint32_t)(pc + peak(u)) << 16) | (uint32_t)start[u];
                const int last = min(take, first + cnt[u]);
#pragma unroll 1
                for (int i = first; i < last; ++i) cgen[total + i] = gen++;
                first += cnt[u];
            }
            sync();
#pragma unroll 1
            for (int i0 = tid; i0 < take; i0 += kGenIlp * nt) {
                double w[kGenIlp], qa[kGenIlp], qb[kGenIlp];
#pragma unroll
                for (int u = 0; u < kGenIlp; ++u) {
                    const int i = i0 + u * nt;
                    w[u] = qa[u] = qb[u] = 1.0;
                    if (i < take) {
                        const uint32_t g = cgen[total + i];
                        qb[u] = P.Q.b[q0 + (g & 0xFFFFu)];
                        if (P.Q.a) qa[u] = P.Q.a[q0 + (g & 0xFFFFu)];
                        w[u] = G.w[(int)gen_p1<MODIFIED>(g) - pc];
                    }
                }
#pragma unroll
                for (int u = 0; u < kGenIlp; ++u) {
                    const int i = i0 + u * nt;
                    if (i < take)
                        okey[total + i] = order_key(__dmul_rn(__dmul_rn(w[u], qa[u]), qb[u]));
                }
            }
            total += chunk_total;
            if (total >= limit) overflow = true;
            sync();
        }
    }
    return total;
}

// the in-thread stages of sort8_words (exchange distance J < 8)
template <int J>
__device__ __forceinline__ void words_local(unsigned long long (&c)[8], int base, int kk) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if (e & J) continue;
        const int f = e | J;
        const bool desc = ((base + e) & kk) == 0;
        const bool gt = c[e] > c[f];
        if (desc ? !gt : gt) {
            const unsigned long long t = c[e];
            c[e] = c[f];
            c[f] = t;
        }
    }
}

// Register-blocked bitonic sort, descending, of m = 8 * nt single 64-bit words
// (thread t holds network positions 8t..8t+7), exchanging through `scratch`
// (m words) for distances of 256 and more; the sorted words end in the
// threads' registers, position 8t + e in c[e] of thread t.
template <typename Sync>
__device__ void sort8_words(unsigned long long* scratch, unsigned long long (&c)[8], int m,
                            int nt, int tid, Sync sync) {
    const int base = 8 * tid;
    const unsigned full = 0xffffffffu;
    for (int kk = 2; kk <= m; kk <<= 1) {
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (j >= 8) {
                const int pt = tid ^ (j >> 3);
                const bool lower = (base & j) == 0;
                const bool desc = (base & kk) == 0;
                unsigned long long o[8];
                if (j >= 256) {
                    sync();
#pragma unroll
                    for (int e = 0; e < 8; ++e) scratch[e * nt + tid] = c[e];
                    sync();
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] = scratch[e * nt + pt];
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) o[e] = __shfl_xor_sync(full, c[e], j >> 3);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const bool gt = c[e] > o[e];
                    if ((lower == desc) ? !gt : gt) c[e] = o[e];
                }
            } else if (j == 4) {
                words_local<4>(c, base, kk);
            } else if (j == 2) {
                words_local<2>(c, base, kk);
            } else {
                words_local<1>(c, base, kk);
            }
        }
    }
}

// Sorts the m = 8 * nt candidates of okey/cgen (padded past n with zeros)
// into greedy order by sorting one 64-bit word per candidate: the order key
// without its top bit (set for every key >= +0.0) and without its low R + 1
// bits, then a "real candidate" bit, then the R-bit index (m = 2^R), so
// equal words' order is the index order, i.e. generation order, and padding
// sorts last.  Keys that agree in every kept bit but differ in a dropped one
// would be misordered: the pass checks every pair of neighbours for that
// (and for a key below +0.0) and returns false, leaving okey/cgen untouched,
// if it finds one; the caller then sorts the pairs themselves.  On success
// okey/cgen hold the candidates in greedy order.
template <typename Sync>
__device__ bool sort8_by_word(unsigned long long* okey, uint32_t* cgen,
                              unsigned long long* scratch, int* s_flag, int n, int m, int nt,
                              int tid, Sync sync) {
    const int rb = 31 - __clz(m);  // index bits
    const unsigned long long imask = (1ull << rb) - 1ull;
    const unsigned long long real = 1ull << rb;
    const unsigned long long kmask = ~((real << 1) - 1ull);
    if (tid == 0) *s_flag = 0;
    sync();
    unsigned long long c[8];
    bool bad = false;
    // which candidate starts at which network position is free (every word
    // carries its index): thread tid takes candidates e * nt + tid, so that
    // the loads of consecutive threads are consecutive words
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = e * nt + tid;
        if (i < n) {
            const unsigned long long k = okey[i];
            bad |= (k >> 63) == 0ull;
            c[e] = ((k << 1) & kmask) | real | (unsigned long long)i;
        } else {
            c[e] = (unsigned long long)i;  // padding: below every real word
        }
    }
    if (bad) atomicOr(s_flag, 1);
    sort8_words(scratch, c, m, nt, tid, sync);
    // neighbours that tie in the kept bits must have equal keys; the word
    // after this thread's last is the next thread's first
    sync();
    scratch[tid] = c[0];
    sync();
    const unsigned long long after = tid + 1 < nt ? scratch[tid + 1] : 0ull;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = 8 * tid + e;
        if (i + 1 < m && (c[e] & real)) {
            const unsigned long long nx = e < 7 ? c[e + 1] : after;
            if ((nx & real) && ((nx ^ c[e]) & kmask) == 0ull &&
                okey[nx & imask] != okey[c[e] & imask])
                bad = true;
        }
    }
    if (bad) atomicOr(s_flag, 1);
    sync();
    if (*s_flag) return false;
    // the sorted words to scratch, position p at p + p / 8 (the stores of
    // positions 8 * tid + e, nine words apart, fall in different banks), then
    // each thread gathers positions e * nt + tid, so that the final stores of
    // consecutive threads are consecutive
#pragma unroll
    for (int e = 0; e < 8; ++e) scratch[9 * tid + e] = c[e];
    sync();
    unsigned long long k[8];
    uint32_t g[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int pos = e * nt + tid;
        const unsigned long long w = scratch[pos + (pos >> 3)];
        const bool r = (w & real) != 0ull;
        const int src = (int)(w & imask);
        k[e] = r ? okey[src] : 0ull;
        g[e] = r ? cgen[src] : 0u;
    }
    sync();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        okey[e * nt + tid] = k[e];
        cgen[e * nt + tid] = g[e];
    }
    sync();
    return true;
}

// Bitonic sort, descending, of 8 * nt 32-bit words (thread t ends with positions
// 8t..8t+7), exchanging through `scratch` (8 * nt words) for distances of 256 and
// more.
template <int J>
__device__ __forceinline__ void words32_local(uint32_t (&c)[8], int base, int kk) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        if (e & J) continue;
        const uint32_t hi = max(c[e], c[e | J]), lo = min(c[e], c[e | J]);
        const bool desc = ((base + e) & kk) == 0;
        c[e] = desc ? hi : lo;
        c[e | J] = desc ? lo : hi;
    }
}
template <typename Sync>
__device__ __forceinline__ void sort8_words32(uint32_t* scratch, uint32_t (&c)[8], int m, int nt,
                                              int tid, Sync sync) {
    const int base = 8 * tid;
    const unsigned full = 0xffffffffu;
#pragma unroll 1
    for (int kk = 2; kk <= m; kk <<= 1) {
#pragma unroll 1
        for (int j = kk >> 1; j >= 8; j >>= 1) {
            const bool keep_max = ((base & j) == 0) == ((base & kk) == 0);
            if (j >= 256) {
                const int pt = tid ^ (j >> 3);
                sync();
#pragma unroll
                for (int e = 0; e < 8; ++e) scratch[e * nt + tid] = c[e];
                sync();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t o = scratch[e * nt + pt];
                    c[e] = keep_max ? max(c[e], o) : min(c[e], o);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const uint32_t o = __shfl_xor_sync(full, c[e], j >> 3);
                    c[e] = keep_max ? max(c[e], o) : min(c[e], o);
                }
            }
        }
        if (kk >= 8) words32_local<4>(c, base, kk);
        if (kk >= 4) words32_local<2>(c, base, kk);
        words32_local<1>(c, base, kk);
    }
}

// Sorts the m = 8 * nt candidates of okey/cgen (n real ones) into greedy order
// through one 32-bit word each: the key's float32 (rounded down) without its low
// R - 1 bits, plus one, above the R-bit index (m = 2^R), zero for padding.  That
// is the order up to keys whose kept bits tie (about ten neighbours of 1024); the
// exact (key, gen) order is then restored by odd-even exchanges of neighbours,
// which end when a pass exchanges nothing.  False, with okey/cgen untouched, when
// eight passes are not enough or a key is negative or not finite in float32.
// Against the 64-bit words of sort8_by_word a compare-exchange is two
// instructions instead of seven and a shuffle one instead of two.
constexpr int kFixPasses = 8;
template <typename Sync>
__device__ bool sort8_by_float(unsigned long long* okey, uint32_t* cgen, void* scratch, int* s_flags,
                               int n, int m, int nt, int tid, Sync sync) {
    const int rb = 31 - __clz(m);
    if (tid <= kFixPasses) s_flags[tid] = 0;
    sync();
    uint32_t c[8];
    bool bad = false;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = e * nt + tid;
        c[e] = (uint32_t)i;
        if (i < n) {
            const unsigned long long k = okey[i];
            const uint32_t f = __float_as_uint(__double2float_rd(key_from_order(k)));
            bad = bad || f > 0x7f7fffffu || (k >> 63) == 0ull;
            c[e] |= ((f >> (rb - 1)) + 1u) << rb;
        }
    }
    if (bad) s_flags[kFixPasses] = 1;
    sync();
    if (s_flags[kFixPasses]) return false;
    sort8_words32(reinterpret_cast<uint32_t*>(scratch), c, m, nt, tid, sync);
    Cand x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int i = (int)(c[e] & (uint32_t)(m - 1));
        const bool real = c[e] >= (uint32_t)m;
        x[e].k = real ? okey[i] : 0ull;
        x[e].g = real ? cgen[i] : 0u;
    }
    // ends of each thread's eight, for the exchange with its neighbours
    unsigned long long* ek = reinterpret_cast<unsigned long long*>(scratch);  // [2 * nt]
    uint32_t* eg = reinterpret_cast<uint32_t*>(ek + 2 * nt);                  // [2 * nt]
    auto order = [&](Cand& a, Cand& b, bool& any) {
        if (cand_gt(b, a)) {
            const Cand t = a;
            a = b;
            b = t;
            any = true;
        }
    };
#pragma unroll 1
    for (int pass = 0; pass < kFixPasses; ++pass) {
        bool any = false;
#pragma unroll
        for (int e = 0; e < 8; e += 2) order(x[e], x[e + 1], any);
#pragma unroll
        for (int e = 1; e < 7; e += 2) order(x[e], x[e + 1], any);
        sync();  // the words' or the last pass's readers are done with scratch
        ek[2 * tid] = x[0].k;
        eg[2 * tid] = x[0].g;
        ek[2 * tid + 1] = x[7].k;
        eg[2 * tid + 1] = x[7].g;
        sync();
        if (tid + 1 < nt) {
            const Cand next{ek[2 * tid + 2], eg[2 * tid + 2]};
            if (cand_gt(next, x[7])) {
                x[7] = next;
                any = true;
            }
        }
        if (tid > 0) {
            const Cand prev{ek[2 * tid - 1], eg[2 * tid - 1]};
            const Cand mine{ek[2 * tid], eg[2 * tid]};
            if (cand_gt(mine, prev)) x[0] = prev;
        }
        if (any) s_flags[pass] = 1;
        sync();
        if (!s_flags[pass]) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                okey[8 * tid + e] = x[e].k;
                cgen[8 * tid + e] = x[e].g;
            }
            sync();
            return true;
        }
    }
    return false;
}

// Pads okey/cgen[n, m) and sorts [0, m) descending by (okey, gen), m the
// power of two >= n: in registers when m = 8 * nt, else in shared memory.
template <typename Sync>
__device__ void sort_pair(unsigned long long* okey, uint32_t* cgen, int n, int m, int nt, int tid,
                          Sync sync) {
    for (int i = n + tid; i < m; i += nt) {
        okey[i] = 0ull;
        cgen[i] = 0u;
    }
    sync();
    if (m == 8 * nt) {
        sort8_block(okey, cgen, m, nt, tid, sync);
        return;
    }
    for (int k = 2; k <= m; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < m; i += nt) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long ka = okey[i], kb = okey[ixj];
                    const uint32_t ga = cgen[i], gb = cgen[ixj];
                    const bool a_gt_b = ka > kb || (ka == kb && ga > gb);
                    const bool desc = (i & k) == 0;
                    if (desc ? !a_gt_b : a_gt_b) {
                        okey[i] = kb;
                        okey[ixj] = ka;
                        cgen[i] = gb;
                        cgen[ixj] = ga;
                    }
                }
            }
            sync();
        }
    }
}

constexpr int kFill = 2;                    // chunks of 32 candidates looked at together
constexpr int kQueued = 32 * (kFill + 1);  // at most 31 waiting, plus one look's candidates
// Greedy by one warp over the sorted candidates.  used_r / used_q, zeroed for
// the pair's peaks, hold the peaks taken, in shared memory or (GLOBAL) in device
// memory.
//
// Most candidates have a taken peak when their turn comes, so the live ones are
// first queued (their positions, in order; `queue` holds kQueued) and resolved 32 at a
// time: a candidate is accepted iff no earlier accepted one of the batch shares
// its reference or query peak.  Conflict masks come from __match_any_sync, and
// lanes decide in rounds, each lane as soon as every earlier conflicting lane has
// decided (the lowest undecided lane always can, so this ends; usually after two
// or three rounds).  Accepted keys are summed in sorted order, as the sequential
// greedy; every lane ends with the same score and match count.
template <bool MODIFIED, bool GLOBAL>
__device__ __forceinline__ void greedy_pair(unsigned long long* okey, const uint32_t* cgen,
                                            uint32_t* used_r, uint32_t* used_q, uint16_t* queue,
                                            int n, double& score, int& matches) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    // from device memory past the L1 cache, which other multiprocessors' and
    // earlier pairs' writes do not reach
    auto word = [](const uint32_t* p) { return GLOBAL ? __ldcg(p) : *p; };
    auto free_peaks = [&](uint32_t g) {
        const int p1 = (int)gen_p1<MODIFIED>(g), p2 = (int)(g & 0xFFFFu);
        return (((word(used_r + (p1 >> 5)) >> (p1 & 31)) | (word(used_q + (p2 >> 5)) >> (p2 & 31))) &
                1u) == 0u;
    };
    int queued = 0, c = 0;
#pragma unroll 1
    for (;;) {
#pragma unroll 1
        while (queued < 32 && c < n) {
            bool live[kFill];
#pragma unroll
            for (int u = 0; u < kFill; ++u) {
                const int i = c + 32 * u + lane;
                live[u] = i < n && free_peaks(cgen[i]);
            }
#pragma unroll
            for (int u = 0; u < kFill; ++u) {
                const unsigned bal = __ballot_sync(full, live[u]);
                if (live[u]) queue[queued + __popc(bal & below)] = (uint16_t)(c + 32 * u + lane);
                queued += __popc(bal);
            }
            c += 32 * kFill;
        }
        __syncwarp();
        if (queued == 0) break;
        const int take = min(queued, 32);
        const int pos = lane < take ? queue[lane] : 0;
        const uint32_t g = cgen[pos];
        const double key = key_from_order(okey[pos]);
        const unsigned p1 = gen_p1<MODIFIED>(g), p2 = g & 0xFFFFu;
        // those queued before the last batch may have lost a peak to it
        const bool alive = lane < take && free_peaks(g);
        const unsigned live = __ballot_sync(full, alive);
        // dead lanes get values no peak index takes, so they match only themselves
        const unsigned m1 = __match_any_sync(full, alive ? p1 : 0x10000u + lane);
        const unsigned m2 = __match_any_sync(full, alive ? p2 : 0x10000u + lane);
        const unsigned earlier = (m1 | m2) & live & below;
        unsigned dec = ~live, acc = 0u;
#pragma unroll 1
        while (dec != full) {
            bool my_dec = (dec >> lane) & 1u, my_acc = (acc >> lane) & 1u;
            if (!my_dec && (earlier & ~dec) == 0u) {
                my_dec = true;
                my_acc = (earlier & acc) == 0u;
            }
            dec = __ballot_sync(full, my_dec);
            acc = __ballot_sync(full, my_acc);
        }
        if ((acc >> lane) & 1u) {
            atomicOr(&used_r[p1 >> 5], 1u << (p1 & 31));
            atomicOr(&used_q[p2 >> 5], 1u << (p2 & 31));
        }
        // accepted keys, in order, over the keys of resolved candidates (there are
        // at least as many of those, all before the first one queued)
        __syncwarp();
        if ((acc >> lane) & 1u)
            okey[matches + __popc(acc & below)] = (unsigned long long)__double_as_longlong(key);
        matches += __popc(acc);
        // the rest of the queue moves up
        uint16_t rest[kFill];
#pragma unroll
        for (int u = 0; u < kFill; ++u)
            rest[u] = 32 * u + lane < queued - take ? queue[32 * (u + 1) + lane] : (uint16_t)0;
        __syncwarp();
        queued -= take;
#pragma unroll
        for (int u = 0; u < kFill; ++u)
            if (32 * u + lane < queued) queue[32 * u + lane] = rest[u];
        __syncwarp();
    }
    // one serial chain of additions, its operands read ahead
#pragma unroll 8
    for (int i = 0; i < matches; ++i)
        score = __dadd_rn(score, __longlong_as_double((long long)okey[i]));
}

// Spectra of up to 8192 peaks have their bitmaps in shared memory; bitmaps for
// every peak index there (16 KB a greedy warp) would halve the resident CTAs.
// Longer ones have theirs in device memory, which the L2 cache holds: 64 pairs of
// 20000 peaks with a candidate each take 0.34 ms at match_limit 2048 and 1.27 ms at
// 16384 (of 8190 peaks 0.20 and 0.52; without bitmaps, each candidate compared
// with every accepted one, 8.9 and 567 ms).  Out of line: the callers' registers
// are for the ordinary case.
constexpr int kUsedWords = kLongPeaks / 32;  // words of each bitmap in shared memory
constexpr int kFullWords = 2048;  // words that hold every peak index
constexpr int kLongWords = 2 * kFullWords;
// greedy warps a multiprocessor with bitmaps in device memory: at 80 registers 25
// warps fit, of which at most every second is one
constexpr int kLongWarps = 12;
struct Greedy {
    double score;
    int matches;
};
template <bool MODIFIED>
__device__ __noinline__ Greedy greedy_long(unsigned long long* okey, const uint32_t* cgen,
                                           uint32_t* bits, uint16_t* queue, int n) {
    Greedy r{0.0, 0};
    greedy_pair<MODIFIED, true>(okey, cgen, bits, bits + kFullWords, queue, n, r.score, r.matches);
    return r;
}
inline bool may_be_long(const SpecSet& s) { return s.n_peaks > 32 * kUsedWords; }
constexpr size_t long_bits_bytes(int sms) {
    return (size_t)sms * kLongWarps * kLongWords * sizeof(uint32_t);
}

// The pair's outputs (dense, or a sparse hit above the threshold).
template <bool SPARSE>
__device__ void write_pair(const PairParams& P, int64_t ri, int64_t qi, int n, double score,
                           int matches, bool overflow) {
    float sc = 0.f;
    if (matches > 0 || n > 0) {
        const double denom = __dmul_rn(P.snR[ri], P.snQ[qi]);
        sc = (n > 0) ? (float)__ddiv_rn(score, denom) : 0.f;
    }
    if (!SPARSE) {
        const int64_t o = ri * P.dense.ld + qi;
        P.dense.score[o] = sc;
        P.dense.matches[o] = matches;
        P.dense.overflow[o] = overflow ? 1 : 0;
    } else if (n > 0 && sc >= P.sparse.threshold) {
        emit_hit(P.sparse, (int)ri, (int)qi, sc, matches, overflow ? 1 : 0);
    }
}

// item -> pair (reference ri, query qi); false for pairs under the diagonal
// of a symmetric whole-matrix launch (copied afterwards)
__device__ __forceinline__ bool pair_of(const PairParams& P, int64_t item, int64_t& ri,
                                        int64_t& qi) {
    if (P.pairs) {
        const int2 pr = P.pairs[item];
        ri = pr.x;
        qi = pr.y;
        return true;
    }
    ri = item / P.Q.n;
    qi = item - ri * P.Q.n;
    return !(P.sym && ri > qi);
}

constexpr int kPairCache = 1024;  // query m/z values pair_kernel keeps in shared memory
constexpr int kPairSlice = 512;   // candidates a warp takes on alone, at most
constexpr int kDeferred = 64;     // pairs with more that a CTA collects

// Shared memory of pair_kernel: candidates, used-peak bitmaps, gen_pair's scratch,
// the warps' greedy queues.
constexpr size_t pair_smem_bytes(int cap, int threads, int cache, int used_words = kUsedWords) {
    return (size_t)cap * 12 + (size_t)used_words * 8 + gen_scratch_bytes(threads, cache) +
           (size_t)threads / 32 * kQueued * sizeof(uint16_t);
}
constexpr int kMaxPairWarps = 16;
static_assert(2 * kUsedWords / kMaxPairWarps / 2 * 32 >= kHeavyPeaks,
              "a light pair's bitmaps fit every warp's share");
// Candidates the buffer holds when pair_kernel takes a spill list: a warp's share
// is as large as match_limit, up to kPairSlice, so that small limits leave no pair
// to the CTAs for want of room (1500 x 1501 uniform spectra at match_limit 16 and
// tolerance 0.5, nearly all pairs spilled: 7.2 ms with a share of 4, 3.0 with 16).
constexpr int list_cap(int cap, int threads) {
    return std::max(cap, threads / 32 * std::min(kPairSlice, cap));
}
// the query's m/z are kept where they fit
constexpr int pair_cache(int cap, int threads, size_t optin) {
    return pair_smem_bytes(cap, threads, kPairCache) <= optin ? kPairCache : 0;
}

// Pairs of the spill list (LIST), or of the whole matrix, where the pipelined kernel
// below does not fit.  Most spilled pairs have somewhat more candidates than the
// join resolves; a CTA spent 15 us on each, most of it at barriers and behind
// the one greedy warp.  So CTAs take only the heavy pairs, first, and then every
// warp takes light ones of its own into a share of the candidate buffer; a pair
// with more candidates than that holds (512 of 2048) is left to the CTA.  With
// the bitmaps of 8192 peaks, 1024 query m/z in shared memory and 80
// registers six CTAs fit an SM (five before): the pairs of 12345 symmetric spectra
// take 180 us (305 before), of sparse 20000 x 20000 113 (216), of modified cosine
// 297 (421).  What is left is the longest heavy pairs.
template <bool SPARSE, bool MODIFIED, bool LIST>
__global__ void __maxnreg__(80) pair_kernel(PairParams P) {
    if (*P.bad || (P.gate && *P.gate != P.gate_value)) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned long long* okey = reinterpret_cast<unsigned long long*>(smem_raw);
    uint32_t* cgen = reinterpret_cast<uint32_t*>(okey + P.cap);
    uint32_t* used = cgen + P.cap;
    const int used_words = 2 * P.used_words;
    const GenScratch gen = gen_scratch(used + used_words, blockDim.x, P.cache);
    uint16_t* queues = reinterpret_cast<uint16_t*>(gen.qmz + P.cache);
    __shared__ int s_scan[32];
    __shared__ int s_deferred[kDeferred];
    __shared__ int s_n_deferred, s_done;

    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    // an overrun list (an error that is reported) has gaps: nothing of it is read
    const bool list = LIST && P.pairs;
    const unsigned long long count = list ? *P.n_pairs : 0ull;
    const unsigned int front = (unsigned int)count, back = (unsigned int)(count >> 32);
    const bool sound = (unsigned long long)front + back <= (list ? P.pairs_cap : 0u);
    const int64_t n_heavy = !list ? P.R.n * P.Q.n : sound ? front : 0;
    const int64_t n_light = sound ? back : 0;
    // a warp's share: a power of two (the sorts pad to one)
    int slice = kPairSlice;
    while (slice * nw > P.cap) slice >>= 1;
    const int share = used_words / nw;

    // candidates, order, greedy and output of a pair, by nt threads; false if
    // it has as many candidates as `limit` below match_limit
    auto resolve = [&](int64_t ri, int64_t qi, int limit, unsigned long long* k, uint32_t* g,
                       uint32_t* used_r, int words, const GenScratch& G, int nt, int t, int* scan,
                       uint16_t* queue, auto sync) {
        const int total = gen_pair<MODIFIED, !LIST>(P, ri, qi, k, g, limit, nt, t, scan, G, sync);
        if (total >= limit && limit < P.match_limit) return false;
        const int n = min(total, P.match_limit);
        double score = 0.0;
        int matches = 0;
        if (n > 0) {
            const int nr = (int)(P.R.off[ri + 1] - P.R.off[ri]);
            const int nq = (int)(P.Q.off[qi + 1] - P.Q.off[qi]);
            // a warp's pairs are light ones, whose peaks fit its share of the bitmaps
            constexpr bool kCta = std::is_same<decltype(sync), BlockSync>::value;
            const bool fits = !kCta || max(nr, nq) <= 32 * (words / 2);
            uint32_t* const bits_r = fits ? used_r : P.long_bits + (size_t)blockIdx.x * kLongWords;
            uint32_t* const bits_q = bits_r + (fits ? words / 2 : kFullWords);
            for (int i = t; i < (nr + 31) / 32; i += nt) bits_r[i] = 0u;
            for (int i = t; i < (nq + 31) / 32; i += nt) bits_q[i] = 0u;
            int m = 1;
            while (m < n) m <<= 1;
            sort_pair(k, g, n, m, nt, t, sync);
            if (t < 32) {
                if (fits) {
                    greedy_pair<MODIFIED, false>(k, g, used_r, used_r + words / 2, queue, n, score,
                                                 matches);
                } else {
                    const Greedy r = greedy_long<MODIFIED>(k, g, bits_r, queue, n);
                    score = r.score;
                    matches = r.matches;
                }
            }
        }
        if (t == 0) write_pair<SPARSE>(P, ri, qi, n, score, matches, total >= P.match_limit);
        sync();
        return true;
    };

    auto whole = [&](int64_t item) {
        int64_t ri, qi;
        if (pair_of(P, item, ri, qi))
            resolve(ri, qi, P.match_limit, okey, cgen, used, used_words, gen, blockDim.x, tid, s_scan,
                    queues, BlockSync{});
    };
    __shared__ unsigned long long s_item;
    int n_whole = 0;
    // One loop for the three sources of pairs that the CTA takes as a whole, so
    // that their code is there once: the whole matrix at a static stride, the
    // heavy pairs one by one, those deferred by the warps.
    bool heavy = true, done = false;
    if (tid == 0) s_n_deferred = s_done = 0;
    for (int64_t iter = 0;; ++iter) {
        int64_t item = -1;
        if (heavy) {
            item = blockIdx.x + iter * gridDim.x;
            if (list) {
                __syncthreads();
                if (tid == 0) s_item = atomicAdd(P.work, 1ull);
                __syncthreads();
                item = (int64_t)s_item;
            }
            heavy = item < n_heavy;
            if (!heavy) item = -1;
        }
        if (!heavy) {
            if (!list) break;
            if (n_whole == 0) {
                if (done) break;
                const GenScratch G{gen.w + kGenPeaks * 32 * wid, gen.qmz + P.cache / nw * wid,
                                   P.cache / nw};
                for (;;) {
                    int i = -1;
                    if (lane == 0 && *(volatile int*)&s_n_deferred <= kDeferred - nw) {
                        const unsigned long long k = atomicAdd(P.work + 1, 1ull);
                        if ((int64_t)k < n_light)
                            i = (int)(P.pairs_cap - 1 - (unsigned int)k);
                        else
                            s_done = 1;
                    }
                    i = __shfl_sync(0xffffffffu, i, 0);
                    if (i < 0) break;
                    const int2 pr = P.pairs[i];
                    if (!resolve(pr.x, pr.y, min(slice, P.match_limit), okey + slice * wid,
                                 cgen + slice * wid, used + share * wid, share, G, 32, lane,
                                 s_scan + wid, queues + kQueued * wid, WarpSync{}) &&
                        lane == 0)
                        s_deferred[atomicAdd(&s_n_deferred, 1)] = i;
                }
                __syncthreads();
                n_whole = s_n_deferred;
                done = s_done;
                __syncthreads();  // read by all before either is written again
                if (tid == 0) s_n_deferred = 0;
                if (n_whole == 0) continue;
            }
            item = s_deferred[--n_whole];
        }
        whole(item);
        if (!heavy) __syncthreads();
    }
}

// ---- pipelined pair kernel ----
// The producer warps generate and sort the candidates of the next pair into one
// of kPipeBufs buffers while kPipeCons consumer warps, pair by pair in turn, run
// the greedy of earlier pairs, so the producers never wait at a barrier while a
// warp resolves.  (With one consumer warp and two buffers the greedy, 57
// thousand cycles a pair against 35 thousand, held the producers up.)  The hand-off
// is two mbarriers per buffer: `full` (every producer thread arrives after
// its writes) and `empty` (the consumer, after reading).  Every wait is
// bounded by %globaltimer (kPipeWaitNs); on expiry the waiting side sets
// kErrPipelineTimeout, raises the CTA's stop flag and leaves, and the other
// side leaves at its next (bounded) wait.  The producers of a CTA take every
// decision together (one thread decides, a producer barrier publishes it),
// so their named barrier is never left half-joined.
//
// Dense, overflow-heavy spectra (1000 to 2000 peaks, match_limit 1024), 800 x 907:
// 24.7 ms (39.4 with one consumer, 64-bit words and a chunk-by-chunk greedy).  A
// CTA's pair takes its producers 34 thousand cycles, 19 generating and 15 sorting,
// and its consumers 25; four CTAs a multiprocessor at 80 registers (six at 64 with
// one consumer and two buffers: the same time).  Bound by dependent integer
// instructions at 57% issue.
constexpr int kPipeBufs = 3;
constexpr int kPipeCons = 2;
constexpr int kGenCache = 2048; // query m/z values kept in shared memory while generating
// shared memory of np producer threads and buffers of cap candidates; the
// scratch serves gen_pair, then the sorts (a 64-bit word per candidate and one
// more per eight: 72 bytes a thread)
constexpr size_t pipe_scratch_bytes(int np) {
    return std::max<size_t>(gen_scratch_bytes(np, kGenCache), (size_t)np * 72);
}
constexpr size_t pipe_smem_bytes(int cap, int np) {
    return (size_t)cap * 12 * kPipeBufs + (size_t)kPipeCons * 2 * kUsedWords * 4 +
           pipe_scratch_bytes(np);
}
constexpr unsigned long long kPipeWaitNs = 2000000000ull;

__device__ __forceinline__ void pipe_bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(bar)),
                 "r"(count));
}
__device__ __forceinline__ void pipe_bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(bar))
                 : "memory");
}
// true once the phase of `parity` has completed; false after kPipeWaitNs or
// when *stop is raised
__device__ __forceinline__ bool pipe_bar_wait(uint64_t* bar, uint32_t parity,
                                              volatile int* stop) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
    const unsigned long long t0 = global_ns();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*stop) return false;
        if (global_ns() - t0 > kPipeWaitNs) return false;
    }
}

template <bool SPARSE, bool MODIFIED>
__global__ void __maxnreg__(80)
pair_kernel_pipe(PairParams P) {
    if (*P.bad) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned long long* okey0 = reinterpret_cast<unsigned long long*>(smem_raw);
    uint32_t* cgen0 = reinterpret_cast<uint32_t*>(okey0 + kPipeBufs * P.cap);
    uint32_t* used0 = cgen0 + kPipeBufs * P.cap;
    void* scratch = used0 + kPipeCons * 2 * kUsedWords;
    __shared__ int s_scan[32];
    __shared__ uint16_t s_queue[kPipeCons][kQueued];
    __shared__ int s_flags[kFixPasses + 1];
    __shared__ unsigned long long s_item;
    __shared__ __align__(8) uint64_t s_full[kPipeBufs], s_empty[kPipeBufs];
    __shared__ long long s_ri[kPipeBufs], s_qi[kPipeBufs];
    __shared__ int s_total[kPipeBufs];  // candidates generated; -1: no more pairs
    __shared__ int s_go;                // producers: 1 to continue
    __shared__ volatile int s_stop;

    const int tid = threadIdx.x;
    const int np = (int)blockDim.x - 32 * kPipeCons;  // producer threads
    const bool producer = tid < np;
    if (tid == 0) {
        for (int b = 0; b < kPipeBufs; ++b) {
            pipe_bar_init(&s_full[b], (uint32_t)np);
            pipe_bar_init(&s_empty[b], 1u);
        }
        s_stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int64_t n_items = P.R.n * P.Q.n;

    if (producer) {
        const GroupSync sync{np};
        const GenScratch gen = gen_scratch(scratch, np, kGenCache);
        int b = 0;
        uint32_t ph = 0;  // parity of buffer b's current use
        int ends = 0;     // end marks posted, one for each consumer
        for (int64_t iter = 0; ends < kPipeCons; ++iter) {
            if (tid == 0) s_item = (unsigned long long)(blockIdx.x + iter * gridDim.x);
            sync();
            const int64_t item = (int64_t)s_item;
            int64_t ri = 0, qi = 0;
            const bool more = item < n_items;
            if (more && !pair_of(P, item, ri, qi)) {
                sync();  // s_item is rewritten by the next fetch
                continue;
            }
            // buffer b free (its consumer is done with its previous pair)?
            if (tid == 0) s_go = pipe_bar_wait(&s_empty[b], ph ^ 1u, &s_stop) ? 1 : 0;
            sync();
            if (!s_go) {
                if (tid == 0 && !s_stop) {
                    atomicOr(P.err, kErrPipelineTimeout);
                    s_stop = 1;
                }
                break;
            }
            unsigned long long* okey = okey0 + (size_t)b * P.cap;
            uint32_t* cgen = cgen0 + (size_t)b * P.cap;
            int total = -1;
            if (more) {
                total = gen_pair<MODIFIED, true>(P, ri, qi, okey, cgen, P.match_limit, np, tid, s_scan, gen,
                                           sync);
                const int n = min(total, P.match_limit);
                if (n > 0) {
                    int m = 1;
                    while (m < n) m <<= 1;
                    // one word per candidate when the pair fills the register
                    // sort; the (key, gen) pairs themselves otherwise
                    if (!(m == 8 * np &&
                          (sort8_by_float(okey, cgen, scratch, s_flags, n, m, np, tid, sync) ||
                           sort8_by_word(okey, cgen, reinterpret_cast<unsigned long long*>(scratch),
                                         s_flags, n, m, np, tid, sync))))
                        sort_pair(okey, cgen, n, m, np, tid, sync);
                }
            } else {
                ++ends;
            }
            if (tid == 0) {
                s_ri[b] = ri;
                s_qi[b] = qi;
                s_total[b] = total;
            }
            sync();
            pipe_bar_arrive(&s_full[b]);
            if (++b == kPipeBufs) {
                b = 0;
                ph ^= 1u;
            }
        }
    } else if (!P.test_stall) {
        // consumer warp w: every kPipeCons-th buffer use, from use w on
        const int lane = tid & 31, w = (tid - np) >> 5;
        uint32_t* used_r = used0 + w * 2 * kUsedWords;
        for (int use = w;; use += kPipeCons) {
            const int b = use % kPipeBufs;
            const uint32_t ph = (uint32_t)(use / kPipeBufs) & 1u;
            int ok = 0;
            if (lane == 0) ok = pipe_bar_wait(&s_full[b], ph, &s_stop) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) {
                if (lane == 0 && !s_stop) {
                    atomicOr(P.err, kErrPipelineTimeout);
                    s_stop = 1;
                }
                break;
            }
            const int total = s_total[b];
            if (total < 0) break;  // no more pairs
            const int64_t ri = s_ri[b], qi = s_qi[b];
            const int n = min(total, P.match_limit);
            double score = 0.0;
            int matches = 0;
            if (n > 0) {
                const int nr = (int)(P.R.off[ri + 1] - P.R.off[ri]);
                const int nq = (int)(P.Q.off[qi + 1] - P.Q.off[qi]);
                const bool fits = max(nr, nq) <= 32 * kUsedWords;
                uint32_t* const bits_r =
                    fits ? used_r : P.long_bits + ((size_t)blockIdx.x * kPipeCons + w) * kLongWords;
                uint32_t* const bits_q = bits_r + (fits ? kUsedWords : kFullWords);
                for (int i = lane; i < (nr + 31) / 32; i += 32) bits_r[i] = 0u;
                for (int i = lane; i < (nq + 31) / 32; i += 32) bits_q[i] = 0u;
                __syncwarp();
                unsigned long long* okey = okey0 + (size_t)b * P.cap;
                const uint32_t* cgen = cgen0 + (size_t)b * P.cap;
                if (fits) {
                    greedy_pair<MODIFIED, false>(okey, cgen, used_r, used_r + kUsedWords,
                                                 s_queue[w], n, score, matches);
                } else {
                    const Greedy r = greedy_long<MODIFIED>(okey, cgen, bits_r, s_queue[w], n);
                    score = r.score;
                    matches = r.matches;
                }
            }
            __syncwarp();
            if (lane == 0) {
                pipe_bar_arrive(&s_empty[b]);
                write_pair<SPARSE>(P, ri, qi, n, score, matches, total >= P.match_limit);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
inline int next_pow2(long long x) {
    int p = 1;
    while (p < x && p < (1 << 30)) p <<= 1;
    return p;
}

struct Plan {
    int mode;
    int tile;
    int n_tiles;
    int nb;
    double width;
    int pair_threads;
    int cap;       // power of two >= match_limit
    int pair_cap;  // candidates of pair_kernel's buffer
    unsigned int spill_cap;
    int sym;               // cms_cosine_config.symmetric
    double cand_per_pair;  // cms_cosine_config.cand_per_pair (0: unknown)
    int width_by_class[kOrderClasses];  // cms_cosine_config.width_by_class
};

int make_plan(const CosineArgs& args, const cms_cosine_config* cfg, bool sparse, Plan& p) {
    p.mode = (cfg && cfg->mode) ? cfg->mode : 1;
    if (p.mode != 1 && p.mode != 2) {
        set_error("cms_cosine_greedy: mode must be 0, 1 or 2");
        return CMS_ERR_INVALID;
    }
    if (cfg && cfg->tile_spectra > 0) {
        p.tile = cfg->tile_spectra;
    } else {
        // about 176 expected candidates per work item (reference x tile) and at most
        // 1792 queries when the caller gives candidates per pair, which is what the
        // pool holds beside the heads of the tile (50000 x 50000 lognormal spectra:
        // 8.9 ms, 9.2 with tiles of 2048), else 1024 queries; at most one item per
        // 100000 pairs so that every resident warp gets tens of items
        const long long pairs = (long long)args.ref.n * (long long)args.qry.n;
        long long t = 1024;
        if (cfg && cfg->cand_per_pair > 0.0)
            t = (long long)std::min(1792.0, 176.0 / cfg->cand_per_pair);
        t = std::min(t, pairs / 100000);
        t = std::max<long long>(32, t);
        p.tile = (int)((t + 31) / 32 * 32);
    }
    if (p.tile > kMaxTile) {
        set_error("cms_cosine_greedy: tile_spectra must be <= %d", kMaxTile);
        return CMS_ERR_UNSUPPORTED;
    }
    p.tile = (int)std::min<int64_t>(p.tile, std::max<int64_t>(1, args.qry.n));
    p.n_tiles = (int)((args.qry.n + p.tile - 1) / p.tile);
    // bucket width: tol by default (a window spans two or three buckets);
    // any width is correct, narrower ones want more buckets per tile
    double w = (cfg && cfg->bucket_width > 0.0) ? cfg->bucket_width : args.tol;
    if (w < 0.25 * args.tol) w = 0.25 * args.tol;
    if (!(w > 0.0)) w = 1e-3;
    p.width = w;
    const double avg_tile_peaks =
        args.qry.n > 0 ? (double)args.qry.n_peaks * p.tile / (double)args.qry.n : 1.0;
    p.nb = (cfg && cfg->n_buckets > 0) ? next_pow2(cfg->n_buckets)
                                       : next_pow2((long long)std::max(1024.0, avg_tile_peaks));
    p.nb = std::min(p.nb, 1 << 22);
    p.cap = next_pow2(std::max(2, args.match_limit));
    // whole-matrix pair kernel (mode 2): pairs usually fill match_limit, and
    // eight candidates a thread sort in registers; spilled pairs vary in size
    p.pair_threads = (cfg && cfg->pair_threads > 0)
                         ? cfg->pair_threads
                         : (p.mode == 2 ? std::max(64, std::min(512, p.cap / 8)) : 128);
    if (p.pair_threads < 64 || p.pair_threads > 512 || p.pair_threads % 32) {
        set_error("cms_cosine_greedy: pair_threads must be a multiple of 32 in [64, 512]");
        return CMS_ERR_INVALID;
    }
    p.pair_cap = p.mode == 2 ? p.cap : list_cap(p.cap, p.pair_threads);
    const long long pairs = (long long)args.ref.n * (long long)args.qry.n;
    long long sc = std::max<long long>(1 << 20, pairs / 64);
    sc = std::min<long long>(sc, std::min<long long>(pairs, 1LL << 28));
    p.spill_cap = (unsigned int)std::max<long long>(sc, 1);
    for (int c = 0; c < kOrderClasses; ++c) {
        const int w = cfg ? cfg->width_by_class[c] : 0;
        if (w < 0) {
            set_error("cms_cosine_greedy: width_by_class entries must be >= 0");
            return CMS_ERR_INVALID;
        }
        p.width_by_class[c] = w;
    }
    (void)sparse;
    return CMS_OK;
}

template <typename T>
int set_func_smem(T* f, size_t bytes) {
    return raise_func_smem(reinterpret_cast<const void*>(f), bytes);
}

// Blocks for n spectra at `per` spectra a block, at most 32 a multiprocessor.
int blocks_for(int64_t n, int per, int sms) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + per - 1) / per, (int64_t)sms * 32));
}
constexpr int kPrepPerBlock = kPrepSpectra * (kPrepThreads / 32);
constexpr int kScatterThreads = 256;  // index scatter: a warp per spectrum

// Prepare one or two spectrum sets (the second may be empty) in one launch.
void launch_prep(const PrepSide& p0, const PrepSide& p1, const IndexGeom& g, uint32_t* bad,
                 uint32_t* err, int max_peaks, int sms, cudaStream_t s, uint32_t* any_long = nullptr) {
    const PrepSides sides{{p0, p1}, blocks_for(p0.S.n, kPrepPerBlock, sms), any_long};
    const int blocks1 = p1.S.n > 0 ? blocks_for(p1.S.n, kPrepPerBlock, sms) : 0;
    prep_kernel<<<sides.blocks0 + blocks1, kPrepThreads, 0, s>>>(sides, g, bad, err, max_peaks);
}
void launch_probe(const ProbeArgs& p, const IndexGeom& g, const uint32_t* bad, uint32_t* err, int sms,
                  cudaStream_t s) {
    probe_kernel<<<blocks_for(p.S.n_peaks, kProbeThreads, sms), kProbeThreads, 0, s>>>(p, g, bad, err);
}

// Launch the join.  Persistent (waves == 0): one resident CTA per slot, each
// warp pulling work until none is left; CTA b owns global-pool slices
// 8b..8b+7, so the grid may not exceed the resident CTAs.  Bounded
// (waves > 0): `waves` times the resident CTAs, each warp exiting after an
// equal share of items, so that the SMs free up CTA by CTA and concurrent
// launches on other streams are scheduled in between while every wave stays
// full; each CTA claims a global-pool slice from jp.slots (zeroed by the
// caller) for its lifetime.
template <bool A_IS_REF, bool SPARSE, bool MODIFIED>
int launch_join(cms_ctx* ctx, JoinParams jp, size_t smem, size_t gpool_warps, int64_t n_items,
                cudaStream_t s, int waves = 0) {
    auto* kern = join_kernel<A_IS_REF, SPARSE, MODIFIED>;
    if (const int rc = set_func_smem(kern, smem)) return rc;
    jp.trace = TraceOut{ctx->trace_rec, ctx->trace_count, ctx->trace_cap, ctx->trace_tag};
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kJoinThreads, smem);
    const int64_t resident = (int64_t)ctx->sm_count * std::max(1, per_sm);
    int64_t grid;
    if (waves > 0) {
        grid = std::min<int64_t>(resident * waves, (n_items + kJoinWarps - 1) / kJoinWarps);
        grid = std::max<int64_t>(1, grid);
        const int64_t per_warp = (n_items + grid * kJoinWarps - 1) / (grid * kJoinWarps);
        if (per_warp > INT32_MAX) {
            set_error("cms_cosine_greedy: too many work items for one launch");
            return CMS_ERR_UNSUPPORTED;
        }
        jp.max_fetch = (int)per_warp;
        if (!jp.slots) jp.gpool = nullptr;
        jp.n_slots = (int)std::min<int64_t>(resident, (int64_t)(gpool_warps / kJoinWarps));
        if (jp.n_slots <= 0) jp.gpool = nullptr;
        if (!jp.gpool) jp.pool_max = jp.pool_smem;
    } else {
        jp.max_fetch = 0;
        jp.slots = nullptr;
        grid = resident;
        if (jp.gpool && (size_t)grid * kJoinWarps > gpool_warps) {
            set_error("cms_cosine_greedy: join grid larger than its scratch");
            return CMS_ERR_CUDA;
        }
    }
    kern<<<(unsigned)grid, kJoinThreads, smem, s>>>(jp);
    CMS_CUDA_TRY(cudaGetLastError());
    return CMS_OK;
}

int enqueue_cosine(cms_ctx* ctx, const CosineArgs& args, const DenseOut* dense,
                   const SparseOut* sparse, const Plan& p, cudaStream_t s);
int run_cosine_graph(cms_ctx* ctx, const CosineArgs& args, const DenseOut* dense,
                     const SparseOut* sparse, const Plan& p, cudaStream_t s);

int run_cosine(cms_ctx* ctx, const CosineArgs& args, const DenseOut* dense,
               const SparseOut* sparse, const cms_cosine_config* cfg, cudaStream_t s) {
    Plan p;
    int rc = make_plan(args, cfg, sparse != nullptr, p);
    if (rc) return rc;
    const int sym = (cfg && cfg->symmetric) ? 1 : 0;
    p.sym = sym;
    p.cand_per_pair = (cfg && cfg->cand_per_pair > 0.0) ? cfg->cand_per_pair : 0.0;
    if (sym && args.ref.n != args.qry.n) {
        set_error("cms_cosine_greedy: symmetric needs as many queries as references "
                  "(%lld != %lld)", (long long)args.ref.n, (long long)args.qry.n);
        return CMS_ERR_INVALID;
    }
    const size_t pair_smem = pair_smem_bytes(p.cap, p.pair_threads, 0);
    if (pair_smem > ctx->smem_optin) {
        set_error("cms_cosine_greedy: match_limit %d needs %zu B shared memory (> %zu)",
                  args.match_limit, pair_smem, ctx->smem_optin);
        return CMS_ERR_UNSUPPORTED;
    }

    // ---- scratch layout ----
    const int64_t nR = args.ref.n, nQ = args.qry.n;
    // global pool extension for every warp the join grid can hold (at most
    // 64 warps per SM are resident)
    const size_t gpool_warps = (size_t)ctx->sm_count * 64;
    const size_t gpool_bytes = gpool_warps * (size_t)kGPool * 16;
    size_t need = 0;
    need += bump_size(64 * sizeof(uint64_t));            // flags, counters
    need += bump_size(nR * sizeof(double)) + bump_size(nQ * sizeof(double));
    if (p.mode == 1) {
        need += bump_size(nR * sizeof(SweepItem)) + bump_size(nQ * sizeof(double));
        need += bump_size((size_t)std::max<int64_t>(1, args.ref.n_peaks) * sizeof(Probe));
        if (args.modified)
            need += bump_size((size_t)std::max<int64_t>(1, args.ref.n_peaks) * sizeof(uint2));
        if (args.ref.a)
            need += bump_size((size_t)std::max<int64_t>(1, args.ref.n_peaks) * sizeof(double));
        const size_t idx = args.modified ? 2 : 1;  // m/z index, neutral-loss index
        need += bump_size(idx * (size_t)p.n_tiles * p.nb * sizeof(uint32_t));
        need += bump_size((size_t)p.n_tiles * scan_chunks(p.nb) * sizeof(uint32_t));
        need += idx * bump_size((size_t)p.n_tiles * (p.nb + 1) * sizeof(uint32_t));
        need += idx * bump_size((size_t)std::max<int64_t>(1, args.qry.n_peaks) * sizeof(Entry));
        if (args.qry.a)
            need += idx * bump_size((size_t)std::max<int64_t>(1, args.qry.n_peaks) * sizeof(double));
        need += bump_size((size_t)p.spill_cap * sizeof(int2));
        need += bump_size(gpool_bytes);
    }
    if (may_be_long(args.ref) || may_be_long(args.qry))
        need += bump_size(long_bits_bytes(ctx->sm_count));
    need += 4096;
    rc = arena_reserve(ctx, ctx->scratch, need, s);
    if (rc) return rc;
    if (!ctx->graphs) return enqueue_cosine(ctx, args, dense, sparse, p, s);
    return run_cosine_graph(ctx, args, dense, sparse, p, s);
}

// The launch sequence of one call, into scratch already reserved for plan p
// (no allocation or synchronisation inside, so that it can be captured).
int enqueue_cosine(cms_ctx* ctx, const CosineArgs& args, const DenseOut* dense,
                   const SparseOut* sparse, const Plan& p, cudaStream_t s) {
    int rc = CMS_OK;
    const int sym = p.sym;
    const int cache = pair_cache(p.pair_cap, p.pair_threads, ctx->smem_optin);
    const size_t pair_smem = pair_smem_bytes(p.pair_cap, p.pair_threads, cache);
    const int64_t nR = args.ref.n, nQ = args.qry.n;
    const size_t gpool_warps = (size_t)ctx->sm_count * 64;
    const size_t gpool_bytes = gpool_warps * (size_t)kGPool * 16;
    Bump bp{(char*)ctx->scratch.ptr, 0, ctx->scratch.bytes};
    uint64_t* small = bp.take<uint64_t>(64);
    uint32_t* bad = reinterpret_cast<uint32_t*>(small);            // word 0
    uint32_t* cls_count = reinterpret_cast<uint32_t*>(small + 1);  // 17 words
    uint32_t* cls_cursor = reinterpret_cast<uint32_t*>(small + 10);  // 17 words
    unsigned long long* spill_count = reinterpret_cast<unsigned long long*>(small + 20);
    unsigned long long* work_join = reinterpret_cast<unsigned long long*>(small + 21);
    unsigned long long* work_pair = reinterpret_cast<unsigned long long*>(small + 22);
    // the bucket counts lie behind the counters: one memset clears both
    const size_t idx = p.mode != 1 ? 0 : (args.modified ? 2 : 1);
    const size_t n_cnt = (size_t)p.n_tiles * p.nb;
    const int n_chunks = p.n_tiles * scan_chunks(p.nb);
    uint32_t* cur = idx ? bp.take<uint32_t>(idx * n_cnt) : nullptr;
    const size_t zeroed = bp.used - (size_t)((char*)small - (char*)ctx->scratch.ptr);
    uint32_t* cur2 = idx == 2 ? cur + n_cnt : nullptr;
    uint32_t* sums = idx ? bp.take<uint32_t>(n_chunks) : nullptr;
    double* rnQ = idx ? bp.take<double>(nQ) : nullptr;
    const size_t ref_peaks = (size_t)std::max<int64_t>(1, args.ref.n_peaks);
    Probe* probe = idx ? bp.take<Probe>(ref_peaks) : nullptr;
    double* wR = idx && args.ref.a ? bp.take<double>(ref_peaks) : nullptr;
    uint2* probe2 = idx == 2 ? bp.take<uint2>(ref_peaks) : nullptr;
    double* snR = bp.take<double>(nR);
    double* snQ = bp.take<double>(nQ);
    uint32_t* long_bits = may_be_long(args.ref) || may_be_long(args.qry)
                              ? bp.take<uint32_t>(long_bits_bytes(ctx->sm_count) / 4)
                              : nullptr;
    CMS_CUDA_TRY(cudaMemsetAsync(small, 0, zeroed, s));

    const IndexGeom g{p.tile, p.n_tiles, p.nb, 1.0 / p.width};
    const int sms = ctx->sm_count;
    {
        StageScope sc(ctx, 0, idx ? 2 : 1, s);
        const int max_peaks = args.modified ? kModifiedMaxPeaks : CMS_MAX_PEAKS;
        launch_prep(PrepSide{args.ref, snR, nullptr, idx ? cls_count : nullptr, nullptr, nullptr, wR},
                    PrepSide{args.qry, snQ, rnQ, nullptr, cur, cur2}, g, bad, ctx->err_word,
                    max_peaks, sms, s);
        if (idx)
            launch_probe(ProbeArgs{args.ref, probe, probe2, args.tol, args.shift, 1}, g, bad,
                         ctx->err_word, sms, s);
    }
    CMS_CUDA_TRY(cudaGetLastError());

    if (sparse) CMS_CUDA_TRY(cudaMemsetAsync(sparse->count, 0, sizeof(unsigned long long), s));

    PairParams pp{};
    pp.R = args.ref;
    pp.Q = args.qry;
    pp.snR = snR;
    pp.snQ = snQ;
    pp.tol = args.tol;
    pp.shift = args.shift;
    pp.match_limit = args.match_limit;
    pp.cap = p.pair_cap;
    pp.cache = cache;
    pp.used_words = kUsedWords;
    pp.long_bits = long_bits;
    pp.pairs = nullptr;
    pp.n_pairs = nullptr;
    pp.pairs_cap = 0;
    pp.work = work_pair;
    pp.dense = dense ? *dense : DenseOut{nullptr, nullptr, nullptr, 0};
    pp.sparse = sparse ? *sparse : SparseOut{};
    pp.sparse.mirror = sym;
    pp.err = ctx->err_word;
    pp.bad = bad;
    pp.sym = sym;
    // dense symmetric output: the lower triangle is copied from the upper
    // one once every pair kernel has written it
    auto mirror = [&]() -> int {
        if (!sym || sparse) return CMS_OK;
        return launch_mirror(pp.dense, nR, bad, ctx->sm_count, s);
    };

    void (*pair_k)(PairParams) =
        p.mode == 2
            ? (sparse ? (args.modified ? pair_kernel<true, true, false> : pair_kernel<true, false, false>)
                      : (args.modified ? pair_kernel<false, true, false>
                                       : pair_kernel<false, false, false>))
            : (sparse ? (args.modified ? pair_kernel<true, true, true> : pair_kernel<true, false, true>)
                      : (args.modified ? pair_kernel<false, true, true>
                                       : pair_kernel<false, false, true>));
    int pair_blocks_per_sm = 1;
    if ((rc = set_func_smem(pair_k, pair_smem))) return rc;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pair_blocks_per_sm, pair_k, p.pair_threads,
                                                  pair_smem);
    pair_blocks_per_sm = std::max(1, pair_blocks_per_sm);
    const int pair_grid = ctx->sm_count * std::min(kLongWarps, pair_blocks_per_sm);

    const size_t pipe_smem = pipe_smem_bytes(p.cap, p.pair_threads);
    if (p.mode == 2 && pipe_smem <= ctx->smem_optin) {
        // whole matrix: the pipelined pair kernel (pair_threads producers
        // plus the consumer warps)
        void (*pipe_k)(PairParams) =
            sparse ? (args.modified ? pair_kernel_pipe<true, true> : pair_kernel_pipe<true, false>)
                   : (args.modified ? pair_kernel_pipe<false, true>
                                    : pair_kernel_pipe<false, false>);
        const int pipe_threads = p.pair_threads + 32 * kPipeCons;
        pp.test_stall = test_stall("pair");
        if ((rc = set_func_smem(pipe_k, pipe_smem))) return rc;
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pipe_k, pipe_threads, pipe_smem);
        StageScope sc(ctx, 4, 1, s);
        per_sm = std::max(1, std::min(kLongWarps / kPipeCons, per_sm));
        pipe_k<<<ctx->sm_count * per_sm, pipe_threads, pipe_smem, s>>>(pp);
        CMS_CUDA_TRY(cudaGetLastError());
        return mirror();
    }
    if (p.mode == 2) {  // one candidate buffer only fits
        StageScope sc(ctx, 4, 1, s);
        pair_k<<<pair_grid, p.pair_threads, pair_smem, s>>>(pp);
        CMS_CUDA_TRY(cudaGetLastError());
        return mirror();
    }

    // ---- mode 1: order, index, join, spill ----
    SweepItem* items = bp.take<SweepItem>(nR);
    const size_t q_peaks = (size_t)std::max<int64_t>(1, args.qry.n_peaks);
    uint32_t* tab = bp.take<uint32_t>((size_t)p.n_tiles * (p.nb + 1));
    Entry* ent = bp.take<Entry>(q_peaks);
    double* ent_a = args.qry.a ? bp.take<double>(q_peaks) : nullptr;
    uint32_t* tab2 = nullptr;
    Entry* ent2 = nullptr;
    double* ent2_a = nullptr;
    if (args.modified) {
        tab2 = bp.take<uint32_t>((size_t)p.n_tiles * (p.nb + 1));
        ent2 = bp.take<Entry>(q_peaks);
        if (args.qry.a) ent2_a = bp.take<double>(q_peaks);
    }
    int2* spill = bp.take<int2>(p.spill_cap);
    unsigned char* gpool = bp.take<unsigned char>(gpool_bytes);

    {
        StageScope sc(ctx, 1, 1, s);
        order_scatter_kernel<<<blocks_for(nR, kOrderThreads, sms), kOrderThreads, 0, s>>>(
            args.ref, snR, cls_count, cls_cursor, items, bad);
    }
    const int scatter_blocks = blocks_for(nQ, kScatterThreads / 32, sms);
    {
        StageScope sc(ctx, 2, 3, s);
        index_sums_kernel<<<n_chunks, kScanThreads, 0, s>>>(g, cur, sums, bad);
        index_scan_kernel<<<n_chunks, kScanThreads, 0, s>>>(g, cur, tab, sums, bad);
        index_scatter_kernel<false><<<scatter_blocks, kScatterThreads, 0, s>>>(args.qry, g, cur, ent,
                                                                               ent_a, bad);
    }
    if (args.modified) {  // neutral-loss index: m/z - precursor, same geometry
        StageScope sc(ctx, 2, 3, s);
        index_sums_kernel<<<n_chunks, kScanThreads, 0, s>>>(g, cur2, sums, bad);
        index_scan_kernel<<<n_chunks, kScanThreads, 0, s>>>(g, cur2, tab2, sums, bad);
        index_scatter_kernel<true><<<scatter_blocks, kScatterThreads, 0, s>>>(
            args.qry, g, cur2, ent2, ent2_a, bad);
    }
    CMS_CUDA_TRY(cudaGetLastError());

    JoinParams jp{};
    jp.A = args.ref;
    jp.B = args.qry;
    jp.items = items;
    jp.probe = probe;
    jp.probe2 = probe2;
    jp.w = wR ? wR : args.ref.b;
    jp.snA = snR;
    jp.snB = snQ;
    jp.rnB = rnQ;
    jp.cls_count = cls_count;
    jp.tab = tab;
    jp.ent = ent;
    jp.ent_a = ent_a;
    jp.tab2 = tab2;
    jp.ent2 = ent2;
    jp.ent2_a = ent2_a;
    jp.g = g;
    jp.tol = args.tol;
    jp.match_limit = args.match_limit;
    jp.init_width_scale = 0.f;
    for (int c = 0; c < kOrderClasses; ++c) jp.width_by_class[c] = p.width_by_class[c];
    if (p.cand_per_pair > 0.0 && args.ref.n > 0) {
        // expected candidates of (A spectrum with n peaks, w queries) ~ n*w*lambda
        const double mean_na = (double)args.ref.n_peaks / (double)args.ref.n;
        const double lambda = p.cand_per_pair / std::max(1.0, mean_na);
        jp.init_width_scale = (float)(0.5 * kPoolMax / lambda);
    }
    jp.warp_smem_bytes = warp_slice_bytes(p.tile);
    jp.pool_smem = join_pool(p.tile);
    jp.pool_max = kPoolMax;
    jp.max_fetch = 0;
    jp.gpool = gpool;
    jp.work = work_join;
    jp.spill = SpillList{spill, spill_count, p.spill_cap};
    jp.dense = pp.dense;
    jp.vec_rows = (((uintptr_t)pp.dense.score | (uintptr_t)pp.dense.matches) & 15) == 0 &&
                  ((uintptr_t)pp.dense.overflow & 3) == 0;
    jp.sparse = pp.sparse;
    jp.err = ctx->err_word;
    jp.bad = bad;
    jp.sym = sym;
    const size_t join_smem = (size_t)warp_slice_bytes(p.tile) * kJoinWarps;
    {
        StageScope sc(ctx, 3, 1, s);
        const int64_t n = nR * (int64_t)p.n_tiles;
        if (args.modified)
            rc = sparse ? launch_join<true, true, true>(ctx, jp, join_smem, gpool_warps, n, s)
                        : launch_join<true, false, true>(ctx, jp, join_smem, gpool_warps, n, s);
        else
            rc = sparse ? launch_join<true, true, false>(ctx, jp, join_smem, gpool_warps, n, s)
                        : launch_join<true, false, false>(ctx, jp, join_smem, gpool_warps, n, s);
        if (rc) return rc;
    }
    CMS_CUDA_TRY(cudaGetLastError());

    pp.pairs = spill;
    pp.n_pairs = spill_count;
    pp.pairs_cap = p.spill_cap;
    {
        StageScope sc(ctx, 4, 1, s);
        pair_k<<<pair_grid, p.pair_threads, pair_smem, s>>>(pp);
        CMS_CUDA_TRY(cudaGetLastError());
    }
    return mirror();
}

// Graph path of run_cosine: replay a captured launch sequence whose key (every
// value the sequence bakes in) equals this call's, else capture it on the
// context's capture stream, instantiate and keep it (most recent first, at
// most kGraphCache per context); graphs are launched on the caller's stream.
constexpr size_t kGraphCache = 8;
int run_cosine_graph(cms_ctx* ctx, const CosineArgs& args, const DenseOut* dense,
                     const SparseOut* sparse, const Plan& p, cudaStream_t s) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    CMS_CUDA_TRY(cudaStreamIsCapturing(s, &cs));
    if (cs != cudaStreamCaptureStatusNone)  // the caller is capturing: just enqueue
        return enqueue_cosine(ctx, args, dense, sparse, p, s);
    std::vector<uint64_t> key;
    key.reserve(48);
    auto put = [&](auto v) {
        static_assert(sizeof(v) <= sizeof(uint64_t), "key field too wide");
        uint64_t u = 0;
        std::memcpy(&u, &v, sizeof(v));
        key.push_back(u);
    };
    auto put_set = [&](const SpecSet& x) {
        put((uintptr_t)x.mz);
        put((uintptr_t)x.a);
        put((uintptr_t)x.b);
        put((uintptr_t)x.off);
        put(x.n);
        put(x.n_peaks);
    };
    put_set(args.ref);
    put_set(args.qry);
    put(args.tol);
    put(args.shift);
    put(args.match_limit);
    put((int)args.modified);
    put((uintptr_t)args.ref.prec);
    put((uintptr_t)args.qry.prec);
    put((int)(dense != nullptr));
    if (dense) {
        put((uintptr_t)dense->score);
        put((uintptr_t)dense->matches);
        put((uintptr_t)dense->overflow);
        put(dense->ld);
    }
    put((int)(sparse != nullptr));
    if (sparse) {
        put((uintptr_t)sparse->r);
        put((uintptr_t)sparse->q);
        put((uintptr_t)sparse->score);
        put((uintptr_t)sparse->matches);
        put((uintptr_t)sparse->overflow);
        put((uintptr_t)sparse->count);
        put(sparse->capacity);
        put(sparse->threshold);
        put(sparse->mirror);
    }
    put(p.mode);
    put(p.tile);
    put(p.nb);
    put(p.width);
    put(p.pair_threads);
    put(p.cap);
    put(p.spill_cap);
    put(p.sym);
    put(p.cand_per_pair);
    for (int c = 0; c < kOrderClasses; ++c) put(p.width_by_class[c]);
    put((uintptr_t)ctx->scratch.ptr);
    put(ctx->scratch.bytes);
    put((uintptr_t)ctx->trace_rec);
    put((uintptr_t)ctx->trace_count);
    put(ctx->trace_cap);
    put(ctx->trace_tag);

    auto& cache = ctx->graph_cache;
    for (size_t i = 0; i < cache.size(); ++i) {
        if (cache[i].key != key) continue;
        if (i) std::rotate(cache.begin(), cache.begin() + i, cache.begin() + i + 1);
        for (int k = 0; k < CMS_PROFILE_STAGES; ++k) ctx->launches[k] += cache[0].launches[k];
        CMS_CUDA_TRY(cudaGraphLaunch(cache[0].exec, s));
        return CMS_OK;
    }

    if (!ctx->capture_stream)
        CMS_CUDA_TRY(cudaStreamCreateWithFlags(&ctx->capture_stream, cudaStreamNonBlocking));
    cudaStream_t cs_stream = ctx->capture_stream;
    int64_t before[CMS_PROFILE_STAGES];
    std::memcpy(before, ctx->launches, sizeof(before));
    CMS_CUDA_TRY(cudaStreamBeginCapture(cs_stream, cudaStreamCaptureModeRelaxed));
    ctx->capturing = true;
    const int rc = enqueue_cosine(ctx, args, dense, sparse, p, cs_stream);
    ctx->capturing = false;
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(cs_stream, &g);
    if (rc != CMS_OK || e != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        (void)cudaGetLastError();
        if (rc != CMS_OK) return rc;
        return cuda_fail(e, "cudaStreamEndCapture");
    }
    cms_graph_entry entry;
    entry.key = std::move(key);
    const cudaError_t ei = cudaGraphInstantiate(&entry.exec, g, 0);
    cudaGraphDestroy(g);
    if (ei != cudaSuccess) return cuda_fail(ei, "cudaGraphInstantiate");
    for (int k = 0; k < CMS_PROFILE_STAGES; ++k) entry.launches[k] = ctx->launches[k] - before[k];
    if (cache.size() >= kGraphCache) {
        cudaGraphExecDestroy(cache.back().exec);
        cache.pop_back();
    }
    cache.insert(cache.begin(), std::move(entry));
    CMS_CUDA_TRY(cudaGraphLaunch(cache[0].exec, s));
    return CMS_OK;
}

bool check_common(const CosineArgs& a, const char* who) {
    if (!check_specset(a.ref, "reference") || !check_specset(a.qry, "query")) return false;
    if (a.match_limit < 1 || !(a.tol >= 0.0) || !std::isfinite(a.tol) || !std::isfinite(a.shift)) {
        set_error("%s: invalid match_limit or tolerance/shift", who);
        return false;
    }
    return true;
}

}  // namespace
}  // namespace cms

extern "C" int cms_cosine_greedy(cms_ctx* ctx, const float* ref_mz, const double* ref_a,
                                 const double* ref_b, const int64_t* ref_off, int64_t n_ref,
                                 int64_t n_ref_peaks, const float* q_mz, const double* q_a,
                                 const double* q_b, const int64_t* q_off, int64_t n_q,
                                 int64_t n_q_peaks, double tolerance, double shift,
                                 int match_limit, float* score, int32_t* matches,
                                 uint8_t* overflow, int64_t ld, const cms_cosine_config* cfg,
                                 void* stream) {
    using namespace cms;
    if (!ctx) {
        set_error("cms_cosine_greedy: null context");
        return CMS_ERR_INVALID;
    }
    CosineArgs args{SpecSet{ref_mz, ref_a, ref_b, ref_off, n_ref, n_ref_peaks},
                    SpecSet{q_mz, q_a, q_b, q_off, n_q, n_q_peaks}, tolerance, shift,
                    match_limit};
    if (!check_common(args, "cms_cosine_greedy")) return CMS_ERR_INVALID;
    if (ld < n_q) {
        set_error("cms_cosine_greedy: ld < n_q");
        return CMS_ERR_INVALID;
    }
    if (n_ref == 0 || n_q == 0) return CMS_OK;
    if (!score || !matches || !overflow) {
        set_error("cms_cosine_greedy: null output pointer");
        return CMS_ERR_INVALID;
    }
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    DenseOut out{score, matches, overflow, ld};
    return run_cosine(ctx, args, &out, nullptr, cfg, (cudaStream_t)stream);
}

extern "C" int cms_cosine_greedy_sparse(cms_ctx* ctx, const float* ref_mz, const double* ref_a,
                                        const double* ref_b, const int64_t* ref_off, int64_t n_ref,
                                        int64_t n_ref_peaks, const float* q_mz,
                                        const double* q_a, const double* q_b,
                                        const int64_t* q_off, int64_t n_q, int64_t n_q_peaks,
                                        double tolerance, double shift, int match_limit,
                                        float threshold, int32_t* hit_ref, int32_t* hit_query,
                                        float* hit_score, int32_t* hit_matches,
                                        uint8_t* hit_overflow, int64_t capacity,
                                        int64_t* hit_count, const cms_cosine_config* cfg,
                                        void* stream) {
    using namespace cms;
    if (!ctx) {
        set_error("cms_cosine_greedy_sparse: null context");
        return CMS_ERR_INVALID;
    }
    CosineArgs args{SpecSet{ref_mz, ref_a, ref_b, ref_off, n_ref, n_ref_peaks},
                    SpecSet{q_mz, q_a, q_b, q_off, n_q, n_q_peaks}, tolerance, shift,
                    match_limit};
    if (!check_common(args, "cms_cosine_greedy_sparse")) return CMS_ERR_INVALID;
    if (!(threshold > 0.0f)) {
        set_error("cms_cosine_greedy_sparse: threshold must be > 0 (every pair scores >= 0)");
        return CMS_ERR_INVALID;
    }
    if (capacity < 0 || !hit_count || (capacity > 0 && (!hit_ref || !hit_query || !hit_score ||
                                                        !hit_matches || !hit_overflow))) {
        set_error("cms_cosine_greedy_sparse: invalid hit buffers");
        return CMS_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    if (n_ref == 0 || n_q == 0) {
        CMS_CUDA_TRY(cudaMemsetAsync(hit_count, 0, sizeof(int64_t), s));
        return CMS_OK;
    }
    SparseOut out{hit_ref, hit_query, hit_score, hit_matches, hit_overflow, capacity,
                  reinterpret_cast<unsigned long long*>(hit_count), threshold};
    return run_cosine(ctx, args, nullptr, &out, cfg, s);
}

extern "C" int cms_modified_cosine(cms_ctx* ctx, const float* ref_mz, const double* ref_a,
                                   const double* ref_b, const int64_t* ref_off,
                                   const double* ref_precursor, int64_t n_ref, int64_t n_ref_peaks,
                                   const float* q_mz, const double* q_a, const double* q_b,
                                   const int64_t* q_off, const double* q_precursor, int64_t n_q,
                                   int64_t n_q_peaks, double tolerance, int match_limit,
                                   float* score, int32_t* matches, uint8_t* overflow, int64_t ld,
                                   const cms_cosine_config* cfg, void* stream) {
    using namespace cms;
    if (!ctx) {
        set_error("cms_modified_cosine: null context");
        return CMS_ERR_INVALID;
    }
    CosineArgs args{SpecSet{ref_mz, ref_a, ref_b, ref_off, n_ref, n_ref_peaks, ref_precursor},
                    SpecSet{q_mz, q_a, q_b, q_off, n_q, n_q_peaks, q_precursor}, tolerance, 0.0,
                    match_limit, true};
    if (!check_common(args, "cms_modified_cosine")) return CMS_ERR_INVALID;
    if (ld < n_q) {
        set_error("cms_modified_cosine: ld < n_q");
        return CMS_ERR_INVALID;
    }
    if (n_ref == 0 || n_q == 0) return CMS_OK;
    if (!score || !matches || !overflow || !ref_precursor || !q_precursor) {
        set_error("cms_modified_cosine: null output or precursor pointer");
        return CMS_ERR_INVALID;
    }
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    DenseOut out{score, matches, overflow, ld};
    return run_cosine(ctx, args, &out, nullptr, cfg, (cudaStream_t)stream);
}

extern "C" int cms_modified_cosine_sparse(
    cms_ctx* ctx, const float* ref_mz, const double* ref_a, const double* ref_b,
    const int64_t* ref_off, const double* ref_precursor, int64_t n_ref, int64_t n_ref_peaks,
    const float* q_mz, const double* q_a, const double* q_b, const int64_t* q_off,
    const double* q_precursor, int64_t n_q, int64_t n_q_peaks, double tolerance, int match_limit,
    float threshold, int32_t* hit_ref, int32_t* hit_query, float* hit_score, int32_t* hit_matches,
    uint8_t* hit_overflow, int64_t capacity, int64_t* hit_count, const cms_cosine_config* cfg,
    void* stream) {
    using namespace cms;
    if (!ctx) {
        set_error("cms_modified_cosine_sparse: null context");
        return CMS_ERR_INVALID;
    }
    CosineArgs args{SpecSet{ref_mz, ref_a, ref_b, ref_off, n_ref, n_ref_peaks, ref_precursor},
                    SpecSet{q_mz, q_a, q_b, q_off, n_q, n_q_peaks, q_precursor}, tolerance, 0.0,
                    match_limit, true};
    if (!check_common(args, "cms_modified_cosine_sparse")) return CMS_ERR_INVALID;
    if (!(threshold > 0.0f)) {
        set_error("cms_modified_cosine_sparse: threshold must be > 0 (every pair scores >= 0)");
        return CMS_ERR_INVALID;
    }
    if (capacity < 0 || !hit_count || (capacity > 0 && (!hit_ref || !hit_query || !hit_score ||
                                                        !hit_matches || !hit_overflow))) {
        set_error("cms_modified_cosine_sparse: invalid hit buffers");
        return CMS_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    if (n_ref == 0 || n_q == 0) {
        CMS_CUDA_TRY(cudaMemsetAsync(hit_count, 0, sizeof(int64_t), s));
        return CMS_OK;
    }
    if (!ref_precursor || !q_precursor) {
        set_error("cms_modified_cosine_sparse: null precursor pointer");
        return CMS_ERR_INVALID;
    }
    SparseOut out{hit_ref, hit_query, hit_score, hit_matches, hit_overflow, capacity,
                  reinterpret_cast<unsigned long long*>(hit_count), threshold};
    return run_cosine(ctx, args, nullptr, &out, cfg, s);
}

// ---------------------------------------------------------------------------
// Allocation-free variant (cms_cosine_greedy_noalloc)
//
// Some callers cannot let a library call cudaMalloc: an application whose
// device memory is already reserved by its own allocator (a framework's
// caching pool that owns almost all of the GPU), a latency-critical loop that
// cannot afford the device-wide synchronisation cudaMalloc/cudaFree may
// imply, or a plugin host that forbids libraries to allocate behind its back.
// For them this entry point runs the dense greedy cosine with the pair kernel
// over every pair, and keeps its only scratch -- validity flags and the two
// per-spectrum norm arrays -- in the fixed device array below instead of a
// context's arena.  The array is part of the library's device image: every
// GPU that loads the library holds it until the process exits.
// ---------------------------------------------------------------------------
namespace cms {
namespace {

constexpr int64_t kNoAllocMaxSpectra = int64_t(1) << 20;  // n_ref + n_q
constexpr size_t kNoAllocHeader = 256;                     // flags and error word
constexpr size_t kNoAllocBytes = kNoAllocHeader + 8 * (size_t)kNoAllocMaxSpectra + 256;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device.  In host code the
// array's name is only a host-side stand-in, so the address is looked up once
// per device, with that device current, and cached.
int noalloc_scratch(unsigned char** out) {
    int dev = 0;
    CMS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("cms_cosine_greedy_noalloc: device ordinal %d out of range", dev);
        return CMS_ERR_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return CMS_OK;
}

}  // namespace
}  // namespace cms

extern "C" int cms_cosine_greedy_noalloc(const float* ref_mz, const double* ref_a,
                                         const double* ref_b, const int64_t* ref_off,
                                         int64_t n_ref, int64_t n_ref_peaks, const float* q_mz,
                                         const double* q_a, const double* q_b,
                                         const int64_t* q_off, int64_t n_q, int64_t n_q_peaks,
                                         double tolerance, double shift, int match_limit,
                                         float* score, int32_t* matches, uint8_t* overflow,
                                         int64_t ld, uint32_t* device_error, void* stream) {
    using namespace cms;
    CosineArgs args{SpecSet{ref_mz, ref_a, ref_b, ref_off, n_ref, n_ref_peaks},
                    SpecSet{q_mz, q_a, q_b, q_off, n_q, n_q_peaks}, tolerance, shift,
                    match_limit};
    if (!check_common(args, "cms_cosine_greedy_noalloc")) return CMS_ERR_INVALID;
    if (ld < n_q) {
        set_error("cms_cosine_greedy_noalloc: ld < n_q");
        return CMS_ERR_INVALID;
    }
    if (n_ref + n_q > kNoAllocMaxSpectra) {
        set_error("cms_cosine_greedy_noalloc: n_ref + n_q = %lld exceeds the fixed scratch "
                  "capacity of %lld spectra; split the call or use cms_cosine_greedy",
                  (long long)(n_ref + n_q), (long long)kNoAllocMaxSpectra);
        return CMS_ERR_UNSUPPORTED;
    }
    if (match_limit > 4096) {
        set_error("cms_cosine_greedy_noalloc: match_limit must be <= 4096");
        return CMS_ERR_UNSUPPORTED;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (n_ref == 0 || n_q == 0) {
        if (device_error) CMS_CUDA_TRY(cudaMemsetAsync(device_error, 0, sizeof(uint32_t), s));
        return CMS_OK;
    }
    if (!score || !matches || !overflow) {
        set_error("cms_cosine_greedy_noalloc: null output pointer");
        return CMS_ERR_INVALID;
    }
    // Every buffer must be memory of the current device: the scratch address
    // below is the current device's, and a kernel handed another GPU's (or
    // host) memory would read or write out of bounds.  Nothing is launched
    // before these checks.
    const char* who = "cms_cosine_greedy_noalloc";
    const std::pair<const void*, const char*> bufs[] = {
        {ref_mz, "ref_mz"}, {ref_a, "ref_a"}, {ref_b, "ref_b"}, {ref_off, "ref_off"},
        {q_mz, "q_mz"},     {q_a, "q_a"},     {q_b, "q_b"},     {q_off, "q_off"},
        {score, "score"},   {matches, "matches"}, {overflow, "overflow"},
        {device_error, "device_error"}};
    int rc = CMS_OK;
    for (const auto& bf : bufs)
        if (bf.first && (rc = check_device_ptr(bf.first, who, bf.second))) return rc;
    if (s) {
        int sdev = -1, dev = 0;
        CMS_CUDA_TRY(cudaStreamGetDevice(s, &sdev));
        CMS_CUDA_TRY(cudaGetDevice(&dev));
        if (sdev != dev) {
            set_error("%s: stream belongs to device %d, not the current device %d", who, sdev,
                      dev);
            return CMS_ERR_INVALID;
        }
    }
    unsigned char* base = nullptr;
    rc = noalloc_scratch(&base);
    if (rc) return rc;
    uint32_t* bad = reinterpret_cast<uint32_t*>(base);
    uint32_t* err = reinterpret_cast<uint32_t*>(base + 4);
    uint32_t* any_long = reinterpret_cast<uint32_t*>(base + 32);
    double* snR = reinterpret_cast<double*>(base + kNoAllocHeader);
    double* snQ = snR + n_ref;
    // the array keeps the previous call's contents: reset the flags
    CMS_CUDA_TRY(cudaMemsetAsync(base, 0, kNoAllocHeader, s));

    int dev = 0, sms = 0;
    CMS_CUDA_TRY(cudaGetDevice(&dev));
    CMS_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const IndexGeom none{1, 1, 1, 1.0};
    launch_prep(PrepSide{args.ref, snR}, PrepSide{args.qry, snQ}, none, bad, err, CMS_MAX_PEAKS, sms,
                s, any_long);
    CMS_CUDA_TRY(cudaGetLastError());

    PairParams pp{};
    pp.R = args.ref;
    pp.Q = args.qry;
    pp.snR = snR;
    pp.snQ = snQ;
    pp.tol = tolerance;
    pp.shift = shift;
    pp.match_limit = match_limit;
    int cap = 2;
    while (cap < match_limit) cap <<= 1;
    pp.cap = cap;
    pp.pairs = nullptr;  // every pair of R x Q, statically strided
    pp.n_pairs = nullptr;
    pp.pairs_cap = 0;
    pp.work = reinterpret_cast<unsigned long long*>(base + 8);
    pp.gate = any_long;
    pp.dense = DenseOut{score, matches, overflow, ld};
    pp.sparse = SparseOut{};
    pp.err = err;
    pp.bad = bad;
    const int pair_threads = 128;
    // Without scratch for the bitmaps of long spectra, a call that has any (known on
    // the device only) keeps all of them in shared memory: one of two launches
    // runs, the other returns at once.
    for (uint32_t full = 0; full < (may_be_long(args.ref) || may_be_long(args.qry) ? 2u : 1u); ++full) {
        pp.gate_value = full;
        pp.used_words = full ? kFullWords : kUsedWords;
        pp.cache = cap <= 2048 ? kPairCache : 0;  // with 4096 it would cost a resident CTA
        const size_t pair_smem = pair_smem_bytes(cap, pair_threads, pp.cache, pp.used_words);
        if ((rc = set_func_smem(pair_kernel<false, false, false>, pair_smem))) return rc;
        int per_sm = 1;
        CMS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, pair_kernel<false, false, false>, pair_threads, pair_smem));
        pair_kernel<false, false, false><<<sms * std::max(1, per_sm), pair_threads, pair_smem, s>>>(pp);
        CMS_CUDA_TRY(cudaGetLastError());
    }
    if (device_error)
        CMS_CUDA_TRY(cudaMemcpyAsync(device_error, err, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    return CMS_OK;
}


// ---------------------------------------------------------------------------
// Resident library (cms_library_*): the indexed side built once, searched by
// many query batches.
// ---------------------------------------------------------------------------
struct cms_library {
    int device = 0;
    cms::SpecSet spec{};  // caller-owned device arrays; must outlive the library
    double tol = 0.0, shift = 0.0, cand_per_pair = 0.0;
    int match_limit = 1;
    cms::IndexGeom g{};
    double* sn = nullptr;
    double* rn = nullptr;
    uint32_t* tab = nullptr;
    cms::Entry* ent = nullptr;
    double* ent_a = nullptr;  // only with m/z weights
    uint32_t* bad = nullptr;
};

namespace {
void library_free(cms_library* L) {
    if (!L) return;
    cudaFree(L->sn);
    cudaFree(L->rn);
    cudaFree(L->tab);
    cudaFree(L->ent);
    cudaFree(L->ent_a);
    cudaFree(L->bad);
    delete L;
}
}  // namespace

extern "C" int cms_library_create(cms_ctx* ctx, const float* mz, const double* a, const double* b,
                                  const int64_t* off, int64_t n, int64_t n_peaks,
                                  double tolerance, double shift, int match_limit,
                                  const cms_cosine_config* cfg, cms_library** out, void* stream) {
    using namespace cms;
    if (!ctx || !out) {
        set_error("cms_library_create: null context or output");
        return CMS_ERR_INVALID;
    }
    *out = nullptr;
    CosineArgs args{SpecSet{mz, a, b, off, n, n_peaks}, SpecSet{mz, a, b, off, n, n_peaks},
                    tolerance, shift, match_limit};
    if (!check_common(args, "cms_library_create")) return CMS_ERR_INVALID;
    if (n <= 0) {
        set_error("cms_library_create: empty library");
        return CMS_ERR_INVALID;
    }
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t s = (cudaStream_t)stream;
    cms_library* L = new cms_library();
    L->device = ctx->device;
    L->spec = args.ref;
    L->tol = tolerance;
    L->shift = shift;
    L->match_limit = match_limit;
    L->cand_per_pair = (cfg && cfg->cand_per_pair > 0.0) ? cfg->cand_per_pair : 0.0;
    const int tile = (int)std::min<int64_t>((cfg && cfg->tile_spectra > 0) ? cfg->tile_spectra
                                                                            : 1024, n);
    if (tile > kMaxTile) {
        delete L;
        set_error("cms_library_create: tile_spectra must be <= %d", kMaxTile);
        return CMS_ERR_UNSUPPORTED;
    }
    double w = (cfg && cfg->bucket_width > 0.0) ? cfg->bucket_width : 2.0 * tolerance;
    if (w < tolerance) w = tolerance;
    if (!(w > 0.0)) w = 1e-3;
    const double avg_tile_peaks = (double)n_peaks * tile / (double)n;
    int nb = (cfg && cfg->n_buckets > 0) ? next_pow2(cfg->n_buckets)
                                         : next_pow2((long long)std::max(1024.0, avg_tile_peaks));
    nb = std::min(nb, 1 << 22);
    L->g = IndexGeom{tile, (int)((n + tile - 1) / tile), nb, 1.0 / w};
    const size_t n_tab = (size_t)L->g.n_tiles * (nb + 1), n_cur = (size_t)L->g.n_tiles * nb;
    const int n_chunks = L->g.n_tiles * scan_chunks(nb);
    uint32_t* cur = nullptr;  // bucket counts, then the chunk sums
    cudaError_t e = cudaMalloc(&L->bad, 64);
    if (e == cudaSuccess) e = cudaMalloc(&L->sn, sizeof(double) * n);
    if (e == cudaSuccess) e = cudaMalloc(&L->rn, sizeof(double) * n);
    if (e == cudaSuccess && a)
        e = cudaMalloc(&L->ent_a, sizeof(double) * std::max<int64_t>(1, n_peaks));
    if (e == cudaSuccess) e = cudaMalloc(&L->tab, sizeof(uint32_t) * n_tab);
    if (e == cudaSuccess) e = cudaMalloc(&L->ent, sizeof(Entry) * std::max<int64_t>(1, n_peaks));
    if (e == cudaSuccess) e = cudaMalloc(&cur, sizeof(uint32_t) * (n_cur + n_chunks));
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        cudaFree(cur);
        library_free(L);
        set_error("cms_library_create: device allocation failed (%s)", cudaGetErrorString(e));
        return CMS_ERR_NOMEM;
    }
    e = cudaMemsetAsync(L->bad, 0, 64, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(cur, 0, sizeof(uint32_t) * n_cur, s);
    if (e == cudaSuccess) {
        const int sms = ctx->sm_count;
        launch_prep(PrepSide{L->spec, L->sn, L->rn, nullptr, cur}, PrepSide{}, L->g, L->bad,
                    ctx->err_word, CMS_MAX_PEAKS, sms, s);
        index_sums_kernel<<<n_chunks, kScanThreads, 0, s>>>(L->g, cur, cur + n_cur, L->bad);
        index_scan_kernel<<<n_chunks, kScanThreads, 0, s>>>(L->g, cur, L->tab, cur + n_cur, L->bad);
        index_scatter_kernel<false><<<blocks_for(n, kScatterThreads / 32, sms), kScatterThreads, 0,
                                      s>>>(L->spec, L->g, cur, L->ent, L->ent_a, L->bad);
        e = cudaGetLastError();
    }
    uint32_t hbad = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hbad, L->bad, sizeof(uint32_t),
                                              cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(cur);
    if (e != cudaSuccess) {
        library_free(L);
        return cuda_fail(e, "cms_library_create");
    }
    if (hbad) {
        library_free(L);
        set_error("cms_library_create: invalid library spectra (offsets or peak counts)");
        return CMS_ERR_DEVICE;
    }
    *out = L;
    return CMS_OK;
}

extern "C" int cms_library_destroy(cms_library* lib) {
    if (!lib) return CMS_OK;
    cudaSetDevice(lib->device);
    cudaDeviceSynchronize();
    library_free(lib);
    return CMS_OK;
}

extern "C" int cms_library_search(cms_ctx* ctx, const cms_library* lib, const float* q_mz,
                                  const double* q_a, const double* q_b, const int64_t* q_off,
                                  int64_t n_q, int64_t n_q_peaks, float threshold,
                                  int32_t* hit_ref, int32_t* hit_query, float* hit_score,
                                  int32_t* hit_matches, uint8_t* hit_overflow, int64_t capacity,
                                  int64_t* hit_count, void* stream) {
    using namespace cms;
    if (!ctx || !lib) {
        set_error("cms_library_search: null context or library");
        return CMS_ERR_INVALID;
    }
    if (ctx->device != lib->device) {
        set_error("cms_library_search: context and library are on different devices");
        return CMS_ERR_INVALID;
    }
    const SpecSet Q{q_mz, q_a, q_b, q_off, n_q, n_q_peaks};
    if (!check_specset(Q, "query")) return CMS_ERR_INVALID;
    if (!(threshold > 0.0f)) {
        set_error("cms_library_search: threshold must be > 0");
        return CMS_ERR_INVALID;
    }
    if (capacity < 0 || !hit_count || (capacity > 0 && (!hit_ref || !hit_query || !hit_score ||
                                                        !hit_matches || !hit_overflow))) {
        set_error("cms_library_search: invalid hit buffers");
        return CMS_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    CMS_CUDA_TRY(cudaSetDevice(ctx->device));
    CMS_CUDA_TRY(cudaMemsetAsync(hit_count, 0, sizeof(int64_t), s));
    if (n_q == 0) return CMS_OK;

    const int cap = list_cap(next_pow2(std::max(2, lib->match_limit)), 128);
    const int cache = pair_cache(cap, 128, ctx->smem_optin);
    const size_t pair_smem = pair_smem_bytes(cap, 128, cache);
    if (pair_smem > ctx->smem_optin) {
        set_error("cms_library_search: match_limit too large for shared memory");
        return CMS_ERR_UNSUPPORTED;
    }
    const long long items = (long long)n_q * lib->g.n_tiles;
    const unsigned int spill_cap =
        (unsigned int)std::min<long long>(std::max<long long>(1 << 16, items), 1 << 24);
    // global-pool slices for up to four resident CTAs per SM (more CTAs per
    // SM run with the shared-memory pool only)
    const size_t gpool_warps =
        (size_t)std::min(ctx->sm_count * 4, kSlotWords * 32) * kJoinWarps;
    const size_t gpool_bytes = gpool_warps * (size_t)kGPool * 16;
    size_t need = bump_size(64 * sizeof(uint64_t)) + bump_size(n_q * sizeof(double)) +
                  bump_size(n_q * sizeof(SweepItem)) +
                  bump_size((size_t)std::max<int64_t>(1, n_q_peaks) * sizeof(Probe)) +
                  bump_size((size_t)spill_cap * sizeof(int2)) +
                  bump_size(kSlotWords * sizeof(uint32_t)) + bump_size(gpool_bytes) + 4096;
    const bool maybe_long = may_be_long(Q) || may_be_long(lib->spec);
    if (maybe_long) need += bump_size(long_bits_bytes(ctx->sm_count));
    int rc = arena_reserve(ctx, ctx->scratch, need, s);
    if (rc) return rc;
    Bump bp{(char*)ctx->scratch.ptr, 0, ctx->scratch.bytes};
    uint64_t* small = bp.take<uint64_t>(64);
    uint32_t* bad = reinterpret_cast<uint32_t*>(small);
    uint32_t* cls_count = reinterpret_cast<uint32_t*>(small + 1);
    uint32_t* cls_cursor = reinterpret_cast<uint32_t*>(small + 10);
    unsigned long long* spill_count = reinterpret_cast<unsigned long long*>(small + 20);
    unsigned long long* work_join = reinterpret_cast<unsigned long long*>(small + 21);
    unsigned long long* work_pair = reinterpret_cast<unsigned long long*>(small + 22);
    uint32_t* slots = bp.take<uint32_t>(kSlotWords);  // cleared with the counters before it
    CMS_CUDA_TRY(cudaMemsetAsync(small, 0, bp.used, s));
    double* snQ = bp.take<double>(n_q);
    SweepItem* sweep = bp.take<SweepItem>(n_q);
    Probe* probe = bp.take<Probe>((size_t)std::max<int64_t>(1, n_q_peaks));
    int2* spill = bp.take<int2>(spill_cap);
    unsigned char* gpool = bp.take<unsigned char>(gpool_bytes);
    uint32_t* long_bits =
        maybe_long ? bp.take<uint32_t>(long_bits_bytes(ctx->sm_count) / 4) : nullptr;

    {
        StageScope sc(ctx, 0, 2, s);
        launch_prep(PrepSide{Q, snQ, nullptr, cls_count}, PrepSide{}, lib->g, bad, ctx->err_word,
                    CMS_MAX_PEAKS, ctx->sm_count, s);
        launch_probe(ProbeArgs{Q, probe, nullptr, lib->tol, lib->shift, 0}, lib->g, bad,
                     ctx->err_word, ctx->sm_count, s);
    }
    {
        StageScope sc(ctx, 1, 1, s);
        order_scatter_kernel<<<blocks_for(n_q, kOrderThreads, ctx->sm_count), kOrderThreads, 0, s>>>(
            Q, snQ, cls_count, cls_cursor, sweep, bad);
    }
    CMS_CUDA_TRY(cudaGetLastError());

    SparseOut so{hit_ref, hit_query, hit_score, hit_matches, hit_overflow, capacity,
                 reinterpret_cast<unsigned long long*>(hit_count), threshold};
    JoinParams jp{};  // width_by_class zero: widths from cand_per_pair
    jp.A = Q;
    jp.B = lib->spec;
    jp.items = sweep;
    jp.probe = probe;
    jp.w = Q.b;
    jp.snA = snQ;
    jp.snB = lib->sn;
    jp.rnB = lib->rn;
    jp.cls_count = cls_count;
    jp.tab = lib->tab;
    jp.ent = lib->ent;
    jp.ent_a = lib->ent_a;
    jp.g = lib->g;
    jp.tol = lib->tol;
    jp.match_limit = lib->match_limit;
    // A search runs as kSearchWaves waves of short-lived CTAs (an equal share
    // of fetches per warp) so that searches on other streams interleave with
    // it on the device; each CTA claims a global-pool slice while it lives.
    jp.pool_smem = join_pool(lib->g.tile);
    jp.pool_max = kPoolMax;
    jp.gpool = gpool;
    jp.slots = slots;
    jp.init_width_scale = 0.f;
    if (lib->cand_per_pair > 0.0 && n_q > 0) {
        const double mean_na = (double)n_q_peaks / (double)n_q;
        const double lambda = lib->cand_per_pair / std::max(1.0, mean_na);
        jp.init_width_scale = (float)(0.5 * jp.pool_max / lambda);
    }
    jp.warp_smem_bytes = warp_slice_bytes(lib->g.tile);
    jp.work = work_join;
    jp.spill = SpillList{spill, spill_count, spill_cap};
    jp.dense = DenseOut{nullptr, nullptr, nullptr, 0};
    jp.sparse = so;
    jp.err = ctx->err_word;
    jp.bad = bad;
    {
        StageScope sc(ctx, 3, 1, s);
        rc = launch_join<false, true, false>(ctx, jp, (size_t)jp.warp_smem_bytes * kJoinWarps,
                                             gpool_warps, items, s, kSearchWaves);
        if (rc) return rc;
    }
    PairParams pp{};
    pp.R = lib->spec;
    pp.Q = Q;
    pp.snR = lib->sn;
    pp.snQ = snQ;
    pp.tol = lib->tol;
    pp.shift = lib->shift;
    pp.match_limit = lib->match_limit;
    pp.cap = cap;
    pp.cache = cache;
    pp.used_words = kUsedWords;
    pp.long_bits = long_bits;
    pp.pairs = spill;
    pp.n_pairs = spill_count;
    pp.pairs_cap = spill_cap;
    pp.work = work_pair;
    pp.dense = DenseOut{nullptr, nullptr, nullptr, 0};
    pp.sparse = so;
    pp.err = ctx->err_word;
    pp.bad = bad;
    {
        StageScope sc(ctx, 4, 1, s);
        if ((rc = set_func_smem(pair_kernel<true, false, true>, pair_smem))) return rc;
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pair_kernel<true, false, true>, 128,
                                                      pair_smem);
        pair_kernel<true, false, true><<<std::max(1, std::min(ctx->sm_count * std::max(1, std::min(kLongWarps, per_sm)),
                                                  (int)std::min<long long>(spill_cap, 1 << 20))),
                            128, pair_smem, s>>>(pp);
    }
    CMS_CUDA_TRY(cudaGetLastError());
    return CMS_OK;
}
