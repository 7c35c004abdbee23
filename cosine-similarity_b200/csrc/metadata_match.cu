// matchms' metadata and m/z-set similarities that the reference prototypes
// beside its CUDA classes (notebooks/prototyping/other_similarities.ipynb
// imports matchms' ParentMassMatch, PrecursorMzMatch and IntersectMz next to
// CosineGreedy, ModifiedCosine and FingerprintSimilarity):
//
//   mass_match_kernel      ParentMassMatch / PrecursorMzMatch: one value per
//                          spectrum (parent mass or precursor m/z, float64);
//                          a pair matches when |r - q| <= tolerance (Dalton)
//                          or |r - q| / ((r + q) / 2) * 1e6 <= tolerance
//                          (ppm), in IEEE float64 in that order of
//                          operations.  Output: one byte (0/1) per pair.
//                          Bound by the output's write: float32 bounds per row
//                          decide all but the pairs within rounding of the
//                          tolerance, and rows of any alignment are written in
//                          16-byte stores.
//   intersect_mz_kernel    IntersectMz: |set(mz_r) & set(mz_q)| / |set(mz_r)
//                          | set(mz_q)| * scaling on the exact float64 m/z
//                          values (0 when both are empty), through a hashed
//                          index of the queries' distinct values: per
//                          (reference, query tile) the reference's distinct
//                          values find their (value, query) entries and count
//                          them per query in shared memory; the tile's row is
//                          filled, and scaling * inter / union in float64 is
//                          stored for the queries that share a value.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "cms_internal.cuh"

namespace cms {
namespace {

constexpr int kMassThreads = 256;
constexpr int kMassCols = 16;                              // columns per thread
constexpr int kMassWarpCols = 32 * kMassCols;              // 512
// Queries per CTA pass.  With the static arrays a CTA of this tile has 63 KB of shared
// memory and three of 512 threads fit a multiprocessor (four up to some 8100 queries).
// A row's bucket walk is done once a tile, so fewer tiles are faster as long as three
// fit: 10007 x 9000 in one pass 308 us, in two of 4504 338 us; 12000 x 12000, where one
// pass leaves two CTAs, in two of 6000 486 us, in one of 12000 503 us.
constexpr int kIxMaxTile = 9216;

__device__ __forceinline__ bool mass_ok(double r, double q, double tol, int ppm) {
    const double d = fabs(__dsub_rn(r, q));
    if (!ppm) return d <= tol;
    // (r + q) / 2: halving is exact scaling, the same rounding as division
    const double mean = __dmul_rn(__dadd_rn(r, q), 0.5);
    return __dmul_rn(__ddiv_rn(d, mean), 1e6) <= tol;
}

// The float32 bounds of one row's matches in ppm.  In exact arithmetic the
// matching q > 0 of a row r > 0 form an interval; rounding blurs its ends by far
// less than the margin below, so with x = float32(q), rounded to nearest,
//   x < out_lo or x > out_hi:  no match;   x > in_lo and x < in_hi:  a match
// (rounding is monotone, and a float32 strictly above in_lo comes from a q
// above in_lo); what lies between is tested as the definition says.  Rows the
// argument does not hold for (r not positive or extreme; a tolerance above
// kMaxBoundPpm, where the ratio's bound of 2e6 gets near) take every column that way, and so
// do negative q, whose mean may be negative.  mid and half describe [out_lo,
// out_hi] once more, rounded outwards far enough that float32(|x - mid|) <= half
// for every x inside.
constexpr double kMaxBoundPpm = 5e5;
struct MassRow {
    float mid, half, out_lo, out_hi;
    float in_lo, in_hi, pad0, pad1;
};
__device__ __forceinline__ MassRow mass_row(double r, double tol) {
    MassRow w{0.0f, INFINITY, -INFINITY, INFINITY, INFINITY, -INFINITY, 0.0f, 0.0f};
    if (!(tol >= 0.0 && tol <= kMaxBoundPpm && r >= 1e-150 && r <= 1e150)) return w;
    const double h = tol * 0.5e-6, m = r * 4e-15;
    const double lo = r * (1.0 - h) / (1.0 + h), hi = r * (1.0 + h) / (1.0 - h);
    w.out_lo = __double2float_rd(lo - m);
    w.out_hi = __double2float_ru(hi + m);
    w.in_lo = __double2float_ru(lo + m);
    w.in_hi = __double2float_rd(hi - m);
    if (w.out_hi < 1e30f) {
        w.mid = __double2float_rn(0.5 * ((double)w.out_lo + (double)w.out_hi));
        const double up = (double)w.out_hi - (double)w.mid, down = (double)w.mid - (double)w.out_lo;
        w.half = __double2float_ru(fmax(up, down) * (1.0 + 0x1p-20) + 1e-30);
    }
    return w;
}

// One pair, from the row's bounds or, between them, as defined.
__device__ __forceinline__ bool ppm_ok(const double* r, const double* q, const MassRow& w, double tol) {
    const double v = *q;
    const float f = __double2float_rn(v);
    if (f > w.in_lo && f < w.in_hi && !(v < 0.0)) return true;
    if (!(f >= w.out_lo && f <= w.out_hi) && !(v < 0.0)) return false;
    return mass_ok(*r, v, tol, 1);
}

// two float32 sums in one instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "add.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// bits 0..3 of m as the bytes of a word
__device__ __forceinline__ uint32_t nibble_bytes(uint32_t m) {
    return ((m & 0xFu) * 0x00204081u) & 0x01010101u;
}

// Writes 32 lanes' 16-bit masks (any: ballot of those that may be nonzero) as 512
// bytes at row..row + 511, `mine` being this lane's first byte: aligned 16-byte
// stores whatever the row's alignment, a lane's piece shifted together with its
// neighbour's, and the 16 bytes left at the two ends of the 512 one by one.
__device__ __forceinline__ void store_masks(uint8_t* mine, int lane, uint32_t mask, unsigned any) {
    const unsigned full = 0xffffffffu;
    const int sh = (int)(-(uintptr_t)mine & 15);  // bytes up to the next boundary
    uint4 piece = make_uint4(0u, 0u, 0u, 0u);
    if (any) {
        const uint32_t next = __shfl_down_sync(full, mask, 1);
        const uint32_t m = ((mask | (next << 16)) >> sh) & 0xFFFFu;
        piece = make_uint4(nibble_bytes(m), nibble_bytes(m >> 4), nibble_bytes(m >> 8),
                           nibble_bytes(m >> 12));
    }
    if (sh == 0) {
        __stcs(reinterpret_cast<uint4*>(mine), piece);
        return;
    }
    if (lane < 31) __stcs(reinterpret_cast<uint4*>(mine + sh), piece);
    const uint32_t end = __shfl_sync(full, mask, lane < sh ? 0 : 31);
    uint8_t* row = mine - 16 * lane;
    if (lane < 16)
        row[lane < sh ? lane : kMassWarpCols - 16 + lane] = (uint8_t)((end >> lane) & 1u);
}

// The last columns of a row, 32 bytes at a time.
__device__ __forceinline__ void store_tail(uint8_t* row, int lane, uint32_t mask, int cols) {
    for (int k = 0; k < cols; k += 32) {
        const uint32_t m = __shfl_sync(0xffffffffu, mask, (k + lane) >> 4);
        if (k + lane < cols) row[k + lane] = (uint8_t)((m >> (lane & 15)) & 1u);
    }
}

// A warp takes `rows` rows x 512 columns, 16 consecutive columns a lane.
//
// Dalton: the columns' float64 values stay in registers, a subtraction and a
// compare per pair; bound by the write (40000 x 50000: 406 us, 75% of the copy
// rate; 49999 columns 566 us, where a store per byte took 5960 us).
//
// ppm: a float64 division per pair took 2240 us, seven times the write.  Most
// rows match none of a warp's columns; the smallest float32 |x - mid| of a
// lane's columns (one and a half instructions per pair) shows it, and zeros go
// out.  A few lanes that may have a match are looked at by half a warp each, a
// column a lane; many at once make their masks themselves.  420 us (49999
// columns: 487 us, 6030 us with a store per byte).
//
// ppm with a tolerance that the bounds do not cover (above kMaxBoundPpm, negative,
// NaN): as in Dalton mode, with a division per pair (8000 x 8192: 115 us; with
// every pair passed over by the bounds 407).
enum MassKind { kDalton, kPpm, kPpmExact };
template <MassKind KIND>
__global__ void __launch_bounds__(kMassThreads, 3)
mass_match_kernel(const double* __restrict__ ref, int64_t n_ref, const double* __restrict__ q,
                  int64_t n_q, double tol, uint8_t* __restrict__ out, int64_t ld, int rows) {
    __shared__ __align__(16) MassRow s_row[kMassThreads / 32][32];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t col_blocks = (n_q + kMassWarpCols - 1) / kMassWarpCols;
    const int64_t units = col_blocks * ((n_ref + rows - 1) / rows);
    const int64_t warps = (int64_t)gridDim.x * (kMassThreads / 32);
    MassRow* const bounds = s_row[threadIdx.x >> 5];
    for (int64_t t = (int64_t)blockIdx.x * (kMassThreads / 32) + (threadIdx.x >> 5); t < units;
         t += warps) {
        const int64_t rb = t / col_blocks, c0 = (t - rb * col_blocks) * kMassWarpCols;
        const int cols = (int)min((int64_t)kMassWarpCols, n_q - c0);
        const double* const qc = q + c0;  // this warp's columns
        const double* rp = ref + rb * rows;
        int left = (int)min((int64_t)rows, n_ref - rb * rows);
        uint8_t* mine = out + rb * rows * ld + c0 + kMassCols * lane;
        if (KIND != kPpm) {
            double v[kMassCols];
#pragma unroll
            for (int k = 0; k < kMassCols; ++k)
                v[k] = kMassCols * lane + k < cols ? qc[kMassCols * lane + k]
                                                   : __longlong_as_double(0x7ff8000000000000ll);
            if (cols == kMassWarpCols && ((ld | (int64_t)(uintptr_t)out) & 15) == 0) {
                // aligned rows: bytes straight into their words
                for (; left; --left, ++rp, mine += ld) {
                    const double r = *rp;
                    uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                    for (int k = 0; k < kMassCols; ++k)
                        w[k >> 2] |= (uint32_t)mass_ok(r, v[k], tol, KIND == kPpmExact) << (8 * (k & 3));
                    __stcs(reinterpret_cast<uint4*>(mine), make_uint4(w[0], w[1], w[2], w[3]));
                }
                continue;
            }
            for (; left; --left, ++rp, mine += ld) {
                const double r = *rp;
                uint32_t mask = 0u;
#pragma unroll
                for (int k = 0; k < kMassCols; ++k)
                    if (mass_ok(r, v[k], tol, KIND == kPpmExact)) mask |= 1u << k;
                if (cols == kMassWarpCols)
                    store_masks(mine, lane, mask, 1u);
                else
                    store_tail(mine - kMassCols * lane, lane, mask, cols);
            }
            continue;
        }
        float2 x[kMassCols / 2];
        uint32_t odd = 0u;
#pragma unroll
        for (int k = 0; k < kMassCols; ++k) {
            const double v = kMassCols * lane + k < cols ? qc[kMassCols * lane + k]
                                                         : __longlong_as_double(0x7ff8000000000000ll);
            (k & 1 ? x[k / 2].y : x[k / 2].x) = __double2float_rn(v);
            odd |= (v < 0.0 ? 1u : 0u) << k;
            if ((k & 3) == 3) asm volatile("" ::: "memory");  // four loads in flight, not sixteen
        }
        for (; left > 0; left -= 32, rp += 32) {
            const int nr = min(32, left);
            __syncwarp();
            if (lane < nr) bounds[lane] = mass_row(rp[lane], tol);
            __syncwarp();
#pragma unroll 1
            for (int rr = 0; rr < nr; ++rr, mine += ld) {
                float a = INFINITY, b = INFINITY;  // a NaN (past the end) never is least
                {
                    const float2 w = *reinterpret_cast<const float2*>(&bounds[rr]);
                    const float2 neg = make_float2(-w.x, -w.x);
#pragma unroll
                    for (int k = 0; k < kMassCols / 2; ++k) {
                        const float2 d = add2(x[k], neg);
                        a = fminf(a, fabsf(d.x));
                        b = fminf(b, fabsf(d.y));
                    }
                    a = fminf(a, b);
                    b = w.y;
                }
                const unsigned any = __ballot_sync(full, a <= b || odd != 0u);
                uint32_t mask = 0u;
                if (any) {
                    if (__popc(any) <= 4) {
                        // half a warp for each of the lanes, a column a lane
                        for (unsigned m = any; m;) {
                            const int l0 = __ffs(m) - 1;
                            m &= m - 1u;
                            const int l1 = m ? __ffs(m) - 1 : -1;
                            m &= m - 1u;
                            const int l = lane < 16 ? l0 : l1, j = 16 * l + (lane & 15);
                            const bool ok = l >= 0 && j < cols && ppm_ok(rp + rr, qc + j, bounds[rr], tol);
                            const unsigned hit = __ballot_sync(full, ok);
                            if (lane == l0) mask = hit & 0xFFFFu;
                            if (lane == l1) mask = hit >> 16;
                        }
                    } else {
                        if ((any >> lane) & 1u) {
                            uint32_t rest = odd;
                            const MassRow& w = bounds[rr];
#pragma unroll
                            for (int k = 0; k < kMassCols; ++k) {
                                const float v = k & 1 ? x[k / 2].y : x[k / 2].x;
                                if (v >= w.out_lo && v <= w.out_hi) rest |= 1u << k;
                                if (v > w.in_lo && v < w.in_hi) mask |= 1u << k;
                            }
                            mask &= ~odd;
                            for (rest &= ~mask; rest; rest &= rest - 1u) {
                                const int k = __ffs(rest) - 1;
                                if (ppm_ok(rp + rr, qc + kMassCols * lane + k, w, tol)) mask |= 1u << k;
                            }
                        }
                        __syncwarp();
                    }
                }
                if (cols == kMassWarpCols)
                    store_masks(mine, lane, mask, any);
                else
                    store_tail(mine - kMassCols * lane, lane, mask, cols);
            }
        }
    }
}

// [a0, a1) of spectrum i, clamped to [0, total]; a clamp sets the error word
__device__ __forceinline__ void spectrum_range(const int64_t* off, int64_t i, int64_t total,
                                               int64_t& a0, int64_t& a1, uint32_t* err) {
    a0 = off[i];
    a1 = off[i + 1];
    if (a0 < 0 || a1 < a0 || a1 > total) {
        if (err) atomicOr(err, kErrBadOffsets);
        a0 = a1 = 0;
    }
}

// ---- IntersectMz through an index of the queries' distinct m/z values ----
// Pairs sharing a value are few against R x Q, so instead of merging every
// pair's peak lists, the queries' distinct (value, query) entries are hashed
// into buckets (count, two-launch scan, scatter), and each (reference, query
// tile) CTA walks the buckets of its reference's distinct values, counting
// shared values per query in shared memory, then writes the tile's dense row.
struct __align__(16) IxEntry {
    double v;
    uint32_t q;
    uint32_t pad;
};

// bucket of an m/z value: its bit pattern (+0 and -0 folded) mixed by the
// splitmix64 finalizer
__device__ __forceinline__ uint32_t ix_bucket(double v, uint32_t mask) {
    unsigned long long z = v == 0.0 ? 0ull : (unsigned long long)__double_as_longlong(v);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (uint32_t)z & mask;
}

// one warp per query spectrum: its distinct values (sorted peaks: a value
// differing from its predecessor) counted per bucket (SCATTER = false) or
// placed (SCATTER = true); ub[j] = distinct values of query j.  kIxUnroll
// chunks of 32 peaks have their loads and atomics in flight together.
constexpr int kIxUnroll = 4;
template <bool SCATTER>
__global__ void ix_index_kernel(const double* __restrict__ qmz, const int64_t* __restrict__ qoff,
                                int64_t n_q, int64_t n_q_peaks, uint32_t mask, uint32_t* cnt_cur,
                                IxEntry* ent, uint32_t* ub, uint32_t* err) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t j = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; j < n_q; j += warps) {
        int64_t b0, b1;
        spectrum_range(qoff, j, n_q_peaks, b0, b1, (!SCATTER && lane == 0) ? err : nullptr);
        uint32_t distinct = 0;
        for (int64_t k0 = b0 + lane; k0 < b1; k0 += 32 * kIxUnroll) {
            double v[kIxUnroll], before[kIxUnroll];
            uint32_t pos[kIxUnroll];
            bool take[kIxUnroll];
#pragma unroll
            for (int u = 0; u < kIxUnroll; ++u) {
                const int64_t k = k0 + 32 * u;
                v[u] = k < b1 ? qmz[k] : 0.0;
                before[u] = k < b1 && k > b0 ? qmz[k - 1] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kIxUnroll; ++u) {
                const int64_t k = k0 + 32 * u;
                take[u] = k < b1 && !(k > b0 && before[u] == v[u]);
                if (!take[u]) continue;
                ++distinct;
                uint32_t* c = &cnt_cur[ix_bucket(v[u], mask)];
                if (SCATTER)
                    pos[u] = atomicAdd(c, 1u);
                else
                    atomicAdd(c, 1u);
            }
            if (SCATTER) {
#pragma unroll
                for (int u = 0; u < kIxUnroll; ++u)
                    if (take[u])
                        *reinterpret_cast<uint4*>(&ent[pos[u]]) =
                            make_uint4((uint32_t)__double2loint(v[u]),
                                       (uint32_t)__double2hiint(v[u]), (uint32_t)j, 0u);
            }
        }
        if (!SCATTER) {
            distinct = __reduce_add_sync(0xffffffffu, distinct);
            if (lane == 0) ub[j] = distinct;
        }
    }
}

// Exclusive scan of the bucket counts into tab[0..nb] (cnt_cur becomes the
// scatter cursor): chunk sums, then every chunk's own scan on top of the sums
// of the chunks before it, both with coalesced accesses.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanChunk = kScanThreads * kScanPer;  // 4096 buckets; divides every bucket count

// sum over the block; the same value for every thread
__device__ __forceinline__ uint32_t block_total(uint32_t x, uint32_t* s_warp) {
    x = __reduce_add_sync(0xffffffffu, x);
    __syncthreads();  // s_warp free from an earlier use
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
    __syncthreads();
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) total += s_warp[w];
    return total;
}

// exclusive scan over the block of one value per thread
template <int THREADS>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    __syncthreads();  // s_warp free from an earlier use
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    uint32_t run = incl - x;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w)
        if (w < wid) run += s_warp[w];
    return run;
}

__global__ void __launch_bounds__(kScanThreads) ix_chunk_sums(const uint32_t* cnt, uint32_t* sums) {
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const uint32_t* c = cnt + (size_t)blockIdx.x * kScanChunk;
    uint32_t x = 0;
#pragma unroll
    for (int r = 0; r < kScanPer; ++r) x += c[r * kScanThreads + threadIdx.x];
    x = block_total(x, s_warp);
    if (threadIdx.x == 0) sums[blockIdx.x] = x;
}

__global__ void __launch_bounds__(kScanThreads) ix_chunk_scan(uint32_t* cnt_cur, uint32_t* tab,
                                                              const uint32_t* sums) {
    __shared__ uint32_t s_val[kScanChunk + kScanThreads];
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const int tid = threadIdx.x;
    uint32_t* c = cnt_cur + (size_t)blockIdx.x * kScanChunk;
    uint32_t* out = tab + (size_t)blockIdx.x * kScanChunk;
    // coalesced in, kScanPer consecutive buckets a thread out of shared memory
    // (a word of padding per kScanPer)
#pragma unroll
    for (int r = 0; r < kScanPer; ++r) {
        const int k = r * kScanThreads + tid;
        s_val[k + k / kScanPer] = c[k];
    }
    uint32_t prev = 0;
    for (int i = tid; i < (int)blockIdx.x; i += kScanThreads) prev += sums[i];
    prev = block_total(prev, s_warp);
    uint32_t x = 0;
#pragma unroll
    for (int r = 0; r < kScanPer; ++r) x += s_val[tid * (kScanPer + 1) + r];
    uint32_t run = prev + block_excl_scan<kScanThreads>(x, s_warp);
#pragma unroll
    for (int r = 0; r < kScanPer; ++r) {
        const uint32_t v = s_val[tid * (kScanPer + 1) + r];
        s_val[tid * (kScanPer + 1) + r] = run;
        run += v;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kScanPer; ++r) {
        const int k = r * kScanThreads + tid;
        const uint32_t v = s_val[k + k / kScanPer];
        out[k] = v;
        c[k] = v;
    }
    if (blockIdx.x == gridDim.x - 1 && tid == kScanThreads - 1) out[kScanChunk] = run;
}

// One CTA per (reference, tile of `tile` queries).  256 reference values at a
// time look up their buckets; the buckets' entries, laid end to end, are taken
// one a thread (owner by binary search over the running counts), so a value
// that every query has costs no more than its entries.  Counts live in shared
// memory between references: a query's first hit puts it on a list, the row is
// filled with the score of no shared value by 16-byte stores, and only the
// list's queries get a division, their score over the fill, and their counter
// back to zero.  10007 x 9000, index and all: 308 us (the row write alone: 110
// us; what is left is the latency of a unit's dependent lookups).  Clearing and
// scanning 8192 counters per unit, with a float64 division for each query, took
// 850 us.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) intersect_mz_kernel(
    const double* __restrict__ rmz, const int64_t* __restrict__ roff, int64_t n_ref,
    int64_t n_ref_peaks, int64_t n_q, const uint32_t* __restrict__ tab,
    const IxEntry* __restrict__ ent, const uint32_t* __restrict__ ub, uint32_t mask,
    double scaling, double* __restrict__ out, int64_t ld, int tile, uint32_t* err) {
    extern __shared__ uint32_t s_cnt[];                              // [tile]
    uint16_t* s_list = reinterpret_cast<uint16_t*>(s_cnt + tile);    // [tile]
    __shared__ uint32_t s_warp[THREADS / 32];
    __shared__ uint32_t s_end[THREADS];  // running entry counts of the values
    __shared__ uint32_t s_first[THREADS];
    __shared__ double s_v[THREADS];
    __shared__ unsigned int s_n;
    const int64_t tiles = (n_q + tile - 1) / tile;
    const int tid = threadIdx.x;
    for (int k = tid; k < tile; k += THREADS) s_cnt[k] = 0u;
    if (tid == 0) s_n = 0u;
    const double none = __dmul_rn(scaling, 0.0);
    for (int64_t u = blockIdx.x; u < n_ref * tiles; u += gridDim.x) {
        const int64_t i = u / tiles, j0 = (u - i * tiles) * tile;
        const int tw = (int)min((int64_t)tile, n_q - j0);
        int64_t a0, a1;
        spectrum_range(roff, i, n_ref_peaks, a0, a1, (tid == 0 && j0 == 0) ? err : nullptr);
        uint32_t ua = 0;  // distinct reference values
        for (int64_t k0 = a0; k0 < a1; k0 += THREADS) {
            const int64_t k = k0 + tid;
            double v = 0.0;
            bool take = false;
            if (k < a1) {
                v = rmz[k];
                take = !(k > a0 && rmz[k - 1] == v);
            }
            uint32_t e0 = 0, c = 0;
            if (take) {
                const uint32_t h = ix_bucket(v, mask);
                e0 = tab[h];
                c = tab[h + 1] - e0;
            }
            const uint32_t excl = block_excl_scan<THREADS>(c, s_warp);
            s_end[tid] = excl + c;
            s_first[tid] = e0 - excl;
            s_v[tid] = v;
            ua += __syncthreads_count(take);
            const uint32_t total = s_end[THREADS - 1];
            for (uint32_t e = tid; e < total; e += THREADS) {
                int o = 0;  // values whose entries end at or before e
#pragma unroll
                for (int step = THREADS / 2; step > 0; step >>= 1)
                    if (s_end[o + step - 1] <= e) o += step;
                const uint4 x = __ldg(reinterpret_cast<const uint4*>(ent + (s_first[o] + e)));
                const int64_t q = (int64_t)x.z - j0;
                if (__hiloint2double((int)x.y, (int)x.x) == s_v[o] && q >= 0 && q < tw &&
                    atomicAdd(&s_cnt[q], 1u) == 0u)
                    s_list[atomicAdd(&s_n, 1u)] = (uint16_t)q;
            }
            __syncthreads();
        }
        // the row's fill: no shared value (and 0 for two empty spectra)
        double* orow = out + i * ld + j0;
        if (ua != 0u) {
            const int pre = min(tw, (int)(((uintptr_t)orow >> 3) & 1));
            if (tid < pre) orow[tid] = none;
            const int nv = (tw - pre) >> 1;
            for (int k = tid; k < nv; k += THREADS)
                __stcs(reinterpret_cast<double2*>(orow + pre) + k, make_double2(none, none));
            if (tid < ((tw - pre) & 1)) orow[tw - 1] = none;
        } else {
            for (int k = tid; k < tw; k += THREADS) orow[k] = ub[j0 + k] ? none : 0.0;
        }
        __syncthreads();
        const unsigned int n = s_n;
        for (unsigned int k = tid; k < n; k += THREADS) {
            const int q = s_list[k];
            const uint32_t inter = s_cnt[q];
            s_cnt[q] = 0u;
            orow[q] = __ddiv_rn(__dmul_rn(scaling, (double)inter),
                                (double)(ua + ub[j0 + q] - inter));
        }
        __syncthreads();
        if (tid == 0) s_n = 0u;
    }
}

int sm_count_of_current() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        sms = 148;
    }
    return sms;
}

// Workspace of one IntersectMz call: entries, bucket counts, bucket table, distinct
// counts, chunk sums.
struct IxSpace {
    uint32_t nb;  // buckets: a power of two >= the query peaks, 2^26 at most
    int chunks;
    size_t ent_bytes, bytes;
};
IxSpace ix_space(int64_t n_q, int64_t n_q_peaks) {
    IxSpace w{};
    w.nb = kScanChunk;
    while (w.nb < (uint64_t)n_q_peaks && w.nb < (1u << 26)) w.nb <<= 1;
    w.chunks = (int)(w.nb / kScanChunk);
    w.ent_bytes = (size_t)std::max<int64_t>(1, n_q_peaks) * sizeof(IxEntry);
    w.bytes = w.ent_bytes + ((size_t)w.nb * 2 + 1 + (size_t)n_q + (size_t)w.chunks) * 4;
    return w;
}

// What every entry point refuses; `launch` says whether there is anything to do.
int ix_check(const char* who, const double* ref_mz, const int64_t* ref_off, int64_t n_ref,
             int64_t n_ref_peaks, const double* q_mz, const int64_t* q_off, int64_t n_q,
             int64_t n_q_peaks, const double* out, int64_t ld, bool& launch) {
    launch = false;
    if (n_ref < 0 || n_q < 0 || n_ref_peaks < 0 || n_q_peaks < 0 || ld < n_q ||
        n_q > 0xFFFFFFFFll || n_q_peaks > 0x7FFFFFFFll) {
        set_error("%s: invalid sizes (ld >= n_q, n_q < 2^32, n_q_peaks < 2^31)", who);
        return CMS_ERR_INVALID;
    }
    if (n_ref == 0 || n_q == 0) return CMS_OK;
    if (!ref_off || !q_off || !out || (n_ref_peaks > 0 && !ref_mz) || (n_q_peaks > 0 && !q_mz)) {
        set_error("%s: null pointer", who);
        return CMS_ERR_INVALID;
    }
    launch = true;
    return CMS_OK;
}

// The launches, in a workspace of ix_space(n_q, n_q_peaks).bytes.
int ix_launch(const double* ref_mz, const int64_t* ref_off, int64_t n_ref, int64_t n_ref_peaks,
              const double* q_mz, const int64_t* q_off, int64_t n_q, int64_t n_q_peaks,
              double scaling, double* out, int64_t ld, uint32_t* device_error, unsigned char* ws,
              cudaStream_t s) {
    const IxSpace w = ix_space(n_q, n_q_peaks);
    const uint32_t nb = w.nb;
    const int sms = sm_count_of_current(), chunks = w.chunks;
    IxEntry* ent = reinterpret_cast<IxEntry*>(ws);
    uint32_t* cnt = reinterpret_cast<uint32_t*>(ws + w.ent_bytes);
    uint32_t* tab = cnt + nb;
    uint32_t* ub = tab + nb + 1;
    uint32_t* sums = ub + n_q;
    // query tile: the queries split evenly over the fewest tiles of at most
    // kIxMaxTile (six bytes of shared memory a query)
    const int64_t tiles = (n_q + kIxMaxTile - 1) / kIxMaxTile;
    const int tile = (int)(((n_q + tiles - 1) / tiles + 7) & ~int64_t(7));
    const size_t smem = (size_t)tile * 6;
    // 512 threads for long rows, 256 where a row is soon filled
    auto* kern = tile > 2048 ? intersect_mz_kernel<512> : intersect_mz_kernel<256>;
    const int threads = tile > 2048 ? 512 : 256;
    if (const int rc = raise_func_smem(reinterpret_cast<const void*>(kern), smem)) return rc;
    CMS_CUDA_TRY(cudaMemsetAsync(cnt, 0, (size_t)nb * 4, s));
    const int igrid = (int)std::max<int64_t>(
        1, std::min<int64_t>((n_q * 32 + 255) / 256, (int64_t)sms * 16));
    ix_index_kernel<false><<<igrid, 256, 0, s>>>(q_mz, q_off, n_q, n_q_peaks, nb - 1, cnt, nullptr,
                                                 ub, device_error);
    ix_chunk_sums<<<chunks, kScanThreads, 0, s>>>(cnt, sums);
    ix_chunk_scan<<<chunks, kScanThreads, 0, s>>>(cnt, tab, sums);
    ix_index_kernel<true><<<igrid, 256, 0, s>>>(q_mz, q_off, n_q, n_q_peaks, nb - 1, cnt, ent,
                                                nullptr, nullptr);
    const int64_t units = n_ref * ((n_q + tile - 1) / tile);
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    per_sm = std::max(1, per_sm);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(units, (int64_t)sms * per_sm));
    kern<<<grid, threads, smem, s>>>(ref_mz, ref_off, n_ref, n_ref_peaks, n_q, tab, ent, ub, nb - 1,
                                     scaling, out, ld, tile, device_error);
    CMS_CUDA_TRY(cudaGetLastError());
    return CMS_OK;
}

}  // namespace
}  // namespace cms

extern "C" int cms_mass_match(const double* ref, int64_t n_ref, const double* q, int64_t n_q,
                              double tolerance, int ppm, uint8_t* out, int64_t ld, void* stream) {
    using namespace cms;
    if (n_ref < 0 || n_q < 0 || ld < n_q || (ppm != 0 && ppm != 1)) {
        set_error("cms_mass_match: invalid sizes or ppm flag (ld >= n_q, ppm 0 or 1)");
        return CMS_ERR_INVALID;
    }
    if (n_ref == 0 || n_q == 0) return CMS_OK;
    if (!ref || !q || !out) {
        set_error("cms_mass_match: null pointer");
        return CMS_ERR_INVALID;
    }
    // Rows a warp takes: as many as leave twelve units a multiprocessor, because its
    // columns are loaded once for all of them, but not so that a second wave of warps
    // is short.  Dalton, cold cache: 8000 x 8192 33 us with 128 rows (1008 units for
    // 3552 resident warps), 26 with 64, 29 with 32, 45 with 8; 16000 x 16384 72 us with
    // 128 (4000 units), 66 with 64, 76 with 32; 12000 x 12288 41 us with 128, 47 with
    // 32; 500 x 100000 25 us with 32, 31 with 64; 40000 x 50000 410 us with 128, 424
    // with 64, where 20000 x 25000 (7700 units of 128) takes 189 and 175.
    // Ten CTAs per resident one, so that the last wave is short (one per resident:
    // 572 us instead of 420 for 40000 x 50000 in ppm).
    const int64_t sms = sm_count_of_current(), col_blocks = (n_q + kMassWarpCols - 1) / kMassWarpCols;
    const int64_t resident = sms * 24;
    auto units_of = [&](int r) { return col_blocks * ((n_ref + r - 1) / r); };
    int rows = 128;
    for (; rows > 4; rows /= 2) {
        const int64_t u = units_of(rows);
        if (u >= (rows == 128 ? 4 : 2) * resident || (u >= sms * 12 && u <= resident)) break;
    }
    const int64_t units = units_of(rows);
    const int per_block = kMassThreads / 32;
    const int grid = (int)std::max<int64_t>(
        1, std::min<int64_t>((units + per_block - 1) / per_block, sms * 30));
    cudaStream_t s = (cudaStream_t)stream;
    auto* kern = !ppm ? mass_match_kernel<kDalton>
                 : tolerance >= 0.0 && tolerance <= kMaxBoundPpm ? mass_match_kernel<kPpm>
                                                                 : mass_match_kernel<kPpmExact>;
    kern<<<grid, kMassThreads, 0, s>>>(ref, n_ref, q, n_q, tolerance, out, ld, rows);
    CMS_CUDA_TRY(cudaGetLastError());
    return CMS_OK;
}

extern "C" int cms_intersect_mz(const double* ref_mz, const int64_t* ref_off, int64_t n_ref,
                                int64_t n_ref_peaks, const double* q_mz, const int64_t* q_off,
                                int64_t n_q, int64_t n_q_peaks, double scaling, double* out,
                                int64_t ld, uint32_t* device_error, void* stream) {
    using namespace cms;
    bool launch;
    int rc = ix_check("cms_intersect_mz", ref_mz, ref_off, n_ref, n_ref_peaks, q_mz, q_off, n_q,
                      n_q_peaks, out, ld, launch);
    if (rc || !launch) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char* ws = nullptr;
    CMS_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void**>(&ws), ix_space(n_q, n_q_peaks).bytes, s));
    rc = ix_launch(ref_mz, ref_off, n_ref, n_ref_peaks, q_mz, q_off, n_q, n_q_peaks, scaling, out, ld,
                   device_error, ws, s);
    cudaFreeAsync(ws, s);  // stream-ordered: after the kernels
    return rc;
}

extern "C" int cms_intersect_mz_workspace(int64_t n_q, int64_t n_q_peaks, int64_t* bytes) {
    using namespace cms;
    if (!bytes || n_q < 0 || n_q_peaks < 0 || n_q > 0xFFFFFFFFll || n_q_peaks > 0x7FFFFFFFll) {
        set_error("cms_intersect_mz_workspace: invalid sizes (n_q < 2^32, n_q_peaks < 2^31)");
        return CMS_ERR_INVALID;
    }
    *bytes = (int64_t)ix_space(n_q, n_q_peaks).bytes;
    return CMS_OK;
}

extern "C" int cms_intersect_mz_in(const double* ref_mz, const int64_t* ref_off, int64_t n_ref,
                                   int64_t n_ref_peaks, const double* q_mz, const int64_t* q_off,
                                   int64_t n_q, int64_t n_q_peaks, double scaling, double* out,
                                   int64_t ld, uint32_t* device_error, void* workspace,
                                   int64_t workspace_bytes, void* stream) {
    using namespace cms;
    bool launch;
    const int rc = ix_check("cms_intersect_mz_in", ref_mz, ref_off, n_ref, n_ref_peaks, q_mz, q_off,
                            n_q, n_q_peaks, out, ld, launch);
    if (rc || !launch) return rc;
    const int64_t need = (int64_t)ix_space(n_q, n_q_peaks).bytes;
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 15) || workspace_bytes < need) {
        set_error("cms_intersect_mz_in: needs a 16-byte aligned workspace of %lld bytes",
                  (long long)need);
        return CMS_ERR_INVALID;
    }
    return ix_launch(ref_mz, ref_off, n_ref, n_ref_peaks, q_mz, q_off, n_q, n_q_peaks, scaling, out,
                     ld, device_error, static_cast<unsigned char*>(workspace), (cudaStream_t)stream);
}
