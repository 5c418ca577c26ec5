// sort.cu - stable LSD radix sort of (int key, int value) pairs on the GPU.
//
// Replaces the reference's thrust::sort_by_key call (SortUsingThrust,
// radix/SPVSOLVER/MultiGPUSolver/DeviceProcess.cu:207-220).  For int keys Thrust's
// sort is a stable radix sort, so the result is uniquely the stable order; this sort
// produces exactly that order.
//
// One cooperative launch (k_sort) does the whole sort: the key range when the caller does
// not know it, then passes of equal digits of at most 9 bits, least significant first.  CTA
// c owns the c-th contiguous part of the keys.  Per pass, with a grid barrier after each
// step:
//   count    each CTA counts its keys' digits (warp-aggregated with __match_any_sync, then
//            shared-memory adds): counts[c][d]
//   prefix   a warp per digit turns counts[.][d] into the exclusive prefix over the CTAs
//            and leaves the digit's total
//   scatter  each CTA scans the totals, ranks its keys stably (warp w owns a contiguous
//            share, 32 keys a round, ranked with __match_any_sync and per-warp running
//            counters) and writes key and value to total prefix + CTA prefix + warp prefix
//            + rank
// Up to 4,096 keys run on one CTA, without barriers.  Keys are sorted as unsigned offsets
// (key - kmin), so negative keys sort correctly and only the bits that the range spans are
// sorted.
//
// What bounds it: latency, of the barriers and of each step's few dependent loads; the keys
// and values stay in L2.  882,080 nearly sorted keys of 17 bits, in us: range 6, then per
// pass count 2.6, prefix 1, scan 0.6, scatter 4.4 and three barriers of 1.2 to 2.2; 34 in
// all (random keys 68: their scatter takes 14, 16,000 keys 21 to 26).  Two CTAs per SM took
// 40 and 72; from 2.5 million keys on they are the faster (us, a call with one / two per SM:
// 2,000,000 nearly sorted 92 / 97, random 226 / 223; 5,000,000 236 / 195 and 467 / 437; 30,000,000
// 1,540 / 1,172 and 2,778 / 2,488).  There a tile's pairs are staged as well: a warp's 32 pairs of
// random keys lay in as many runs, and memory saw a sector for each word, which from 5 million
// keys on was slower than the separate launches of before (us, a call with those / without the
// stage / with it: 3,178,892 random of 30 bits 381 / 356 / 271; 10,000,000 of 24 bits 766 / 932 / 598;
// 30,000,000 of 30 bits 2,644 / 2,876 / 1,787, nearly sorted 1,054 / 1,172 / 1,002).  It replaces three launches per 8-bit pass, 13 to 16 per sort with
// the range's and those of passes beyond the range, which returned at once; finding the
// range alone took 27 us at 882,080 keys (19,456 atomics on one address).
#include <limits.h>

#include <type_traits>

#include "mps_common.cuh"
#include "mps_internal.h"

namespace mps {

constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortRounds = 12;                          // most rounds of 32 keys per warp and tile
constexpr int kSortTile = kSortThreads * kSortRounds;    // most keys of a tile
constexpr int kRadix = 1 << kRadixDigitBits;
constexpr int kSortStage = kSortTile * 2 * (int)sizeof(int);
static_assert(kRadix == kSortThreads, "a thread per digit");

// Exclusive scan of len unsigned values, in place, by one CTA of 1024 threads.
__global__ void __launch_bounds__(1024) k_scan_excl(unsigned* __restrict__ a, int len, unsigned* __restrict__ total) {
    __shared__ unsigned wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = (len + 1023) / 1024;
    const int b = min(len, tid * per), e = min(len, b + per);
    unsigned s = 0;
    for (int i = b; i < e; ++i) s += a[i];
    unsigned inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
        const unsigned x = wsum[lane];
        unsigned xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, xi, o);
            if (lane >= o) xi += v;
        }
        wsum[lane] = xi - x;
        if (lane == 31 && total) *total = xi;
    }
    __syncthreads();
    unsigned run = inc - s + wsum[w];
    for (int i = b; i < e; ++i) {
        const unsigned c = a[i];
        a[i] = run;
        run += c;
    }
}

// Multi-CTA exclusive scan (scan_exclusive with a tile-sum buffer): tiles of
// kScanTile elements loaded coalesced into shared memory; k_scan_tile_sums writes
// each tile's sum, k_scan_tiles scans one tile (4 contiguous items per thread plus
// a block scan of the thread sums) starting from the tile's offset.  The tile sums
// are scanned in place by k_scan_tiles as a single tile.
constexpr int kScanThreads = 1024;
constexpr int kScanTile = 4 * kScanThreads;

__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned* ws, unsigned& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned s = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        ws[lane] = s;
    }
    __syncthreads();
    const unsigned ex = x - v + (w > 0 ? ws[w - 1] : 0u);
    total = ws[31];
    return ex;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(const unsigned* __restrict__ a, int len,
                                                                 unsigned* __restrict__ sums) {
    __shared__ unsigned ws[32];
    const int base = blockIdx.x * kScanTile;
    unsigned s = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = base + q * kScanThreads + threadIdx.x;
        if (i < len) s += a[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned t = ws[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(unsigned* __restrict__ a, int len,
                                                             const unsigned* __restrict__ offsets,
                                                             unsigned* __restrict__ total_dev) {
    __shared__ unsigned t[kScanTile];
    __shared__ unsigned ws[32];
    const int base = blockIdx.x * kScanTile;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = base + q * kScanThreads + threadIdx.x;
        t[q * kScanThreads + threadIdx.x] = i < len ? a[i] : 0u;
    }
    __syncthreads();
    const int o4 = 4 * threadIdx.x;
    const unsigned v0 = t[o4], v1 = t[o4 + 1], v2 = t[o4 + 2], v3 = t[o4 + 3];
    unsigned total;
    const unsigned off = (offsets ? offsets[blockIdx.x] : 0u);
    const unsigned ex = block_exclusive(v0 + v1 + v2 + v3, ws, total) + off;
    t[o4] = ex;
    t[o4 + 1] = ex + v0;
    t[o4 + 2] = ex + v0 + v1;
    t[o4 + 3] = ex + v0 + v1 + v2;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = base + q * kScanThreads + threadIdx.x;
        if (i < len) a[i] = t[q * kScanThreads + threadIdx.x];
    }
    if (total_dev && threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) *total_dev = off + total;
}

// Scratch of a sort: the barrier's word, per-CTA key ranges, digit totals, digit counts
// [CTA][digit], then the alternate key and value arrays.
struct SortScratch {
    unsigned* bar;
    int* range;         // [2][CTAs]
    unsigned* total;    // [kRadix]
    unsigned* counts;   // [CTAs][kRadix]
    int *keys, *vals;   // [n]
};

// bits: the keys lie in [0, 2^bits); < 0: any int range (found first).  STAGED: a tile's pairs go
// through shared memory (kSortStage bytes) in the order of their digits, so that a warp writes
// whole runs
template <bool STAGED>
__global__ void __launch_bounds__(kSortThreads, 2) k_sort(int n, int part, int* keys, int* vals, int bits, SortScratch s,
                                                       unsigned* err, unsigned bit) {
    __shared__ unsigned wcount[kSortWarps][kRadix];
    __shared__ unsigned off[kRadix];
    __shared__ unsigned wsum[32];
    extern __shared__ int staged[];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int c = blockIdx.x, ctas = gridDim.x;
    const int beg = min(n, c * part), end = min(n, beg + part);
    int kmin = 0;
    if (bits < 0) {
        int lo = INT_MAX, hi = INT_MIN;
#pragma unroll 6
        for (int i = beg + tid; i < end; i += kSortThreads) {
            const int k = keys[i];
            lo = min(lo, k);
            hi = max(hi, k);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        int* const r = reinterpret_cast<int*>(wsum);
        if (lane == 0) {
            r[w] = lo;
            r[16 + w] = hi;
        }
        __syncthreads();
        if (w == 0) {
            const int v = r[lane];   // lanes 0..15 minima, 16..31 maxima
            const int l2 = __reduce_min_sync(0xffffffffu, lane < 16 ? v : INT_MAX);
            const int h2 = __reduce_max_sync(0xffffffffu, lane < 16 ? INT_MIN : v);
            if (lane == 0) {
                s.range[c] = l2;
                s.range[ctas + c] = h2;
            }
        }
        if (!coop_barrier(s.bar, err, bit)) return;
        lo = INT_MAX;
        hi = INT_MIN;
        for (int i = lane; i < ctas; i += 32) {
            lo = min(lo, __ldcg(s.range + i));
            hi = max(hi, __ldcg(s.range + ctas + i));
        }
        kmin = __reduce_min_sync(0xffffffffu, lo);
        const unsigned range = (unsigned)__reduce_max_sync(0xffffffffu, hi) - (unsigned)kmin;
        bits = range == 0u ? 0 : 32 - __clz((int)range);
        __syncthreads();
    }
    const int passes = (bits + kRadixDigitBits - 1) / kRadixDigitBits;
    if (passes == 0) return;
    const int dbits = (bits + passes - 1) / passes;
    const unsigned dmask = (1u << dbits) - 1u;
    int *ka = keys, *va = vals, *kb = s.keys, *vb = s.vals;
    for (int pass = 0; pass < passes; ++pass) {
        const int shift = pass * dbits;
        auto digit = [&](int key) { return (((unsigned)key - (unsigned)kmin) >> shift) & dmask; };
        // a part of one tile is loaded once per pass, values included (the other CTAs wrote
        // these pairs in this launch: through L2)
        const bool one = end - beg <= kSortTile;
        int key[kSortRounds], val[kSortRounds];
        auto load = [&](int t0, int tend, int rounds, bool values) {
            const int base = t0 + w * 32 * rounds + lane;
#pragma unroll
            for (int r = 0; r < kSortRounds; ++r) {
                if (r < rounds) {
                    const int i = base + 32 * r;
                    key[r] = i < tend ? __ldcg(ka + i) : 0;
                    if (values) val[r] = i < tend ? __ldcg(va + i) : 0;
                }
            }
        };
        // ---- count ----
        off[tid] = 0;
        __syncthreads();
        for (int t0 = beg; t0 < end; t0 += kSortTile) {
            const int tend = min(end, t0 + kSortTile);
            const int rounds = (tend - t0 + kSortThreads - 1) / kSortThreads;   // of 32 keys per warp
            load(t0, tend, rounds, one);
#pragma unroll
            for (int r = 0; r < kSortRounds; ++r) {
                if (r < rounds) {
                    const bool ok = t0 + w * 32 * rounds + lane + 32 * r < tend;
                    const unsigned d = ok ? digit(key[r]) : (unsigned)kRadix;
                    const unsigned peers = __match_any_sync(0xffffffffu, d);
                    if (ok && (peers & lt) == 0) atomicAdd(&off[d], (unsigned)__popc(peers));
                }
            }
        }
        __syncthreads();
        const unsigned mine = off[tid];
        if (ctas > 1) {
            s.counts[(size_t)c * kRadix + tid] = mine;
            if (!coop_barrier(s.bar, err, bit)) return;
            // ---- prefix over the CTAs, a warp per digit, a run of CTAs per lane ----
            auto prefix = [&](auto run_of) {
                constexpr int kRun = run_of.value;
                for (int d = w * ctas + c; d < kRadix; d += ctas * kSortWarps) {   // spread over the SMs
                    unsigned x[kRun], sum = 0;
#pragma unroll
                    for (int q = 0; q < kRun; ++q) {
                        const int k = lane * kRun + q;
                        x[q] = k < ctas ? __ldcg(s.counts + (size_t)k * kRadix + d) : 0u;
                    }
#pragma unroll
                    for (int q = 0; q < kRun; ++q) sum += x[q];
                    unsigned inc = sum;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
                        if (lane >= o) inc += v;
                    }
                    unsigned run = inc - sum;
#pragma unroll
                    for (int q = 0; q < kRun; ++q) {
                        const int k = lane * kRun + q;
                        if (k < ctas) s.counts[(size_t)k * kRadix + d] = run;
                        run += x[q];
                    }
                    if (lane == 31) s.total[d] = inc;
                }
            };
            constexpr int kHalf = (kRadixMaxCtas / 2 + 31) / 32;
            if (ctas <= kRadixMaxCtas / 2) prefix(std::integral_constant<int, kHalf>());
            else prefix(std::integral_constant<int, 2 * kHalf>());
            if (!coop_barrier(s.bar, err, bit)) return;
        }
        // exclusive sum of the threads' x (in the order of the digits)
        auto below = [&](unsigned x) {
            unsigned inc = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (lane == 31) wsum[w] = inc;
            __syncthreads();
            if (w == 0) {
                const unsigned y = lane < kSortWarps ? wsum[lane] : 0u;
                unsigned yi = y;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned v = __shfl_up_sync(0xffffffffu, yi, o);
                    if (lane >= o) yi += v;
                }
                wsum[lane] = yi - y;
            }
            __syncthreads();
            return inc - x + wsum[w];
        };
        // ---- first position of each digit's keys of this CTA ----
        {
            const unsigned total = ctas > 1 ? __ldcg(s.total + tid) : mine;
            const unsigned before = ctas > 1 ? __ldcg(s.counts + (size_t)c * kRadix + tid) : 0u;
            off[tid] = below(total) + before;
        }
        // ---- scatter ----
        for (int t0 = beg; t0 < end; t0 += kSortTile) {
            const int tend = min(end, t0 + kSortTile);
            const int rounds = (tend - t0 + kSortThreads - 1) / kSortThreads;   // of 32 keys per warp
            for (int q = 0; q < kSortWarps; ++q) wcount[q][tid] = 0;
            __syncthreads();
            const int base = t0 + w * 32 * rounds + lane;
            if (!one) load(t0, tend, rounds, true);
            unsigned at[kSortRounds];   // digit | rank << 10
#pragma unroll
            for (int r = 0; r < kSortRounds; ++r) {
                if (r < rounds) {
                    const bool ok = base + 32 * r < tend;
                    const unsigned d = ok ? digit(key[r]) : (unsigned)kRadix;
                    const unsigned peers = __match_any_sync(0xffffffffu, d);
                    const unsigned lower = peers & lt;
                    const unsigned seen = ok ? wcount[w][d] : 0u;
                    __syncwarp();
                    if (ok && lower == 0) wcount[w][d] = seen + (unsigned)__popc(peers);
                    __syncwarp();
                    at[r] = d | (seen + (unsigned)__popc(lower)) << 10;
                }
            }
            __syncthreads();
            if constexpr (STAGED) {
                int* const tkey = staged;
                int* const tval = staged + kSortTile;
                unsigned tile = 0;
#pragma unroll
                for (int q = 0; q < kSortWarps; ++q) tile += wcount[q][tid];
                const unsigned first = below(tile);   // of the digit's pairs in the tile
                unsigned run = first;
#pragma unroll
                for (int q = 0; q < kSortWarps; ++q) {
                    const unsigned x = wcount[q][tid];
                    wcount[q][tid] = run;
                    run += x;
                }
                const unsigned next = off[tid] + tile;
                off[tid] -= first;   // place in the tile -> position
                __syncthreads();
#pragma unroll
                for (int r = 0; r < kSortRounds; ++r) {
                    if (r < rounds) {
                        const unsigned d = at[r] & 1023u;
                        if (d < (unsigned)kRadix) {
                            const unsigned u = wcount[w][d] + (at[r] >> 10);
                            tkey[u] = key[r];
                            tval[u] = val[r];
                        }
                    }
                }
                __syncthreads();
#pragma unroll 4
                for (int u = tid; u < tend - t0; u += kSortThreads) {
                    const int k = tkey[u];
                    const unsigned dst = off[digit(k)] + (unsigned)u;
                    if (dst < (unsigned)n) {   // not where another CTA gave up at a barrier
                        kb[dst] = k;
                        vb[dst] = tval[u];
                    }
                }
                __syncthreads();
                off[tid] = next;   // the next tile's first positions
            } else {
                unsigned run = off[tid];
#pragma unroll
                for (int q = 0; q < kSortWarps; ++q) {
                    const unsigned x = wcount[q][tid];
                    wcount[q][tid] = run;
                    run += x;
                }
                off[tid] = run;   // the next tile's first positions
                __syncthreads();
#pragma unroll
                for (int r = 0; r < kSortRounds; ++r) {
                    if (r < rounds) {
                        const unsigned d = at[r] & 1023u;
                        if (d < (unsigned)kRadix) {
                            const unsigned dst = wcount[w][d] + (at[r] >> 10);
                            if (dst < (unsigned)n) {   // not where another CTA gave up at a barrier
                                kb[dst] = key[r];
                                vb[dst] = val[r];
                            }
                        }
                    }
                }
                __syncthreads();
            }
        }
        if (!coop_barrier(s.bar, err, bit)) return;
        int* t = ka; ka = kb; kb = t;
        t = va; va = vb; vb = t;
    }
    if (ka != keys) {
        for (int i = beg + tid; i < end; i += kSortThreads) {
            keys[i] = __ldcg(ka + i);
            vals[i] = __ldcg(va + i);
        }
    }
}

cudaError_t sort_barrier_polls(int polls) { return cudaMemcpyToSymbol(c_coop_polls, &polls, sizeof(polls)); }

int radix_bits(unsigned range) {
    int bits = 0;
    while (bits < 32 && (range >> bits) != 0u) ++bits;
    return bits;
}

cudaError_t radix_sort_pairs(int n, int* keys, int* vals, int bits, void* scratch, unsigned* err, unsigned bit,
                             cudaStream_t st, int max_ctas) {
    if (n <= 1 || bits == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // all resident on the whole GPU; a stream or context with a part of its SMs refuses such a
    // launch and gets half as many until one fits.  One CTA has no barriers and is an
    // ordinary launch.
    for (int most = max(1, min(min(max_ctas, radix_ctas_for(n)), n < kRadixTwoPerSm ? sms : 2 * sms));; most /= 2) {
        int part = div_up(n, most);
        part = (part + kSortThreads - 1) / kSortThreads * kSortThreads;
        const int ctas = div_up(n, part);
        SortScratch s;
        unsigned* p = (unsigned*)scratch;
        s.bar = p;
        s.range = (int*)(p + 8);
        s.total = p + 8 + 2 * ctas;
        s.counts = s.total + kRadix;
        s.keys = (int*)(s.counts + (size_t)ctas * kRadix);
        s.vals = s.keys + n;
        if (ctas == 1) {
            MPS_COUNT_LAUNCH k_sort<false><<<1, kSortThreads, 0, st>>>(n, part, keys, vals, bits, s, err, bit);
            return cudaGetLastError();
        }
        cudaError_t e = cudaMemsetAsync(s.bar, 0, sizeof(unsigned), st);
        if (e) return e;
        void* args[] = {(void*)&n, (void*)&part, (void*)&keys, (void*)&vals, (void*)&bits, (void*)&s, (void*)&err, (void*)&bit};
        const bool staged = n >= kRadixTwoPerSm;
        const void* const kernel = staged ? (const void*)k_sort<true> : (const void*)k_sort<false>;
        if (staged && (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortStage))) return e;
        e = cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(kSortThreads), args, staged ? kSortStage : 0, st);
        if (e == cudaSuccess) MPS_COUNT_LAUNCH 0;
        if (!coop_refused(e)) return e;
        if (e == cudaErrorNotSupported) most = 2;   // one CTA next
    }
}

cudaError_t scan_exclusive(unsigned* a, int len, unsigned* total_dev, cudaStream_t st, unsigned* tile_sums) {
    if (len <= 0) return cudaSuccess;
    const int tiles = (len + kScanTile - 1) / kScanTile;
    if (tiles == 1) {
        MPS_COUNT_LAUNCH k_scan_tiles<<<1, kScanThreads, 0, st>>>(a, len, nullptr, total_dev);
    } else if (tile_sums && tiles <= kScanTile) {
        MPS_COUNT_LAUNCH k_scan_tile_sums<<<tiles, kScanThreads, 0, st>>>(a, len, tile_sums);
        MPS_COUNT_LAUNCH k_scan_tiles<<<1, kScanThreads, 0, st>>>(tile_sums, tiles, nullptr, nullptr);
        MPS_COUNT_LAUNCH k_scan_tiles<<<tiles, kScanThreads, 0, st>>>(a, len, tile_sums, total_dev);
    } else {
        MPS_COUNT_LAUNCH k_scan_excl<<<1, 1024, 0, st>>>(a, len, total_dev);
    }
    return cudaGetLastError();
}

size_t scan_tile_sums_capacity() { return (size_t)kScanTile; }

}  // namespace mps
