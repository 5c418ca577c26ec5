// cg_small.cuh - the inner CG of one refinement pass in one cooperative launch, for systems
// whose rows fit in the SMs' shared memory.
//
// A small solve is a chain of kernels of 2 to 9 us, five per iteration and each of them all
// latency: launch, ring set-up, last-block reductions (2,000 particles: 29 us per iteration
// for 0.5 MB of rows).  Here a CTA owns consecutive slices for the whole solve: their FP16
// rows are loaded into shared memory once, x, r, p and q of its rows stay there, and an
// iteration has three grid barriers (1.15 us each):
//   q = A p     p_j = z_j + beta p_j is formed as it is gathered ({z, p} in one 8-byte read),
//               so the new direction needs no barrier of its own
//   p.q         -> alpha; x, r of the own rows, r.r, the rows' share of the level-1 residual
//   r.r         -> done?; every CTA adds the shares up and does the coarse correction of its own
//               aggregates: one dense level, or a V-cycle over two (the down sweep over all of
//               level 1 in every CTA, from its stencils in shared memory, which costs less than
//               two more barriers); z
//   z.r         -> beta
// Every CTA adds the CTAs' partial sums in the same order, so all hold the same scalars.
// us, kernel chain -> here: an iteration 29 -> 13 (one coarse level), a step of 2,000 particles
// 1,122 -> 853, of 9,248 (two levels) 1,542 -> 1,219, the Poisson solve of 8,000 particles
// 901 -> 808, of 17,576 1,138 -> 988; then it stops fitting (cg_small_slices_for: with rows of
// 256 entries 24,320 rows for Jacobi or one coarse level, 19,456 with two levels of up to 368
// aggregates; with rows of 240 entries 29,184), so there is no size at which the chain is the
// better one.  What bounds it: the three barriers with
// the partial sums behind them, 2 us each, and one round of gathers from L2.
// The arithmetic per entry and row is the kernel chain's (k_spmv_ring_split, k_cg_update or
// k_mg_update_restrict and k_mg_fine_z, k_cg_p); sums over rows are taken per warp in FP32 and
// above in FP64, as there.
#pragma once

namespace mps {

constexpr int kCgThreads = 256;
constexpr int kCgMaxSlices = 6;      // slices per CTA
constexpr int kCgInv = 16;           // rows of the coarse inverse kept in shared memory
constexpr int kCgAgg = 1024;         // level-1 aggregates at most
struct CgSmall {
    float2* zp;         // [n] z and the last direction
    double* part;       // [4][CTAs] partial sums: p.q, r.r, z.r, z.q
    float* coarse;      // [aggregates + CTAs] share of aggregate I in CTA b at I + b
    unsigned* bar;
    int spc;            // slices per CTA
    int K;              // room for a row's entries, whole chunks
    int levels, flex, maxit;   // levels of the preconditioner: 0 (Jacobi), 1, 2
    double scale, tol;  // r = scale * residual; stop at this norm of r
};
// bytes of shared memory: rows, 5 values per row (x, r, p, q, preconditioner) and its sums per
// warp; per level-1 aggregate its residual, correction, CTAs and, with two levels, stencil
// (values and 16-bit neighbours), residual after the first sweep, diagonal
inline size_t cg_small_smem(int K, int spc, int levels, int n1) {
    return (size_t)spc * K * 128 + (size_t)spc * 32 * (5 + kCgThreads / 32) * 4 +
           (levels ? (size_t)((n1 + 7) & ~7) * (levels > 1 ? 4 * 4 + 4 + 27 * 6 : 3 * 4) : 0);
}

constexpr size_t kCgSmem = 200 * 1024;   // shared memory that the rows can take, beside 25 KB of static arrays
// Slices per CTA for n rows with room for `row` entries each on `sms` SMs, 0: they do not fit.
// A slice with 32-bit columns would be read as empty: with at most 32,768 rows there is none.
inline int cg_small_slices_for(int n, int row, int sms, int levels, int n1) {
    if (n <= 0 || n > 32768 || sms <= 0 || levels > 2 || (levels > 0 && n1 > kCgAgg)) return 0;
    const int spc = div_up(div_up(n, 32), sms);
    return spc <= kCgMaxSlices && cg_small_smem(row, spc, levels, n1) <= kCgSmem ? spc : 0;
}

// The CTAs' partial sums `part` added in order by warp 0; valid in every thread.  SLOT: place
// of the result, reused only after another grid barrier.
template <int SLOT>
__device__ __forceinline__ double cg_total(const double* part) {
    __shared__ double tot;
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) s += __ldcg(part + b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(~0u, s, o);
        if (threadIdx.x == 0) tot = s;
    }
    __syncthreads();
    return tot;
}

__global__ void __launch_bounds__(kCgThreads, 1) k_cg_small(const __grid_constant__ Dev d, const __grid_constant__ Mg mg,
                                                            const __grid_constant__ CgSmall c) {
    constexpr int W = kCgThreads / 32;
    extern __shared__ __align__(16) unsigned char cg_sm[];
    __shared__ int km[kCgMaxSlices];
    __shared__ int agg_lo, agg_hi, nneed;
    __shared__ float ec[kCgMaxSlices * 32];                        // correction of the own aggregates
    __shared__ short seg0[kCgMaxSlices * 32], seg1[kCgMaxSlices * 32];   // their rows in this CTA
    __shared__ float r2[kMgMaxDense], e2[kMgMaxDense];             // last level
    __shared__ short child[kMgMaxDense * 8];                       // level 2: its children
    __shared__ short par[kCgMaxSlices * 32 * 28];                  // own aggregates: parents of the neighbours, own parent
    __shared__ short need[kMgMaxDense];                            // rows of its correction that the CTA reads
    __shared__ float inv[kCgInv][kMgMaxDense];                     // the inverse's rows for the first of them
    __shared__ double psum[2][kCgMaxSlices];
    const int R = c.spc * 32, b = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int sl0 = b * c.spc, row0 = sl0 * 32, nsl = (d.n + 31) >> 5;
    // a slice's c.K x 32 columns and weights
    unsigned* const cols = (unsigned*)cg_sm;
    unsigned* const wts = cols + (size_t)c.spc * c.K * 16;
    float* const sx = (float*)(wts + (size_t)c.spc * c.K * 16);
    float* const sr = sx + R;
    float* const sp = sr + R;
    float* const sq = sp + R;
    float* const sm = sq + R;
    float* const acc = sm + R;   // [W][R]

    // level 1
    const MgLevel& L1 = mg.L[1];
    const MgLevel& L2 = mg.L[2];
    const int na = c.levels ? L1.n : 0, np = (na + 7) & ~7, n2 = c.levels > 1 ? L2.n : 0, nd = n2 ? n2 : na;
    float* const rc = acc + W * R;
    float* const e1 = rc + np;
    short* const cta = (short*)(e1 + np);          // first and last CTA with rows of the aggregate
    float* const res = (float*)(cta + 2 * np);
    float* const dinv = res + np;
    float* const st = dinv + np;                   // [27][np] stencil
    short* const nb = (short*)(st + 27 * np);      // [27][np] neighbour, -1: none
    const float omega = mg.omega;

    if (t < kCgMaxSlices) km[t] = t < c.spc && sl0 + t < nsl ? max(d.skmax[sl0 + t], 0) : 0;
    if (t == 0) {
        agg_lo = kCgAgg;
        agg_hi = -1;
        nneed = 0;
    }
    __syncthreads();
    for (int s = 0; s < c.spc; ++s) {
        const int n16 = ((km[s] + 15) & ~15) * 4;   // 16-byte pieces, rows padded to whole chunks
        const size_t e0 = (size_t)(sl0 + s) * d.K * 32;
        const uint4* const gc = (const uint4*)(d.nbr16 + e0);
        const uint4* const gw = (const uint4*)(d.w16 + e0);
        uint4* const lc = (uint4*)(cols + (size_t)s * c.K * 16);
        uint4* const lw = (uint4*)(wts + (size_t)s * c.K * 16);
        for (int k = t; k < n16; k += kCgThreads) {
            lc[k] = gc[k];
            lw[k] = gw[k];
        }
    }
    // the thread's row (threads below R)
    const int i = row0 + t;
    const bool mine = t < R && i < d.n, in = mine && d.inner[i];
    const int agg = in && c.levels ? mg.agg1[i] : -1;
    const double dg = in ? d.diag16[i] : 0.0;
    if (t < R) {
        sx[t] = sp[t] = sq[t] = 0.f;
        sr[t] = in ? (float)(d.r[i] * c.scale) : 0.f;
        sm[t] = in ? d.m32[i] : 0.f;
    }
    // the CTAs of every aggregate, the aggregates with rows in this one
    for (int I = t; I < na; I += kCgThreads) {
        const int b0 = mg.rb[I], b1 = mg.rb[I + 1];
        cta[2 * I] = (short)(b0 / R);
        cta[2 * I + 1] = (short)((b1 - 1) / R);
        if (b0 < row0 + R && b1 > row0) {
            atomicMin(&agg_lo, I);
            atomicMax(&agg_hi, I);
        }
        if (c.levels > 1) dinv[I] = L1.dinv[I];
    }
    if (c.levels > 1)
        for (int k = t; k < 27 * na; k += kCgThreads) {
            const int I = k / 27, s = k % 27, J = L1.nb[k];
            st[s * np + I] = J >= 0 ? L1.a[k] : 0.f;
            nb[s * np + I] = (short)J;
        }
    for (int k = t; k < nd; k += kCgThreads) need[k] = -1;
    __syncthreads();
    const int own = agg_hi - agg_lo + 1;   // at most R, an aggregate has a row
    for (int k = t; k < own; k += kCgThreads) {
        seg0[k] = (short)(max(mg.rb[agg_lo + k], row0) - row0);
        seg1[k] = (short)(min(mg.rb[agg_lo + k + 1], row0 + R) - row0);
    }
    // rows of the last level's correction that its own aggregates read
    if (c.levels > 1) {
        for (int k = t; k < own * 27; k += kCgThreads) {
            const int e = (agg_lo + k / 27) * 27 + k % 27;
            const int P = L1.nb[e] >= 0 ? L1.nbp[e] : -1;
            par[k / 27 * 28 + k % 27] = (short)P;
            if (P >= 0) need[P] = 1;
        }
        for (int k = t; k < own; k += kCgThreads) {
            const int P = L1.par[agg_lo + k];
            par[k * 28 + 27] = (short)P;
            need[P] = 1;
        }
        for (int k = t; k < n2 * 8; k += kCgThreads) child[k] = (short)L2.child[k];
    } else {
        for (int k = t; k < own; k += kCgThreads) need[agg_lo + k] = 1;
    }
    __syncthreads();
    if (warp == 0) {   // their list
        int n = 0;
        for (int k = 0; k < nd; k += 32) {
            const bool on = k + lane < nd && need[k + lane] > 0;
            const unsigned m = __ballot_sync(~0u, on);
            if (on) need[n + __popc(m & ((1u << lane) - 1u))] = (short)(k + lane);
            n += __popc(m);
            __syncwarp();
        }
        if (lane == 0) nneed = n;
    }
    __syncthreads();
    for (int k = t; k < min(nneed, kCgInv) * nd; k += kCgThreads) inv[k / nd][k % nd] = mg.ainv[need[k / nd] * nd + k % nd];
    float zt = 0.f;   // z of the thread's row

    // sums over the CTA's rows of v0 and v1 (threads below R) into the CTA's places of part
    auto put = [&](float v0, float v1, double* g0, double* g1) {
        if (warp < c.spc) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v0 += __shfl_down_sync(~0u, v0, o);
                v1 += __shfl_down_sync(~0u, v1, o);
            }
            if (lane == 0) {
                psum[0][warp] = (double)v0;
                psum[1][warp] = (double)v1;
            }
        }
        __syncthreads();
        if (t < 2 && (t == 0 || g1)) {
            double s = 0.0;
            for (int k = 0; k < c.spc; ++k) s += psum[t][k];
            (t == 0 ? g0 : g1)[b] = s;
        }
    };
    double* const g_pq = c.part;
    double* const g_rr = g_pq + gridDim.x;
    double* const g_rz = g_rr + gridDim.x;
    double* const g_zq = g_rz + gridDim.x;

    double rz = 0.0, pq = 0.0, r0 = 0.0, rn = 0.0;
    float beta = 0.f;
    int it = 0;
    bool ok = true;
    for (bool first = true;; first = false) {
        if (!first) {
            // ---- q = A p over the rows in shared memory, a warp per chunk of 16 entries
            if (t < R) sp[t] = __fmaf_rn(beta, sp[t], zt);
            for (int s = 0; s < c.spc; ++s) {
                const float2* const zr = c.zp + (sl0 + s) * 32;
                const unsigned* const lc = cols + (size_t)s * c.K * 16;
                const unsigned* const lw = wts + (size_t)s * c.K * 16;
                const int nch = (km[s] + 15) >> 4;
                float a0 = 0.f, a1 = 0.f;   // rows 2 (lane mod 16) and the next, every other entry
#pragma unroll 2
                for (int ch = warp; ch < nch; ch += W) {
                    unsigned cw[8], ww[8];
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        cw[g] = lc[(ch * 8 + g) * 32 + lane];
                        ww[g] = lw[(ch * 8 + g) * 32 + lane];
                    }
                    float2 x0[8], x1[8];
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        x0[g] = zr[(int)(short)(cw[g] & 0xffffu)];
                        x1[g] = zr[(int)cw[g] >> 16];
                    }
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        const float2 wv = __half22float2(*(const __half2*)&ww[g]);
                        a0 = __fmaf_rn(wv.x, __fmaf_rn(beta, x0[g].y, x0[g].x), a0);
                        a1 = __fmaf_rn(wv.y, __fmaf_rn(beta, x1[g].y, x1[g].x), a1);
                    }
                }
                a0 += __shfl_xor_sync(~0u, a0, 16);
                a1 += __shfl_xor_sync(~0u, a1, 16);
                acc[warp * R + s * 32 + 2 * (lane & 15) + (lane >> 4)] = lane < 16 ? a0 : a1;
            }
            __syncthreads();
            float pqv = 0.f;
            if (t < R) {
                float a = 0.f;
#pragma unroll
                for (int w = 0; w < W; ++w) a += acc[w * R + t];
                const float q = in ? (float)(dg * (double)sp[t] - d.c.coef_lap * (double)a) : 0.f;
                sq[t] = q;
                pqv = sp[t] * q;
            }
            put(pqv, 0.f, g_pq, nullptr);
            if (!(ok = coop_barrier(c.bar, d.err))) break;
            pq = cg_total<0>(g_pq);
        }
        // ---- x, r; the share of the level-1 residual
        const float alpha = first ? 0.f : (float)(pq != 0.0 ? rz / pq : 0.0);
        float rrv = 0.f;
        if (t < R) {
            if (in) {
                sx[t] = __fmaf_rn(alpha, sp[t], sx[t]);
                sr[t] = __fmaf_rn(-alpha, sq[t], sr[t]);
            }
            rrv = sr[t] * sr[t];
        }
        put(rrv, 0.f, g_rr, nullptr);   // its barrier: every row of sr is written
        for (int k = warp; k < own; k += W) {
            float s = 0.f;
            for (int j = seg0[k] + lane; j < seg1[k]; j += 32) s += sr[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(~0u, s, o);
            if (lane == 0) c.coarse[agg_lo + k + b] = s;
        }
        if (!(ok = coop_barrier(c.bar, d.err))) break;
        // the aggregates' residuals: their shares in the order of the CTAs
        for (int I = t; I < na; I += kCgThreads) {
            float share = 0.f;
            for (int k = cta[2 * I]; k <= cta[2 * I + 1]; ++k) share += __ldcg(c.coarse + I + k);
            rc[I] = share;
            if (c.levels > 1) e1[I] = omega * dinv[I] * share;
        }
        rn = sqrt(cg_total<1>(g_rr));   // its barrier: rc and e1 are complete
        if (first) r0 = rn;
        else ++it;
        if (rn <= c.tol || it >= c.maxit || !(rn == rn)) break;
        // ---- coarse correction of the own aggregates, z
        if (c.levels > 1) {
            // residual after the first sweep, its sums over the children (octant order)
            for (int I = t; I < na; I += kCgThreads) {
                float v = rc[I];
#pragma unroll
                for (int s = 0; s < 27; ++s) v -= st[s * np + I] * e1[max((int)nb[s * np + I], 0)];
                res[I] = v;
            }
            __syncthreads();
            for (int k = t; k < n2; k += kCgThreads) {
                float v = 0.f;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int I = child[k * 8 + q];
                    if (I >= 0) v += res[I];
                }
                r2[k] = v;
            }
            __syncthreads();
        }
        const float* const rl = c.levels > 1 ? r2 : rc;   // the last level's residual
        for (int k = warp; k < nneed; k += W) {
            const float* const ai = k < kCgInv ? inv[k] : mg.ainv + need[k] * nd;
            float v = 0.f;
            for (int J = lane; J < nd; J += 32) v += ai[J] * rl[J];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
            if (lane == 0) {
                if (c.levels > 1) e2[need[k]] = v;
                else ec[need[k] - agg_lo] = v;
            }
        }
        __syncthreads();
        if (c.levels > 1) {
            for (int k = warp; k < own; k += W) {   // up sweep of the own aggregates
                const int I = agg_lo + k;
                float v = 0.f;
                if (lane < 27) {
                    const int J = nb[lane * np + I];
                    if (J >= 0) v = st[lane * np + I] * (e1[J] + e2[par[k * 28 + lane]]);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
                if (lane == 0) ec[k] = e1[I] + e2[par[k * 28 + 27]] + omega * dinv[I] * (rc[I] - v);
            }
            __syncthreads();
        }
        float rzv = 0.f, zqv = 0.f;
        if (t < R) {
            zt = in ? sm[t] * sr[t] + (agg >= 0 ? ec[agg - agg_lo] : 0.f) : 0.f;
            rzv = sr[t] * zt;
            zqv = zt * sq[t];
            if (mine) c.zp[i] = make_float2(zt, sp[t]);
        }
        put(rzv, zqv, g_rz, c.flex ? g_zq : nullptr);
        if (!(ok = coop_barrier(c.bar, d.err))) break;
        const double rzn = cg_total<2>(g_rz);
        if (first) beta = 0.f;
        else if (c.flex) beta = (float)(pq != 0.0 ? -cg_total<3>(g_zq) / pq : 0.0);
        else beta = (float)(rz != 0.0 ? rzn / rz : 0.0);
        rz = rzn;
    }
    if (mine) d.d32[i] = sx[t];
    if (b == 0 && t == 0) {
        d.scal[S_RZ] = rz;
        d.scal[S_RNORM] = rn;
        d.scal[S_R0NORM] = r0;
        d.scal[S_TOL] = c.tol;
        d.scal[S_MAXIT] = (double)c.maxit;
        d.scal[S_ITER] = ok ? (double)it : -1.0;   // a barrier that ran out: nothing to use
        d.scal[S_CONV] = 1.0;
    }
}

}  // namespace mps
