// ref_pairs.cuh - the pair sums of the reference-named particle operators.
//
// Include only from ref_kernels.cu (compiled without multiply-add contraction): the
// sums below are the reference's, term by term and in its order (cells k outer, j, i
// inner; a cell's particles in sorted order), so they round as its serial loops do.
//
// A warp owns T consecutive targets of the sorted order (mostly one cell's) and walks
// the candidates of their 27 cells once for all of them:
//   screen  32 candidates a round, a lane each; per target one squared distance, one
//           ballot, and the accepted candidates appended to the target's queue in
//           shared memory (rank within the ballot = traversal order);
//   terms   when a queue could overflow: a lane per queued pair, so the square root,
//           divisions and gathers run with full warps instead of under the union of 32
//           targets' accepts;
//   sums    a lane per (component, target) adds the queued terms one after another.
// Adding +0 for a pair that the exact test then rejects leaves a sum's bits alone: a
// sum that starts at +0 never becomes -0.
//
// What bounds it: instruction issue (per target about 560 warp instructions to walk the
// cells, 17 per round of 32 candidates screened, 64 to 90 per 32 accepted pairs), the
// screen's votes and population counts first.  A thread per target over global memory,
// which this replaces, ran the terms of every candidate that any of its warp's 32 targets
// accepted and left most of the chip idle below 100k particles.  Measured in us, before
// and after: 15,625 particles pressure 312 / 50, heat 324 / 53, turbulence 414 / 62,
// predictor 531 / 94; 103,823 pressure 334 / 137, gradient 462 / 177; 884,736 pressure
// 1,520 / 1,160, gradient 2,450 / 1,406 (from 40,000 particles on RpSlice takes over these).
// In sparse fluid there is little to share; a lane per target is faster there (rp_walk_sums).
#pragma once

namespace mps {

constexpr int kRpWarps = 4;        // warps per CTA
constexpr int kRpCap = 64;         // queue entries per target: a round adds at most 32 to at most 32
constexpr int kRpStride = 68;      // floats per queue row: 16-byte aligned, 17 16-byte units (odd: no bank conflicts)
constexpr float kRpHuge = 1e18f;   // coordinates above it can overflow a squared distance

// what a target brings to its pair terms
struct RpTarget {
    Scalar3 pos;
    Scalar3 vel;
    float s;      // scalar of the operator (pressure, temperature, strain)
};

// ---- operators: NS sums per target, NX sums over rarer pairs, terms and scalars ----
struct RpExplicitly {
    static constexpr int NS = 3, NX = 9;
    static constexpr bool kIndex = true;   // its terms read the candidate
    static constexpr bool kLe = false, kPos = false, kVel = true, kScalar = false;
    static __device__ __forceinline__ void terms(const RefBind& b, float re, const RpTarget& t, int x, float d,
                                                 float (&v)[NS]) {
        const float w = weight(re, d);
        const Scalar3 v1 = b.vel[x];
        v[0] = (v1.x - t.vel.x) * w;
        v[1] = (v1.y - t.vel.y) * w;
        v[2] = (v1.z - t.vel.z) * w;
    }
    // largest distance of a pair with a part in the other sums
    static __device__ __forceinline__ float rare_radius(const CParameter& P) {
        const float rc = P.r_coeff * P.InitialParticleDistance;
        const float reg = P.GradientInfluenceRadiusCoefficient * P.InitialParticleDistance;
        return fmaxf(P.bExplicitPressure ? rc : 0.0f, P.bTurbulance ? reg : 0.0f);
    }
    static __device__ __forceinline__ void rare_terms(const RefBind& b, float re, const RpTarget& t, int x, float d,
                                                      float (&ex)[NX]) {
        const CParameter& P = b.param;
        const float rc = P.r_coeff * P.InitialParticleDistance;
        const float reg = P.GradientInfluenceRadiusCoefficient * P.InitialParticleDistance;
        const Scalar3 dq = s3sub(b.pos[x], t.pos);
#pragma unroll
        for (int c = 0; c < NX; ++c) ex[c] = 0.0f;
        if (P.bExplicitPressure && d < rc) {
            const Scalar3 a = s3mul(dq, P.ArtificialPressure * weight(re, d) / (d * d)), c = s3mul(dq, (rc - d) / d);
            ex[0] = a.x; ex[1] = a.y; ex[2] = a.z;
            ex[3] = c.x; ex[4] = c.y; ex[5] = c.z;
        }
        if (P.bTurbulance && d < reg) {   // turbulent kinetic energy gradient (:477-485)
            const Scalar3 k = s3mul(dq, (b.strain[x] - t.s) * weight(reg, d) / (d * d));
            ex[6] = k.x; ex[7] = k.y; ex[8] = k.z;
        }
    }
};
struct RpPressure {
    static constexpr int NS = 1, NX = 0;
    static constexpr bool kIndex = false;
    static constexpr bool kLe = false, kPos = false, kVel = false, kScalar = false;
    static __device__ __forceinline__ void terms(const RefBind&, float re, const RpTarget&, int, float d,
                                                 float (&v)[NS]) {
        v[0] = weight(re, d);
    }
};
struct RpGradient {
    static constexpr int NS = 3, NX = 0;
    static constexpr bool kIndex = true;
    static constexpr bool kLe = false, kPos = true, kVel = false, kScalar = true;
    static __device__ __forceinline__ void terms(const RefBind& b, float re, const RpTarget& t, int x, float d,
                                                 float (&v)[NS]) {
        const Scalar3 q = b.pos[x];
        const float s = b.pressure[x] + t.s, w = weight(re, d);
        // the reference's (float)(0.5 * (double)s * (double)w): the double product is
        // exact, so one float multiplication rounds alike wherever 0.5 s is exact
        const float pc = (fabsf(s) < 1e-30f && s != 0.0f) ? (float)(0.5 * (double)s * (double)w) : (0.5f * s) * w;
        v[0] = pc * (q.x - t.pos.x) / (d * d);
        v[1] = pc * (q.y - t.pos.y) / (d * d);
        v[2] = pc * (q.z - t.pos.z) / (d * d);
    }
};
struct RpTemperature {
    static constexpr int NS = 1, NX = 0;
    static constexpr bool kIndex = true;
    static constexpr bool kLe = true, kPos = false, kVel = false, kScalar = true;
    static __device__ __forceinline__ void terms(const RefBind& b, float re, const RpTarget& t, int x, float d,
                                                 float (&v)[NS]) {
        const CParameter& P = b.param;
        const float num = (b.temperature[x] - t.s) * weight(re, d);
        const float den = d * d * (1 / P.FruidThermalConductivity + P.FruidThermalResistance / d);
        v[0] = num / den;
    }
};
struct RpTurbulence {
    static constexpr int NS = 9, NX = 0;
    static constexpr bool kLe = false, kPos = true, kVel = true, kScalar = false;
    static __device__ __forceinline__ void terms(const RefBind& b, float re, const RpTarget& t, int x, float d,
                                                 float (&v)[NS]) {
        const Scalar3 q = b.pos[x], v1 = b.vel[x];
        const float w = weight(re, d), d2 = d * d;
        const float du[3] = {v1.x - t.vel.x, v1.y - t.vel.y, v1.z - t.vel.z};
        const float dx[3] = {q.x - t.pos.x, q.y - t.pos.y, q.z - t.pos.z};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int c = 0; c < 3; ++c) v[3 * a + c] = (du[a] * dx[c] * w) / d2;
    }
};

// two single-precision lanes per instruction, each rounded as the scalar operation
__device__ __forceinline__ unsigned long long rp_pack(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void rp_unpack(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long rp_add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * b as a * b + (-0), which rounds alike (and keeps the product's sign of zero).  ptxas
// fuses a packed multiplication into a packed addition that follows it, whatever the
// rounding modifiers and -fmad say, so nz = (-0, -0) has to come from the kernel's
// arguments: a constant is folded away and the sum is fused all the same.
__device__ __forceinline__ unsigned long long rp_mul2(unsigned long long a, unsigned long long b, unsigned long long nz) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
    return r;
}

template <class Op>
struct RpShape {
    static constexpr int NP = Op::NS > 2 ? Op::NS : 2;   // queue planes: squared distance and index, then terms
    static constexpr int NXR = Op::NX > 0 ? Op::NX : 1;
};

// Pair sums of one warp's T targets.  Lane t < T holds target t (id = first + t): `live`,
// its position and cell, its RpTarget.  Returns in lane t the NS sums and NX sums.
template <class Op, int T>
struct RpWarp {
    static constexpr int NS = Op::NS, NX = Op::NX, NP = RpShape<Op>::NP, NXR = RpShape<Op>::NXR;
    static constexpr int kQueue = NP * T * kRpStride;
    // rarer pairs: sums of every target, then a queue of 64 (distance, index, target),
    // whose first rows take the terms of 32 pairs
    static constexpr int kRare = NX > 0 ? NX * T + 3 * 64 + NX * 32 : 0;
    static constexpr int kFloats = kQueue + ((kRare + T + 3) & ~3);   // shared memory of a warp
    static constexpr int NA = (NS * T + 31) / 32;                 // sums held per lane

    float* sm;
    float re, re2x, mind;
    unsigned long long nz2;   // (-0, -0), see rp_mul2
    int lane, first;
    RpTarget me;        // lane t: target t
    unsigned long long tx[T / 2], ty[T / 2], tz[T / 2];   // the group's targets, two a register pair
    int cnt[T];
    int rcnt;            // pairs in the queue of rarer pairs
    float rare_re;
    float acc[NA];

    __device__ __forceinline__ RpWarp(const RefBind& b, float* smem, float radius, float minus_zero, int first_id, const RpTarget& t)
        : sm(smem), re(radius), re2x(ref_screen2(radius)), mind((float)(radius * 1e-3)),
          nz2(rp_pack(minus_zero, minus_zero)),
          lane(threadIdx.x & 31), first(first_id), me(t) {
#pragma unroll
        for (int t_ = 0; t_ < T; ++t_) cnt[t_] = 0;
#pragma unroll
        for (int a = 0; a < NA; ++a) acc[a] = 0.0f;
        if constexpr (NX > 0) {
            for (int i = lane; i < NX * T; i += 32) sm[kQueue + i] = 0.0f;
        }
        rcnt = 0;
        rare_re = 0.0f;
        if constexpr (NX > 0) rare_re = Op::rare_radius(b.param);
        __syncwarp();
    }

    // candidate x of each lane against the targets of `um` (two at a time), the accepted
    // ones queued; the target itself is dropped with the exact test
    __device__ __forceinline__ void screen(int x, const Scalar3& q, unsigned um) {
        const unsigned lt = (1u << lane) - 1u;
        const unsigned long long nx = rp_pack(-q.x, -q.x), ny = rp_pack(-q.y, -q.y), nz = rp_pack(-q.z, -q.z);
        constexpr int Q = 2;
#pragma unroll
        for (int t0 = 0; t0 < T; t0 += Q) {
            if (!(um >> t0 & ((1u << Q) - 1u))) continue;
            float d2[Q];
#pragma unroll
            for (int h = 0; h < Q; h += 2) {
                const int p = (t0 + h) / 2;
                const unsigned long long dx = rp_add2(tx[p], nx), dy = rp_add2(ty[p], ny), dz = rp_add2(tz[p], nz);
                rp_unpack(rp_add2(rp_add2(rp_mul2(dx, dx, nz2), rp_mul2(dy, dy, nz2)), rp_mul2(dz, dz, nz2)), d2[h],
                          d2[h + 1]);
            }
            unsigned m[Q];
#pragma unroll
            for (int h = 0; h < Q; ++h) m[h] = __ballot_sync(~0u, d2[h] < re2x);
#pragma unroll
            for (int h = 0; h < Q; ++h) {
                const int t = t0 + h;
                if (d2[h] < re2x) {
                    float* const row = sm + t * kRpStride + cnt[t] + __popc(m[h] & lt);
                    row[0] = d2[h];
                    row[T * kRpStride] = __int_as_float(x);
                }
                cnt[t] += __popc(m[h]);
            }
        }
    }
    // the same against all of the group where a squared distance may overflow (the
    // reference accepts an infinite one)
    __device__ __forceinline__ void screen_all(int x, const Scalar3& q, unsigned grp) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const float dx = __shfl_sync(~0u, me.pos.x, t) - q.x, dy = __shfl_sync(~0u, me.pos.y, t) - q.y,
                        dz = __shfl_sync(~0u, me.pos.z, t) - q.z;
            const float d2 = dx * dx + dy * dy + dz * dz;
            const bool hit = (grp >> t & 1u) && !(d2 >= re2x && d2 <= 3.402823466e38f);
            const unsigned m = __ballot_sync(~0u, hit);
            if (hit) {
                float* const row = sm + t * kRpStride + cnt[t] + __popc(m & ((1u << lane) - 1u));
                row[0] = d2;
                row[T * kRpStride] = __int_as_float(x);
            }
            cnt[t] += __popc(m);
        }
    }

    // Rarer pairs: a lane per pair computes the terms, then a lane per sum adds them in
    // the order the pairs were queued.  Empties the queue (at most 64 pairs).
    __device__ __forceinline__ void flush_rare(const RefBind& b) {
        if constexpr (NX > 0) {
            float* const xsum = sm + kQueue;
            float* const q = xsum + NX * T;
            float* const rows = q + 3 * 64;
            __syncwarp();
#pragma unroll 1
            for (int e0 = 0; e0 < rcnt; e0 += 32) {
                const int e = e0 + lane, k = min(rcnt - e0, 32);
                const int t = lane < k ? __float_as_int(q[128 + e]) : 0;
                RpTarget g;
                g.pos.x = __shfl_sync(~0u, me.pos.x, t);
                g.pos.y = __shfl_sync(~0u, me.pos.y, t);
                g.pos.z = __shfl_sync(~0u, me.pos.z, t);
                g.s = __shfl_sync(~0u, me.s, t);
                if (lane < k) {
                    float ex[NXR];
                    Op::rare_terms(b, re, g, __float_as_int(q[64 + e]), q[e], ex);
#pragma unroll
                    for (int c = 0; c < NX; ++c) rows[lane * NX + c] = ex[c];
                }
                __syncwarp();
                if (lane < NX)
                    for (int r = 0; r < k; ++r) {
                        float* const s = xsum + __float_as_int(q[128 + e0 + r]) * NX + lane;
                        *s = *s + rows[r * NX + lane];
                    }
                __syncwarp();
            }
            rcnt = 0;
        }
    }

    // queued pairs -> terms -> sums; empties the queues
    __device__ __forceinline__ void flush(const RefBind& b) {
        // entries of target t to lane t (through shared memory: selecting them by lane
        // would put the counts into local memory)
        int* const scnt = reinterpret_cast<int*>(sm + kQueue + kRare);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            if (lane == 0) scnt[t] = cnt[t];
            cnt[t] = 0;
        }
        __syncwarp();
        const int mine = lane < T ? scnt[lane] : 0;
        // the queues as one sequence, target by target, 32 pairs a round
        int end = mine;
#pragma unroll
        for (int o = 1; o < T; o <<= 1) {
            const int v = __shfl_up_sync(~0u, end, o);
            if (lane >= o) end += v;
        }
        const int total = __shfl_sync(~0u, end, T - 1), start = lane < T ? end - mine : 0x7fffffff;
#pragma unroll 1
        for (int e0 = 0; e0 < total; e0 += 32) {
            const int e = e0 + lane;
            int t = 0;   // the last target whose pairs start at or before e
#pragma unroll
            for (int o = T / 2; o > 0; o >>= 1) {
                const int v = __shfl_sync(~0u, start, t + o);
                if (v <= e) t += o;
            }
            float* const row = sm + t * kRpStride + (e - __shfl_sync(~0u, start, t));
            RpTarget g;
            if constexpr (Op::kPos) {
                g.pos.x = __shfl_sync(~0u, me.pos.x, t);
                g.pos.y = __shfl_sync(~0u, me.pos.y, t);
                g.pos.z = __shfl_sync(~0u, me.pos.z, t);
            }
            if constexpr (Op::kVel) {
                g.vel.x = __shfl_sync(~0u, me.vel.x, t);
                g.vel.y = __shfl_sync(~0u, me.vel.y, t);
                g.vel.z = __shfl_sync(~0u, me.vel.z, t);
            }
            if constexpr (Op::kScalar) g.s = __shfl_sync(~0u, me.s, t);
            bool rare = false;
            float d = 0.0f;
            int x = 0;
            if (e < total) {
                float v[NS];
#pragma unroll
                for (int c = 0; c < NS; ++c) v[c] = 0.0f;
                x = __float_as_int(row[T * kRpStride]);
                d = ref_sqrt(row[0]);
                const bool ok = (Op::kLe ? d <= re : d < re) && x != first + t;
                if (d < mind) d = mind;
                if (ok) Op::terms(b, re, g, x, d, v);
                if constexpr (NX > 0) rare = ok && d < rare_re;
#pragma unroll
                for (int c = 0; c < NS; ++c) row[c * T * kRpStride] = v[c];
            }
            if constexpr (NX > 0) {
                const unsigned m = __ballot_sync(~0u, rare);
                if (m) {
                    float* const q = sm + kQueue + NX * T + rcnt + __popc(m & ((1u << lane) - 1u));
                    if (rare) {
                        q[0] = d;
                        q[64] = __int_as_float(x);
                        q[128] = __int_as_float(t);
                    }
                    rcnt += __popc(m);
                    if (rcnt > 32) flush_rare(b);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int l = a * 32 + lane, t = l % T;
            const int n = __shfl_sync(~0u, mine, t);
            if (l < NS * T) {
                const float* const row = sm + ((l / T) * T + t) * kRpStride;
                float s = acc[a];
                int e = 0;
                for (; e + 4 <= n; e += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(row + e);
                    s += v.x;
                    s += v.y;
                    s += v.z;
                    s += v.w;
                }
                for (; e < n; ++e) s += row[e];
                acc[a] = s;
            }
        }
        __syncwarp();
    }

    // bounds of the coordinates that truncate toward zero to cell index c
    static __device__ __forceinline__ float low(int c, float cs) { return (float)(c <= 0 ? c - 1 : c) * cs; }
    static __device__ __forceinline__ float high(int c, float cs) { return (float)(c >= 0 ? c + 1 : c) * cs; }

    // position of candidate x < e (NaN, which no test accepts, where there is none)
    static __device__ __forceinline__ Scalar3 fetch(const RefBind& b, int x, int e) {
        const float nan = __int_as_float(0x7fffffff);
        Scalar3 q = s3(nan, nan, nan);
        if (x < e && b.out_id[x] >= 0) q = b.pos[x];
        return q;
    }

    // Candidates of the targets `grp`, all in cell (cx, cy, cz).
    __device__ __forceinline__ void walk(const RefBind& b, unsigned grp, int cx, int cy, int cz) {
        const Integer3 G = b.box.m_GridSize;
        const float cs = b.box.m_CellSize;
        // lane m < 27: cell m of the traversal (k outer, j, i inner)
        int s = 0, len = 0;
        unsigned mask = 0;
        const int i = lane % 3 - 1, j = (lane / 3) % 3 - 1, k = lane / 9 - 1;
        if (grp && lane < 27) {
            const int m = cell_key(G, (int)((unsigned)cx + (unsigned)i), (int)((unsigned)cy + (unsigned)j),
                                   (int)((unsigned)cz + (unsigned)k));
            if (m >= 0 && m < b.cell_num) {
                s = b.cell_start[m];
                if (s != -1) len = max(b.cell_end[m] - s, 0);
            }
            mask = grp;
        }
        // Targets that can have a neighbour in the cell: those within re of its box.  A
        // particle within re <= cell size of a target lies in the box of the cell that its
        // own indices give (ref_cell truncates toward zero, the box is widened by the
        // rounding of that), and with at least 4 cells along y and z no other of the 27
        // offsets shares that cell's key; elsewhere every target is tested.
        const bool cull = G.y >= 4 && G.z >= 4 && re <= cs * 1.0001f && max(abs(cx), max(abs(cy), abs(cz))) < (1 << 20);
        if (cull) {
            const Scalar3 lo = b.box.m_BufferedZone.m_MinBound;
            const float pad = cs * (1e-3f + 1e-6f * (float)(max(cx, max(cy, cz)) + 2));
            const float x0 = low(cx + i, cs) - pad, x1 = high(cx + i, cs) + pad, y0 = low(cy + j, cs) - pad;
            const float y1 = high(cy + j, cs) + pad, z0 = low(cz + k, cs) - pad, z1 = high(cz + k, cs) + pad;
            unsigned near = 0;
#pragma unroll 1
            for (int t = 0; t < T; ++t) {
                const float px = __shfl_sync(~0u, me.pos.x, t) - lo.x, py = __shfl_sync(~0u, me.pos.y, t) - lo.y,
                            pz = __shfl_sync(~0u, me.pos.z, t) - lo.z;
                const float ax = fmaxf(0.0f, fmaxf(x0 - px, px - x1)), ay = fmaxf(0.0f, fmaxf(y0 - py, py - y1)),
                            az = fmaxf(0.0f, fmaxf(z0 - pz, pz - z1));
                if (!(ax * ax + ay * ay + az * az > re2x)) near |= 1u << t;
            }
            mask &= near;
        }
        const bool far_target = __any_sync(~0u, lane < T && (grp >> lane & 1u) &&
                                                    fmaxf(fabsf(me.pos.x), fmaxf(fabsf(me.pos.y), fabsf(me.pos.z))) > kRpHuge);
        // targets of other cells: NaN, which no screen accepts
        const float nan = __int_as_float(0x7fffffff);
        const bool mine = lane < T && (grp >> lane & 1u);
        const Scalar3 tp = mine ? me.pos : s3(nan, nan, nan);
#pragma unroll
        for (int p = 0; p < T / 2; ++p) {
            tx[p] = rp_pack(__shfl_sync(~0u, tp.x, 2 * p), __shfl_sync(~0u, tp.x, 2 * p + 1));
            ty[p] = rp_pack(__shfl_sync(~0u, tp.y, 2 * p), __shfl_sync(~0u, tp.y, 2 * p + 1));
            tz[p] = rp_pack(__shfl_sync(~0u, tp.z, 2 * p), __shfl_sync(~0u, tp.z, 2 * p + 1));
        }
        // non-empty cells in order; after the last group one empty round, which flushes
        // what is queued
        unsigned cells = grp ? __ballot_sync(~0u, len > 0) : 1u;
        const int limit = grp ? kRpCap - 32 : 0;
        while (cells) {
            const int m = __ffs(cells) - 1;
            cells &= cells - 1u;
            const int s0 = __shfl_sync(~0u, s, m), e = s0 + __shfl_sync(~0u, len, m);
            const unsigned um = __shfl_sync(~0u, mask, m);
            int x = s0 + lane;
            Scalar3 q = fetch(b, x, e), qn;
#pragma unroll 1
            for (int r = s0;;) {
                r += 32;
                const bool more = r < e;
                if (more) qn = fetch(b, x + 32, e);   // the next round's, before this one is screened
                const bool huge = fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))) > kRpHuge;
                if (far_target || __any_sync(~0u, huge)) screen_all(x, q, grp);
                else if (um) screen(x, q, um);
                int most = 0;
#pragma unroll
                for (int t = 0; t < T; ++t) most = max(most, cnt[t]);
                if (most > limit) flush(b);
                if (!more) break;
                q = qn;
                x += 32;
            }
        }
    }

    // all targets of the warp: `live` in lane t, its cell in (cx, cy, cz)
    __device__ __forceinline__ void run(const RefBind& b, bool live, int cx, int cy, int cz) {
        unsigned todo = __ballot_sync(~0u, live), grp = todo;
        while (grp) {
            const int l = todo ? __ffs(todo) - 1 : 0;
            const int gx = __shfl_sync(~0u, cx, l), gy = __shfl_sync(~0u, cy, l), gz = __shfl_sync(~0u, cz, l);
            grp = __ballot_sync(~0u, live && cx == gx && cy == gy && cz == gz) & todo;
            walk(b, grp, gx, gy, gz);
            todo &= ~grp;
        }
        flush_rare(b);
    }
    // sum c of this lane's target (lanes t < T; every lane calls it)
    __device__ __forceinline__ float sum(int c) const {
        const int l = c * T + (lane < T ? lane : 0);
        float r = 0.0f;
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const float v = __shfl_sync(~0u, acc[a], l & 31);
            r = (l >> 5) == a ? v : r;
        }
        return r;
    }
    __device__ __forceinline__ float rare_sum(int c) const { return sm[kQueue + NX * (lane < T ? lane : 0) + c]; }
};

// Many targets: a warp owns 32 consecutive ones, a lane each.  Consecutive particles of the
// sorted order follow a column of cells in z, so they lie in one cell or in two on top of each
// other and share nearly all candidates:
//   cull    32 candidates a round, a lane each, against the box around the targets; what is
//           in reach goes to a ring in shared memory
//   screen  every candidate of the ring against all 32 targets at once (its coordinates
//           broadcast, two candidates per packed instruction); a lane appends what it accepts
//           to its own list, without votes or ranks
//   terms   when a list could overflow: the lists as one sequence, a lane per pair
//   sums    a lane per (component, target) adds the terms in order
// Per candidate that is about 8 instructions for 32 targets where RpWarp needs 17 for 8, at a
// quarter of the warps.  A list entry is one word and its squared distance is computed
// again with the terms: with both kept, 15.6 instead of 10.9 KB per warp, the gradient took 1,083
// instead of 884 us at 884,736 particles and, beside the pressure on other streams, lost it all.
template <class Op>
struct RpSlice {
    static constexpr int NS = Op::NS;
    static_assert(Op::NX == 0, "no rarer pairs");
    static constexpr int kCap = 48, kStride = 49;             // a list: at most 32 entries and 16 new ones
    static constexpr int kPlane = 32 * kStride;               // a word per entry: the candidate or, if the
                                                              // terms need no more, the squared distance
    static constexpr int G = NS > 1 ? 8 : 32, NG = 32 / G;    // targets whose terms are held at a time
    static constexpr int kMore = NS > 1 ? 9 + (NS - 1) * (G * kStride + 9) : 0;   // terms past the first, which takes its entry's place
    static constexpr int kRing = (kPlane + kMore + 3) & ~3, kSum = kRing + 4 * 64;
    static constexpr int kFloats = kSum + NS * 32;
    static_assert(NS * G <= 32 || NS == 1, "a lane per sum");

    float* sm;
    float re, re2x, mind;
    unsigned long long nz2;
    int lane, first, cnt;
    RpTarget me;

    __device__ __forceinline__ RpSlice(float* smem, float radius, float minus_zero, int first_id,
                                       const RpTarget& t)
        : sm(smem), re(radius), re2x(ref_screen2(radius)), mind((float)(radius * 1e-3)),
          nz2(rp_pack(minus_zero, minus_zero)), lane(threadIdx.x & 31), first(first_id), cnt(0), me(t) {
#pragma unroll
        for (int c = 0; c < NS; ++c) sm[kSum + c * 32 + lane] = 0.0f;
        __syncwarp();
    }

    // row of component c of target t's terms
    __device__ __forceinline__ float* row(int c, int t) const {
        return c == 0 ? sm + t * kStride : sm + kPlane + 9 + (c - 1) * (G * kStride + 9) + (t % G) * kStride;
    }

    // Lists -> terms -> sums; empties the lists.  Terms of several components are called, not
    // inlined, at the places that need them: their code would not fit the instruction cache
    // (the gradient took twice as long).
    __device__ __forceinline__ void flush(const RefBind& b) {
        if constexpr (NS > 1) {
            flush_call(b, sm, re, cnt, me);
        } else {
            flush_lists(b);
        }
        cnt = 0;
    }
    static __device__ __noinline__ void flush_call(const RefBind& b, float* sm, float re, int cnt, RpTarget me) {
        RpSlice(sm, re, cnt, me).flush_lists(b);
    }
    __device__ __forceinline__ RpSlice(float* smem, float radius, int n, const RpTarget& t)
        : sm(smem), re(radius), re2x(0.0f), mind((float)(radius * 1e-3)), nz2(0), lane(threadIdx.x & 31), first(0),
          cnt(n), me(t) {}
    __device__ __forceinline__ void flush_lists(const RefBind& b) {
        __syncwarp();
        int end = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(~0u, end, o);
            if (lane >= o) end += v;
        }
        const int start = end - cnt;
#pragma unroll 1
        for (int g = 0; g < NG; ++g) {
            const int e1 = __shfl_sync(~0u, end, g * G + G - 1);
#pragma unroll 1
            for (int e0 = __shfl_sync(~0u, start, g * G); e0 < e1; e0 += 32) {
                const int e = e0 + lane;
                int t = g * G;   // the last target whose pairs start at or before e
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) {
                    const int v = __shfl_sync(~0u, start, t + o);
                    if (v <= e) t += o;
                }
                const int at = e - __shfl_sync(~0u, start, t);
                RpTarget q;
                if constexpr (Op::kPos || Op::kIndex) {
                    q.pos.x = __shfl_sync(~0u, me.pos.x, t);
                    q.pos.y = __shfl_sync(~0u, me.pos.y, t);
                    q.pos.z = __shfl_sync(~0u, me.pos.z, t);
                }
                if constexpr (Op::kVel) {
                    q.vel.x = __shfl_sync(~0u, me.vel.x, t);
                    q.vel.y = __shfl_sync(~0u, me.vel.y, t);
                    q.vel.z = __shfl_sync(~0u, me.vel.z, t);
                }
                if constexpr (Op::kScalar) q.s = __shfl_sync(~0u, me.s, t);
                if (e < e1) {
                    float v[NS];
#pragma unroll
                    for (int c = 0; c < NS; ++c) v[c] = 0.0f;
                    float d2 = row(0, t)[at];
                    int x = 0;
                    if constexpr (Op::kIndex) {
                        x = __float_as_int(d2);
                        const Scalar3 p = b.pos[x];
                        const float dx = q.pos.x - p.x, dy = q.pos.y - p.y, dz = q.pos.z - p.z;
                        d2 = dx * dx + dy * dy + dz * dz;
                    }
                    float d = ref_sqrt(d2);
                    const bool ok = Op::kLe ? d <= re : d < re;
                    if (d < mind) d = mind;
                    if (ok) Op::terms(b, re, q, x, d, v);
#pragma unroll
                    for (int c = 0; c < NS; ++c) row(c, t)[at] = v[c];
                }
            }
            __syncwarp();
            const int t = g * G + lane % G, n = __shfl_sync(~0u, cnt, t), most = __reduce_max_sync(~0u, n);
            const int c = lane < NS * G ? lane / G : 0;
            const float* const r = row(c, t);
            float s = sm[kSum + c * 32 + t];
#pragma unroll 1
            for (int e = 0; e < most; e += 4) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = e + u < n ? r[e + u] : 0.0f;
#pragma unroll
                for (int u = 0; u < 4; ++u) s += v[u];   // + 0 leaves a sum that starts at + 0 alone
            }
            __syncwarp();
            if (lane < NS * G) sm[kSum + c * 32 + t] = s;
        }
        cnt = 0;
    }

    // Candidates of the targets `grp`, all in cells (cx, cy, cz) and (cx, cy, cz + 1); this
    // lane's target in cell layer tz
    __device__ __forceinline__ void walk(const RefBind& b, unsigned grp, int cx, int cy, int cz, bool two, int tz) {
        const Integer3 dims = b.box.m_GridSize;
        const bool mine = grp >> lane & 1u;
        float* const rx = sm + kRing;
        float* const ry = rx + 64;
        float* const rz = ry + 64;
        int* const ri = reinterpret_cast<int*>(rz + 64);
        const float nan = __int_as_float(0x7fffffff);
        const bool far_target = __any_sync(
            ~0u, mine && fmaxf(fabsf(me.pos.x), fmaxf(fabsf(me.pos.y), fabsf(me.pos.z))) > kRpHuge);
        const int id = first + lane;
        unsigned long long tx = 0, ty = 0, tz2 = 0;   // (-t, -t) per coordinate
        float lo[3], hi[3];
        bool in = false;
        int wp = 0, rp = 0, own_until = 0;   // ring positions below own_until may hold targets
        // 16 candidates of the ring against every target
        auto screen = [&](int at, bool self) {
            float* const list = sm + lane * kStride;
            unsigned qa = (unsigned)__cvta_generic_to_shared(list + cnt);
            const unsigned q0 = (unsigned)__cvta_generic_to_shared(list);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                ulonglong2 X[2], Y[2], Z[2];
                int4 I[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int o = at + 8 * part + 4 * c;
                    X[c] = *reinterpret_cast<const ulonglong2*>(rx + o);
                    Y[c] = *reinterpret_cast<const ulonglong2*>(ry + o);
                    Z[c] = *reinterpret_cast<const ulonglong2*>(rz + o);
                    I[c] = *reinterpret_cast<const int4*>(ri + o);
                }
                float d2[8];
                int x[8];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const unsigned long long dx = rp_add2(h ? X[c].y : X[c].x, tx), dy = rp_add2(h ? Y[c].y : Y[c].x, ty),
                                                 dz = rp_add2(h ? Z[c].y : Z[c].x, tz2);
                        rp_unpack(rp_add2(rp_add2(rp_mul2(dx, dx, nz2), rp_mul2(dy, dy, nz2)), rp_mul2(dz, dz, nz2)),
                                  d2[4 * c + 2 * h], d2[4 * c + 2 * h + 1]);
                    }
                    x[4 * c] = I[c].x;
                    x[4 * c + 1] = I[c].y;
                    x[4 * c + 2] = I[c].z;
                    x[4 * c + 3] = I[c].w;
                }
                if (self) {
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (x[u] == id) d2[u] = nan;   // the target itself
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float entry = Op::kIndex ? __int_as_float(x[u]) : d2[u];
                    asm volatile(
                        "{\n .reg .pred a;\n setp.lt.f32 a, %1, %2;\n @a st.shared.f32 [%0], %3;\n"
                        " @a add.u32 %0, %0, 4;\n}\n"
                        : "+r"(qa)
                        : "f"(d2[u]), "f"(re2x), "f"(entry)
                        : "memory");
                }
            }
            cnt = (int)(qa - q0) >> 2;
            if (__any_sync(~0u, cnt > kCap - 16)) flush(b);
        };
        auto drain = [&]() {   // the ring's last, incomplete 32
            if (wp > rp) {
                if (lane >= wp - rp) {
                    rx[(rp & 32) + lane] = nan;
                    ri[(rp & 32) + lane] = -1;
                }
                __syncwarp();
                screen(rp & 32, true);
                if (wp - rp > 16) screen((rp & 32) + 16, true);
                __syncwarp();
            }
            wp = rp = own_until = 0;
        };
#pragma unroll 1
        for (int up = -1; up <= (two ? 2 : 1); ++up) {   // layers of cells
            if (up == -1 || two) {
                // a layer's targets: those at most one layer away (two: each layer has its own)
                in = mine && (tz == cz ? up <= 1 : up >= 0);
                const Scalar3 p = in ? me.pos : s3(nan, nan, nan);
                tx = rp_pack(-p.x, -p.x);
                ty = rp_pack(-p.y, -p.y);
                tz2 = rp_pack(-p.z, -p.z);
                const float v[3] = {p.x, p.y, p.z};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    lo[a] = in ? v[a] : 3.4e38f;
                    hi[a] = in ? v[a] : -3.4e38f;
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        lo[a] = fminf(lo[a], __shfl_xor_sync(~0u, lo[a], o));
                        hi[a] = fmaxf(hi[a], __shfl_xor_sync(~0u, hi[a], o));
                    }
                }
            }
            // lane m < 9: cell m of the layer (j outer, i inner)
            int s = 0, len = 0;
            if (lane < 9) {
                const int m = cell_key(dims, (int)((unsigned)cx + (unsigned)(lane % 3 - 1)),
                                       (int)((unsigned)cy + (unsigned)(lane / 3 - 1)), (int)((unsigned)cz + (unsigned)up));
                if (m >= 0 && m < b.cell_num) {
                    s = b.cell_start[m];
                    if (s != -1) len = max(b.cell_end[m] - s, 0);
                }
            }
            unsigned cells = __ballot_sync(~0u, len > 0);
            int x0 = 0, e = 0;
            auto fetch = [&](int x) {
                return RpWarp<Op, 8>::fetch(b, x, e);
            };
            auto next_cell = [&]() {
                if (!cells) return false;
                const int m = __ffs(cells) - 1;
                cells &= cells - 1u;
                x0 = __shfl_sync(~0u, s, m);
                e = x0 + __shfl_sync(~0u, len, m);
                return true;
            };
            bool more = next_cell();
            Scalar3 qn = s3(nan, nan, nan);
            if (more) qn = fetch(x0 + lane);
#pragma unroll 1
            while (more) {
                const Scalar3 q = qn;
                const int x = x0 + lane;
                const bool own = x0 < first + 32 && x0 + 32 > first;
                x0 += 32;
                if (x0 >= e) more = next_cell();
                if (more) qn = fetch(x0 + lane);   // the next round's, under this one's work
                const bool huge = fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))) > kRpHuge;
                if (far_target || __any_sync(~0u, huge)) {
                    // a squared distance may overflow (the reference accepts an infinite one)
                    drain();
#pragma unroll 1
                    for (int c = 0; c < 32; ++c) {
                        const int xc = __shfl_sync(~0u, x, c);
                        const float dx = me.pos.x - __shfl_sync(~0u, q.x, c), dy = me.pos.y - __shfl_sync(~0u, q.y, c),
                                    dz = me.pos.z - __shfl_sync(~0u, q.z, c);
                        const float d2 = dx * dx + dy * dy + dz * dz;
                        if (in && xc != id && d2 == d2 && !(d2 >= re2x && d2 <= 3.402823466e38f)) {
                            sm[lane * kStride + cnt] = Op::kIndex ? __int_as_float(xc) : d2;
                            ++cnt;
                        }
                        if (__any_sync(~0u, cnt > kCap - 16)) flush(b);
                    }
                    continue;
                }
                // the box in the order and rounding of a pair's squared distance: never above it
                const float ax = fmaxf(fmaxf(lo[0] - q.x, q.x - hi[0]), 0.0f), ay = fmaxf(fmaxf(lo[1] - q.y, q.y - hi[1]), 0.0f),
                            az = fmaxf(fmaxf(lo[2] - q.z, q.z - hi[2]), 0.0f);
                const bool keep = q.x == q.x && !(ax * ax + ay * ay + az * az >= re2x);
                const unsigned m = __ballot_sync(~0u, keep);
                if (keep) {
                    const int pos = (wp + __popc(m & ((1u << lane) - 1u))) & 63;
                    rx[pos] = q.x;
                    ry[pos] = q.y;
                    rz[pos] = q.z;
                    ri[pos] = x;
                }
                wp += __popc(m);
                own_until = own ? wp : own_until;
                if (wp - rp >= 32) {
                    __syncwarp();
                    const bool self = own_until > rp;
                    screen(rp & 32, self);
                    screen((rp & 32) + 16, self);
                    rp += 32;
                    __syncwarp();
                }
            }
            if (two) drain();
        }
        drain();
    }

    // all targets of the warp: `live`, their cells (tx, ty, tz)
    __device__ __forceinline__ void run(const RefBind& b, bool live, int tx, int ty, int tz) {
        for (unsigned todo = __ballot_sync(~0u, live); todo;) {
            const int l = __ffs(todo) - 1;
            const int gx = __shfl_sync(~0u, tx, l), gy = __shfl_sync(~0u, ty, l), gz = __shfl_sync(~0u, tz, l);
            const bool here = (todo >> lane & 1u) && tx == gx && ty == gy;
            const unsigned up = __ballot_sync(~0u, here && gz != 0x7fffffff && tz == gz + 1);
            const unsigned grp = __ballot_sync(~0u, here && tz == gz) | up;
            walk(b, grp, gx, gy, gz, up != 0u, tz);
            todo &= ~grp;
        }
        flush(b);
    }
    // sum c of this lane's target
    __device__ __forceinline__ float sum(int c) const { return sm[kSum + c * 32 + lane]; }
};

// Sparse fluid: a cell holds fewer than about `few` particles, seen from 16 targets spread over
// the sorted order, half of which at least have the target `few` places on more than a cell
// away.  Every warp of a call comes to the same answer, from one round of loads.
__device__ __forceinline__ bool rp_sparse(const RefBind& b, int n, int few) {
    const int lane = threadIdx.x & 31;
    bool near = false;
    if (lane < 16) {
        const int x = (int)((long long)n * (2 * lane + 1) / 32);
        const Scalar3 p = b.pos[x], q = b.pos[min(x + few, n - 1)];
        near = fmaxf(fabsf(p.x - q.x), fmaxf(fabsf(p.y - q.y), fabsf(p.z - q.z))) < b.box.m_CellSize;
    }
    return __popc(__ballot_sync(~0u, near)) < 8;
}

// A lane per target, each walking its own 27 cells.  The bounds of a layer's nine cells are
// loaded together into `run` (a column of shared memory per thread), so a target without
// neighbours waits for memory six times, not 54.  It needs no votes, ranks and second pass per
// pair and no warp per few targets, but runs the terms of every candidate that any of 32
// targets accepts: for many accepted pairs per candidate or few candidates per cell.
template <class Op>
__device__ __forceinline__ void rp_walk_sums(const RefBind& b, const RpTarget& t, int id, bool walk, int cx, int cy, int cz,
                                             float re, int2* run, int stride, float (&acc)[Op::NS],
                                             float (&xacc)[RpShape<Op>::NXR]) {
    const float mind = (float)(re * 1e-3), re2x = ref_screen2(re);
    float rare_re = 0.0f;
    if constexpr (Op::NX > 0) rare_re = Op::rare_radius(b.param);
#pragma unroll
    for (int c = 0; c < Op::NS; ++c) acc[c] = 0.0f;
#pragma unroll
    for (int c = 0; c < RpShape<Op>::NXR; ++c) xacc[c] = 0.0f;
    if (!walk) return;
#pragma unroll 1
    for (int k = -1; k <= 1; ++k) {
        int s[9], m[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            m[q] = cell_key(b.box.m_GridSize, (int)((unsigned)cx + (unsigned)(q % 3 - 1)),
                            (int)((unsigned)cy + (unsigned)(q / 3 - 1)), (int)((unsigned)cz + (unsigned)k));
            s[q] = m[q] >= 0 && m[q] < b.cell_num ? b.cell_start[m[q]] : -1;
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) run[q * stride] = make_int2(s[q], s[q] != -1 ? b.cell_end[m[q]] : -1);
#pragma unroll 1
        for (int q = 0; q < 9; ++q) {
            const int2 r = run[q * stride];
#pragma unroll 1
            for (int x = r.x; x < r.y; ++x) {
                const int out = b.out_id[x];
                const Scalar3 p = b.pos[x];
                const float dx = t.pos.x - p.x, dy = t.pos.y - p.y, dz = t.pos.z - p.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                if (out < 0 || x == id || (d2 >= re2x && d2 <= 3.402823466e38f)) continue;
                float d = ref_sqrt(d2);
                if (!(Op::kLe ? d <= re : d < re)) continue;
                if (d < mind) d = mind;
                float v[Op::NS];
                Op::terms(b, re, t, x, d, v);
#pragma unroll
                for (int c = 0; c < Op::NS; ++c) acc[c] += v[c];
                if constexpr (Op::NX > 0) {
                    if (d < rare_re) {
                        float ex[Op::NX];
                        Op::rare_terms(b, re, t, x, d, ex);
#pragma unroll
                        for (int c = 0; c < Op::NX; ++c) xacc[c] += ex[c];
                    }
                }
            }
        }
    }
}

}  // namespace mps
