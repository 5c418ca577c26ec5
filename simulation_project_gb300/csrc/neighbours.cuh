// neighbours.cuh - the FP32 neighbour passes: predictor and PPE rows, a lane per target.
//
// A warp takes a slice of 32 consecutive particles of the cell-sorted order (the SELL-32
// slice of the rows), a lane each.  Consecutive particles follow a column of cells in z, so
// the slice fills a short piece of a column and its targets share almost all of their
// candidates: the nine z-runs around the piece.  The warp reads the runs once, 32 candidates
// per load, keeps those within reach of the box around its targets (about 0.55 of them)
// in a ring in shared memory and tests every kept one against all 32 targets, the
// candidate's coordinates broadcast and two candidates per packed FP32 instruction.
//
// Both passes are bound by instruction issue (DRAM traffic is 1.9 GB of written rows for the
// list, almost nothing for the predictor).  A warp per target with 32 candidates per
// round needed ballots, population counts and a queue to bring the accepted third of its
// candidates together, 25 instructions per round and 2000 warp instructions per target; here
// a candidate costs about 13 instructions with its terms (predictor) or 7 (list) per 32
// targets, and no sum crosses lanes.
//
// Sums: at most 32 terms are added in FP32, then folded into a two-word sum (Knuth's
// TwoSum), so the totals are closer to the exact ones than the lane-strided sums of a
// warp per target were.
//
// us before -> now, rotating bucket (254 neighbours per interior target), a warp per target and
// a transpose of the rows before:    2,000        108,186      882,080 particles
//   predictor                        49 -> 23     250 -> 108   1746 -> 691
//   rows (list + transpose)          80 -> 46     364 -> 192   2485 -> 1359
// The predictor issues in 0.67 of the cycles with the FMA pipe next; the rows wait for
// shared memory and L1 (the gathers and three stores per entry keep the LSU's data stage
// busy for half of the time) with the sixteen warps that fit beside the lists.
#pragma once

namespace mps {

constexpr int kNpWarps = 4;        // warps of a k_predict CTA
constexpr int kNbOff = 4095;       // longest run that a 16-bit list entry (run << 12 | offset) can index
constexpr int kGradStride = 66;    // 16-bit words per target's gradient list (KG = 64, rows 33 banks apart)

__device__ __forceinline__ unsigned long long f2_pack(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// dist2_f32 of two candidates (the same roundings): q - p with np = -p
__device__ __forceinline__ void dist2_f32x2(unsigned long long qx, unsigned long long qy, unsigned long long qz,
                                            unsigned long long npx, unsigned long long npy, unsigned long long npz,
                                            float& d0, float& d1) {
    unsigned long long r;
    asm("{\n .reg .b64 x, y, z;\n"
        " add.rn.f32x2 x, %1, %4;\n add.rn.f32x2 y, %2, %5;\n add.rn.f32x2 z, %3, %6;\n"
        " mul.rn.f32x2 x, x, x;\n fma.rn.f32x2 x, y, y, x;\n fma.rn.f32x2 %0, z, z, x;\n}\n"
        : "=l"(r)
        : "l"(qx), "l"(qy), "l"(qz), "l"(npx), "l"(npy), "l"(npz));
    f2_unpack(r, d0, d1);
}
// (hi, lo) += x with the rounding error of hi kept in lo
__device__ __forceinline__ void two_sum(float& hi, float& lo, float x) {
    const float s = __fadd_rn(hi, x), b = __fsub_rn(s, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
    hi = s;
}

// 64 candidates in shared memory: positions by component, and per candidate either its
// velocity (predictor) or its list code (rows)
template <bool LIST> struct NbRing;
template <> struct __align__(16) NbRing<false> {
    float x[64], y[64], z[64];
    float4 v[64];
};
template <> struct __align__(16) NbRing<true> {
    float x[64], y[64], z[64];
    unsigned code[64];
};

// A piece of the slice whose targets share their nine runs: consecutive lanes `mem` in one
// column of cells, over at most two cells in z (one where the cells are smaller than the
// radius, so that no target gets candidates from outside its 27 cells).  Lanes 0..8 hold
// the runs, `lo` and `hi` the box around the targets.
struct NbPiece {
    unsigned mem;
    int rs, rl;
    float lo[3], hi[3];
};
__device__ __forceinline__ NbPiece nb_piece(const Dev& d, unsigned todo, int h, const float4& p) {
    const Integer3 G = d.box.m_GridSize;
    const int lane = threadIdx.x & 31, lead = __ffs(todo) - 1;
    const int col = h / G.z, cz = h % G.z;
    const int col0 = __shfl_sync(~0u, col, lead), z0 = __shfl_sync(~0u, cz, lead);
    NbPiece s;
    s.mem = __ballot_sync(~0u, (todo >> lane & 1u) && col == col0 && cz - z0 <= d.c.wide_cells);
    const int z1 = __shfl_sync(~0u, cz, 31 - __clz(s.mem));
    const bool in = s.mem >> lane & 1u;
    const float v[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        s.lo[a] = in ? v[a] : 3.4e38f;
        s.hi[a] = in ? v[a] : -3.4e38f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            s.lo[a] = fminf(s.lo[a], __shfl_xor_sync(~0u, s.lo[a], o));
            s.hi[a] = fmaxf(s.hi[a], __shfl_xor_sync(~0u, s.hi[a], o));
        }
    s.rs = s.rl = 0;
    if (lane < 9) {
        const int x = col0 / G.y + lane / 3 - 1, y = col0 % G.y + lane % 3 - 1;
        if (x >= 0 && x < G.x && y >= 0 && y < G.y) {
            int first = -1, last = -1;
#pragma unroll
            for (int dz = -1; dz <= 2; ++dz) {
                const int z = z0 + dz;
                if (z < 0 || z > min(z1 + 1, G.z - 1)) continue;
                const int c = cell_key(G, x, y, z);
                const int st = d.cstart[c];
                if (st >= 0) {
                    if (first < 0) first = st;
                    last = d.cend[c];
                }
            }
            if (first >= 0) {
                s.rs = first;
                s.rl = last - first;
            }
        }
    }
    return s;
}

// The candidates of runs [r0, r1) of a piece (of the first one from `from` on, of the last
// one up to `to`), in order, those in reach of its box put into the ring; block(base, centre) takes 32 of them (ring positions base..base+31) at a time,
// centre: some of them are of the targets' own run.  The last block is filled up with
// points that no target accepts.
template <bool LIST, class Block>
__device__ __forceinline__ void nb_walk(const Dev& d, const NbPiece& s, int r0, int r1, int from, int to, float cut,
                                        NbRing<LIST>& R, Block&& block) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int r = r0 - 1, b = 0, len = 0, start = 0;
    auto advance = [&]() {
        b += 32;
        while (b >= len) {
            if (++r == r1) return false;
            len = __shfl_sync(~0u, s.rl, r);
            if (r == r1 - 1) len = min(len, to);
            start = __shfl_sync(~0u, s.rs, r);
            b = r == r0 ? from : 0;
        }
        return true;
    };
    // the next round's candidates are in flight under a round's work, two rounds' for the
    // list (fewer warps); for the predictor the second one cost registers and 13 % more time
    struct Round {
        float4 q;
        int o, r, j;
        bool on, any;
    };
    auto fetch = [&]() {
        Round f;
        f.any = r < r1 && advance();
        f.o = b + lane;
        f.r = r;
        f.j = start + f.o;
        f.on = f.any && f.o < len;
        f.q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (f.on) f.q = d.opos[f.j];
        return f;
    };
    int wp = 0, rp = 0, c0 = 1 << 30, c1 = 0;
    Round n1 = fetch(), n2;
    if constexpr (LIST) n2 = fetch();
    while (n1.any) {
        const float4 c = n1.q;
        const int o = n1.o, j = n1.j, cr = n1.r;
        const bool on = n1.on;
        if constexpr (LIST) {
            n1 = n2;
            n2 = fetch();
        } else {
            n1 = fetch();
        }
        const float dx = fmaxf(fmaxf(__fsub_rn(s.lo[0], c.x), __fsub_rn(c.x, s.hi[0])), 0.f),
                    dy = fmaxf(fmaxf(__fsub_rn(s.lo[1], c.y), __fsub_rn(c.y, s.hi[1])), 0.f),
                    dz = fmaxf(fmaxf(__fsub_rn(s.lo[2], c.z), __fsub_rn(c.z, s.hi[2])), 0.f);
        const bool keep = on && dist2_f32(dx, dy, dz) < cut;
        const unsigned m = __ballot_sync(~0u, keep);
        if (keep) {
            const int pos = (wp + __popc(m & lt)) & 63;
            R.x[pos] = c.x;
            R.y[pos] = c.y;
            R.z[pos] = c.z;
            if constexpr (LIST) R.code[pos] = (unsigned)cr << 12 | (unsigned)o;
            else R.v[pos] = d.ovel[j];
        }
        if (cr == 4 && c0 > wp) c0 = wp;
        wp += __popc(m);
        if (cr == 4) c1 = wp;
        if (wp - rp >= 32) {
            __syncwarp();
            block(rp & 32, c1 > rp && c0 < rp + 32);
            rp += 32;
            __syncwarp();
        }
    }
    if (wp > rp) {
        if (lane >= wp - rp) R.x[(rp & 32) + lane] = 1e30f;
        __syncwarp();
        block(rp & 32, c1 > rp && c0 < rp + 32);
        __syncwarp();
    }
}

// Laplacian of the velocity -> viscosity / gravity / drag predictor.  S warps share a slice
// (three runs each with S = 3): with fewer slices than the chip has schedulers the runs are
// what there is to spread.  80 registers for S = 1, six CTAs on an SM (five with 96: 725 us
// instead of 691 at 882,080 particles).
template <int S>
__global__ void __launch_bounds__(S == 1 ? kNpWarps * 32 : S * 32, S == 1 ? 6 : 1) k_predict(const __grid_constant__ Dev d) {
    constexpr int W = S == 1 ? kNpWarps : S;
    __shared__ NbRing<false> ring[W];
    __shared__ float part[S > 1 ? S - 1 : 1][6][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = S == 1 ? blockIdx.x * W + warp : blockIdx.x;
    if (sl * 32 >= d.n) return;   // warp-uniform; CTA-uniform for S > 1
    const int i = sl * 32 + lane;
    const bool live = i < d.n;
    const float qnan = __int_as_float(0x7fc00000);
    const int h = live ? d.key[i] : 0;
    const float4 p = live ? d.opos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v = live ? d.ovel[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float re = (float)d.c.re_lap, re2s = re * re;
    const float cut = d.c.reach2, wmax = d.c.wmax_lap;
    float hi[3] = {0.f, 0.f, 0.f}, lo[3] = {0.f, 0.f, 0.f};
    for (unsigned todo = __ballot_sync(~0u, live); todo;) {
        const NbPiece s = nb_piece(d, todo, h, p);
        todo &= ~s.mem;
        const bool in = s.mem >> lane & 1u;
        const float px = in ? -p.x : qnan;   // a lane outside the piece accepts nothing
        const unsigned long long npx = f2_pack(px, px), npy = f2_pack(-p.y, -p.y), npz = f2_pack(-p.z, -p.z);
        const unsigned long long nvxy = f2_pack(-v.x, -v.y);
        NbRing<false>& R = ring[warp];
        nb_walk<false>(d, s, S == 1 ? 0 : 3 * warp, S == 1 ? 9 : 3 * warp + 3, 0, 1 << 30, cut, R, [&](int base, bool) {
            unsigned long long axy = 0ull;
            float az = 0.f;
#pragma unroll(S == 1 ? 1 : 2)
            for (int c = base; c < base + 32; c += 4) {
                const ulonglong2 X = *(const ulonglong2*)&R.x[c], Y = *(const ulonglong2*)&R.y[c],
                                 Z = *(const ulonglong2*)&R.z[c];
                float d2[4];
                dist2_f32x2(X.x, Y.x, Z.x, npx, npy, npz, d2[0], d2[1]);
                dist2_f32x2(X.y, Y.y, Z.y, npx, npy, npz, d2[2], d2[3]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float rinv;
                    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rinv) : "f"(d2[u]));
                    // re / max(r, mind) - 1; a coincident point (rinv = inf) gets the largest weight
                    const float w = fminf(__fmaf_rn(re, rinv, -1.f), wmax);
                    const ulonglong2 V = *(const ulonglong2*)&R.v[c + u];
                    asm("{\n .reg .pred a;\n .reg .b64 t, ww;\n .reg .f32 z, zz;\n"
                        " setp.lt.f32 a, %2, %3;\n mov.b64 ww, {%4, %4};\n mov.b64 {z, zz}, %6;\n"
                        " @a add.rn.f32x2 t, %5, %7;\n @a sub.rn.f32 z, z, %8;\n"
                        " @a fma.rn.f32x2 %0, t, ww, %0;\n @a fma.rn.f32 %1, z, %4, %1;\n}\n"
                        : "+l"(axy), "+f"(az)
                        : "f"(d2[u]), "f"(re2s), "f"(w), "l"(V.x), "l"(V.y), "l"(nvxy), "f"(v.z));
                }
            }
            float ax, ay;
            f2_unpack(axy, ax, ay);
            two_sum(hi[0], lo[0], ax);
            two_sum(hi[1], lo[1], ay);
            two_sum(hi[2], lo[2], az);
        });
    }
    if constexpr (S > 1) {
        if (warp > 0) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                part[warp - 1][a][lane] = hi[a];
                part[warp - 1][3 + a][lane] = lo[a];
            }
        }
        __syncthreads();
        if (warp > 0) return;
#pragma unroll
        for (int w = 0; w < S - 1; ++w)
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                two_sum(hi[a], lo[a], part[w][a][lane]);
                lo[a] += part[w][3 + a][lane];
            }
    }
    if (live)
        nb_epilogue<float, NB_PREDICT>(d, i, (double)hi[0] + (double)lo[0], (double)hi[1] + (double)lo[1],
                                       (double)hi[2] + (double)lo[2], 0, 0);
}

// shared memory of a k_list CTA: the lists of accepted candidates [K + 16][32], the gradient
// lists (the rings of candidates lie there before the first of them is written), the first
// particle of each run of each piece, what the second warp hands to the first
constexpr int kNbPieces = 32, kNbHand = 9;   // a slice has at most as many pieces as targets
static_assert(2 * sizeof(NbRing<true>) <= 32 * kGradStride * 2, "the rings lie in the gradient lists");
inline size_t nb_list_smem(int L) {
    return (size_t)(L + 16) * 64 + 32 * kGradStride * 2 + kNbPieces * 9 * 4 + kNbHand * 32 * 4;
}

// Rows of the PPE: Laplacian rows straight into the SELL-32 slices (16- or 32-bit columns,
// FP32 and FP16 weights, see k_rows_sell for `flags`), gradient rows, PND, sum of weights.
// Two warps per slice first list each target's accepted candidates as 16-bit codes (run << 12 |
// offset in the run) in shared memory, in candidate order: the first warp the first half from
// the bottom of the list up, the second one the second half from the top down, so neither
// has to know the other's count.  Then all lanes write entry k of their rows together, so
// every store is a full line of the slice, each warp half of the entries; the distance is
// computed again from the listed candidate's position (an L1 gather), which is cheaper than 4 more
// bytes of shared memory per entry.  L: entries that a list has room for (25 KB per slice with
// 296, 31 KB with 384; sixteen or fourteen warps per SM).  112 registers, 8 candidates and 4
// entries at a time: 16 and 8 of them spilled (1620 us instead of 1360 at 882,080 particles).
// Bit 4 of flags, a row longer than L or a run too long for the codes: the candidates are walked
// twice by one warp, once for the rows' lengths and ends and once for the entries, 32 at a time
// culled against the box around the targets, with no list; same rows and sums, bit for bit (cells
// three times the radius, 216,000 particles: 5.7 ms with a warp per target, 24 without the cull,
// 3.8 now).
__global__ void __maxnreg__(112) k_list(const __grid_constant__ Dev d, int flags, int L) {
    extern __shared__ __align__(16) unsigned char nb_sm[];
    unsigned short* const list = (unsigned short*)nb_sm;
    unsigned short* const glist = list + (size_t)(L + 16) * 32;
    int* const rtab = (int*)(glist + 32 * kGradStride);
    int* const hand = rtab + kNbPieces * 9;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sl = blockIdx.x, r0 = sl * 32, i = r0 + lane;
    NbRing<true>& R = ((NbRing<true>*)glist)[warp];
    const bool live = i < d.n;
    const bool narrow = (flags & 1) != 0, w16 = (flags & 2) != 0, full32 = (flags & 4) != 0;
    const float qnan = __int_as_float(0x7fc00000);
    const int h = live ? d.key[i] : 0;
    const float4 p = live ? d.opos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float re = (float)d.c.re_lap, re2s = re * re, mind = (float)d.c.mind_lap;
    const float reg = (float)d.c.re_grad;
    const float cut = d.c.reach2, wmax = d.c.wmax_lap, wgmax = d.c.wmax_grad;
    const unsigned all = __ballot_sync(~0u, live);
    // first list position of this warp's lane and the step to the next one, in bytes
    const unsigned q0 = smem_u32(list) + 2u * lane + (warp ? 64u * (unsigned)(L + 15) : 0u);
    const int step = warp ? -64 : 64;
    unsigned qa = q0;
    auto listed = [&]() { return (int)(warp ? q0 - qa : qa - q0) >> 6; };
    int over = 0, piece = 0, rt = 0, mycode = 4 << 12;
    bool direct = (flags & 16) != 0;

    // ---- the targets' accepted candidates
    for (unsigned todo = direct ? 0u : all; todo; ++piece) {
        const NbPiece s = nb_piece(d, todo, h, p);
        todo &= ~s.mem;
        if (__any_sync(~0u, s.rl > kNbOff)) {
            direct = true;   // in both warps
            break;
        }
        if (warp == 0 && lane < 9) rtab[piece * 9 + lane] = s.rs - (lane << 12);   // code + entry = particle
        const bool in = s.mem >> lane & 1u;
        const int own = i - __shfl_sync(~0u, s.rs, 4), half = (__shfl_sync(~0u, s.rl, 4) / 2) & ~31;
        if (in) {
            rt = piece * 9;
            mycode = 4 << 12 | own;
        }
        const float px = in ? -p.x : qnan;
        const unsigned long long npx = f2_pack(px, px), npy = f2_pack(-p.y, -p.y), npz = f2_pack(-p.z, -p.z);
        nb_walk<true>(d, s, warp ? 4 : 0, warp ? 9 : 5, warp ? half : 0, warp ? 1 << 30 : half, cut, R,
                      [&](int base, bool centre) {
            // eight candidates are read while the eight before them are listed: the list's
            // stores keep the compiler from moving loads across them
            ulonglong2 X[2], Y[2], Z[2];
            uint4 code[2];
            auto load = [&](int at) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    X[c] = *(const ulonglong2*)&R.x[at + 4 * c];
                    Y[c] = *(const ulonglong2*)&R.y[at + 4 * c];
                    Z[c] = *(const ulonglong2*)&R.z[at + 4 * c];
                    code[c] = *(const uint4*)&R.code[at + 4 * c];
                }
            };
            load(base);
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                float d2[8];
                unsigned cd[8];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    dist2_f32x2(X[c].x, Y[c].x, Z[c].x, npx, npy, npz, d2[4 * c], d2[4 * c + 1]);
                    dist2_f32x2(X[c].y, Y[c].y, Z[c].y, npx, npy, npz, d2[4 * c + 2], d2[4 * c + 3]);
                    cd[4 * c] = code[c].x;
                    cd[4 * c + 1] = code[c].y;
                    cd[4 * c + 2] = code[c].z;
                    cd[4 * c + 3] = code[c].w;
                }
                if (part < 3) load(base + 8 * part + 8);
                if (centre) {
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (cd[u] == (unsigned)mycode) d2[u] = qnan;   // the target itself
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    asm volatile(
                        "{\n .reg .pred a;\n .reg .b16 c, e;\n mov.b32 {c, e}, %3;\n setp.lt.f32 a, %1, %2;\n"
                        " @a st.shared.u16 [%0], c;\n @a add.s32 %0, %0, %4;\n}\n"
                        : "+r"(qa)
                        : "f"(d2[u]), "f"(re2s), "r"(cd[u]), "r"(step)
                        : "memory");
                if (listed() > L) {   // a row longer than the list
                    over = 1;
                    qa = q0 + (unsigned)(step * L);
                }
            }
        });
    }
    hand[warp * 64 + lane] = listed();
    hand[warp * 64 + 32 + lane] = over;
    __syncthreads();

    // ---- direct walk: f(j, d2) for every accepted candidate of this lane's target, in order
    auto walk = [&](auto&& f) {
        for (unsigned todo = all; todo;) {
            const NbPiece s = nb_piece(d, todo, h, p);
            todo &= ~s.mem;
            const bool in = s.mem >> lane & 1u;
            for (int r = 0; r < 9; ++r) {
                const int start = __shfl_sync(~0u, s.rs, r), end = start + __shfl_sync(~0u, s.rl, r);
                for (int b = start; b < end; b += 32) {   // 32 candidates, those in reach of the box
                    const float4 c = d.opos[min(b + lane, end - 1)];
                    const float dx = fmaxf(fmaxf(__fsub_rn(s.lo[0], c.x), __fsub_rn(c.x, s.hi[0])), 0.f),
                                dy = fmaxf(fmaxf(__fsub_rn(s.lo[1], c.y), __fsub_rn(c.y, s.hi[1])), 0.f),
                                dz = fmaxf(fmaxf(__fsub_rn(s.lo[2], c.z), __fsub_rn(c.z, s.hi[2])), 0.f);
                    for (unsigned m = __ballot_sync(~0u, b + lane < end && dist2_f32(dx, dy, dz) < cut); m; m &= m - 1u) {
                        const int u = __ffs(m) - 1;
                        const float d2 = dist2_f32(__fsub_rn(__shfl_sync(~0u, c.x, u), p.x),
                                                   __fsub_rn(__shfl_sync(~0u, c.y, u), p.y),
                                                   __fsub_rn(__shfl_sync(~0u, c.z, u), p.z));
                        if (in && b + u != i && d2 < re2s) f(b + u, d2);
                    }
                }
            }
        }
    };
    const int low = hand[lane];   // entries from the bottom of the list
    int cnt = low + hand[64 + lane], jlo = i, jhi = i;
    direct = direct || __any_sync(~0u, cnt > L || hand[32 + lane] + hand[96 + lane] > 0);   // in both warps
    if (direct && warp) return;   // no barrier follows in the direct walk
    if (direct) {
        cnt = 0;
        walk([&](int j, float) {
            if (cnt == 0) jlo = j;
            if (cnt < d.K) jhi = j;
            ++cnt;
        });
    }
    const int cap = min(cnt, d.K), kmax = __reduce_max_sync(~0u, cap);
    // FP16 weights are padded with zeros (column offset 0) to whole chunks of 16 entries, so that
    // k_spmv_ring_split needs no bounds
    const int kpad = w16 ? (kmax + 15) & ~15 : kmax;
    const int khalf = (kmax + 63) / 64 * 32;   // entries of the first warp: [0, khalf)
    auto decode = [&](unsigned code) { return rtab[rt + (code >> 12)] + (int)code; };
    auto code_of = [&](int k) { return (unsigned)list[(k < low ? k : L + 15 + low - k) * 32 + lane]; };
    if (!direct && cap > 0) {
        jlo = decode(code_of(0));
        jhi = decode(code_of(cap - 1));
    }
    // columns ascend within a row, so its ends decide whether the slice fits 16 bits
    const bool n16 = narrow && __all_sync(~0u, jlo - r0 >= -32768 && jhi - r0 <= 32767);
    const bool c32 = full32 || !n16;

    // ---- entry k of every row
    const size_t e0 = (size_t)sl * d.K * 32 + lane;
    float* const ws = (float*)d.nbrw + e0;
    __half* const wh = d.w16 + e0;
    int* const n32 = d.nbr + e0;
    unsigned short* const c16 = d.nbr16 + e0;
    // sums of the weights, of the gradient-radius weights (PND) and of the FP16 weights: b of
    // at most 32 entries, folded into the two-word a
    float a[3] = {0.f, 0.f, 0.f}, al[3] = {0.f, 0.f, 0.f}, b[3] = {0.f, 0.f, 0.f};
    int gcnt = 0;
    // the weight within the gradient radius, zero outside (where re / r - 1 < 0)
    auto grad_weight = [&](float rinv) { return fminf(fmaxf(__fmaf_rn(reg, rinv, -1.f), 0.f), wgmax); };
    auto entry = [&](int k, int j, float w, float rinv) {
        ws[k * 32] = w;
        if (c32) n32[k * 32] = j;
        if (n16) c16[k * 32] = (unsigned short)(short)(j - r0);
        const __half hw = __float2half_rn(w);
        if (w16) wh[k * 32] = hw;
        b[0] += w;
        b[1] += grad_weight(rinv);
        b[2] += __half2float(hw);
    };
    auto pad = [&](int k) {
        if (w16 && k < kpad) {
            wh[k * 32] = __ushort_as_half((unsigned short)0);
            if (n16) c16[k * 32] = 0;
        }
    };
    auto fold = [&]() {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            two_sum(a[q], al[q], b[q]);
            b[q] = 0.f;
        }
    };
    float f[3] = {0.f, 0.f, 0.f}, fl[3] = {0.f, 0.f, 0.f};   // sums over the other half
    if (direct) {
        int k = 0;
        int* const grow = d.gnbr + (size_t)i * d.KG;
        float* const grr = (float*)d.gnbrr + (size_t)i * d.KG;
        walk([&](int j, float d2) {
            if (k >= d.K) return;
            float rinv, rr;
            const float w = lap_weight_f32(d2, re, mind, wmax, rinv, rr);
            entry(k, j, w, rinv);
            if (rr < reg) {
                if (gcnt < d.KG) {
                    grow[gcnt] = j;
                    grr[gcnt] = rr;
                }
                ++gcnt;
            }
            if ((++k & 31) == 0) fold();
            if (k == khalf)
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    f[q] = a[q];
                    fl[q] = al[q];
                    a[q] = al[q] = 0.f;
                }
        });
        for (int t = k; t < kpad; ++t) pad(t);
        fold();
        if (k < khalf) {   // the whole row lies in the first half
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                f[q] = a[q];
                fl[q] = al[q];
                a[q] = al[q] = 0.f;
            }
        }
    } else {
        const int idle = min(i, d.n - 1), kb = warp ? khalf : 0, ke = warp ? kpad : min(khalf, kpad);
        // the first warp's gradient entries from the bottom of the list, the second one's from its top
        unsigned ga = smem_u32(glist + lane * kGradStride + (warp ? d.KG - 1 : 0));
        const int gs = warp ? -2 : 2;
        auto grad = [&](bool on, float rr, unsigned code) {   // without a branch
            asm volatile(
                "{\n .reg .pred a, s;\n .reg .b16 c, e;\n setp.ne.s32 a, %3, 0;\n setp.lt.and.f32 a, %4, %5, a;\n"
                " setp.lt.and.s32 s, %1, %6, a;\n mov.b32 {c, e}, %2;\n @s st.shared.u16 [%0], c;\n"
                " @s add.s32 %0, %0, %7;\n @a add.s32 %1, %1, 1;\n}\n"
                : "+r"(ga), "+r"(gcnt)
                : "r"(code), "r"((int)on), "f"(rr), "f"(reg), "r"(d.KG), "r"(gs)
                : "memory");
        };
        // U entries at a time without a branch, the next U positions in flight under their work
        constexpr int U = 4;
        unsigned code[U];
        int j[U];
        float4 q[U];
        const int kmin = __reduce_min_sync(~0u, cap);
        auto fetch = [&](int k) {
            if (k + U <= kmin) {
#pragma unroll
                for (int u = 0; u < U; ++u) code[u] = code_of(k + u);
#pragma unroll
                for (int u = 0; u < U; ++u) j[u] = decode(code[u]);
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    code[u] = k + u < cap ? code_of(k + u) : (unsigned)mycode;
                    j[u] = k + u < cap ? decode(code[u]) : idle;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) q[u] = __ldg(d.opos + j[u]);
        };
        // COMMON: a 16-bit slice with FP16 weights alone, every row reaching the group's end
        const bool common = n16 && !c32 && w16;
        auto group = [&](auto COMMON, int k) {
            unsigned cc[U];
            int cj[U];
            float w[U], rinv[U], rr[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                cc[u] = code[u];
                cj[u] = j[u];
                w[u] = lap_weight_f32(
                    dist2_f32(__fsub_rn(q[u].x, p.x), __fsub_rn(q[u].y, p.y), __fsub_rn(q[u].z, p.z)), re, mind, wmax,
                    rinv[u], rr[u]);
            }
            if (k + U < ke) fetch(k + U);
            if constexpr (COMMON.value) {
                float* const pw = ws + k * 32;
                unsigned short* const pc = c16 + k * 32;
                __half* const ph = wh + k * 32;
                __half2 hw[U / 2];
#pragma unroll
                for (int u = 0; u < U; u += 2) hw[u / 2] = __floats2half2_rn(w[u], w[u + 1]);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    pw[u * 32] = w[u];
                    pc[u * 32] = (unsigned short)(short)(cj[u] - r0);
                    ph[u * 32] = u & 1 ? __high2half(hw[u / 2]) : __low2half(hw[u / 2]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float2 wf = __half22float2(hw[u / 2]);
                    b[0] += w[u];
                    b[1] += grad_weight(rinv[u]);
                    b[2] += u & 1 ? wf.y : wf.x;
                    grad(true, rr[u], cc[u]);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (k + u < cap) entry(k + u, cj[u], w[u], rinv[u]);
                    else pad(k + u);
                    grad(k + u < cap, rr[u], cc[u]);
                }
            }
            if (((k + U) & 31) == 0) fold();
        };
        if (kb < ke) fetch(kb);
#pragma unroll 1
        for (int k = kb; k < ke; k += U) {
            if (common && k + U <= kmin) group(std::true_type(), k);
            else group(std::false_type(), k);
        }
        fold();
        __syncthreads();   // the counts in `hand` have been read, the gradient lists are written
        if (warp) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                hand[q * 32 + lane] = __float_as_int(a[q]);
                hand[(3 + q) * 32 + lane] = __float_as_int(al[q]);
            }
        }
        hand[(6 + warp) * 32 + lane] = gcnt;
        __syncthreads();
        // gradient rows, four targets at a time (a row is contiguous)
        const int g0 = hand[6 * 32 + lane], g1 = hand[7 * 32 + lane], gc = min(g0 + g1, d.KG);
        int glow = min(g0, d.KG);
        if (__any_sync(~0u, g0 + g1 > d.KG)) {   // in both warps
            // the halves of a full list have met and overwritten each other: the first KG
            // entries of every row again, from the whole list in its order
            if (warp == 0) {
                int g = 0;
                for (int k = 0; k < cap && g < d.KG; ++k) {
                    const unsigned cg = code_of(k);
                    const float4 qg = __ldg(d.opos + decode(cg));
                    float ri, rr;
                    lap_weight_f32(dist2_f32(__fsub_rn(qg.x, p.x), __fsub_rn(qg.y, p.y), __fsub_rn(qg.z, p.z)), re, mind,
                                   wmax, ri, rr);
                    if (rr < reg) glist[lane * kGradStride + g++] = (unsigned short)cg;
                }
            }
            __syncthreads();
            glow = gc;
        }
        for (int t0 = 16 * warp; t0 < 16 * warp + 16; t0 += 4) {
            int tj[8];
            float4 tq[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + u / 2, s = lane + (u & 1) * 32;
                const int g = __shfl_sync(~0u, gc, t), gb = __shfl_sync(~0u, glow, t), rtt = __shfl_sync(~0u, rt, t);
                tj[u] = -1;
                if (s < g) {
                    const unsigned cg = glist[t * kGradStride + (s < gb ? s : d.KG - 1 + gb - s)];
                    tj[u] = rtab[rtt + (cg >> 12)] + (int)cg;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) tq[u] = __ldg(d.opos + max(tj[u], 0));
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int t = t0 + u / 2, s = lane + (u & 1) * 32;
                const float tx = __shfl_sync(~0u, p.x, t), ty = __shfl_sync(~0u, p.y, t), tz = __shfl_sync(~0u, p.z, t);
                float ri, rr;
                lap_weight_f32(dist2_f32(__fsub_rn(tq[u].x, tx), __fsub_rn(tq[u].y, ty), __fsub_rn(tq[u].z, tz)), re,
                               mind, wmax, ri, rr);
                if (tj[u] >= 0) {
                    const size_t e = (size_t)(r0 + t) * d.KG + s;
                    d.gnbr[e] = tj[u];
                    ((float*)d.gnbrr)[e] = rr;
                }
            }
        }
        if (warp) return;
        gcnt = g0 + g1;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            f[q] = a[q];
            fl[q] = al[q];
            a[q] = __int_as_float(hand[q * 32 + lane]);
            al[q] = __int_as_float(hand[(3 + q) * 32 + lane]);
        }
    }
    // first half, then the second half's sum
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        two_sum(f[q], fl[q], a[q]);
        fl[q] += al[q];
    }

    // ---- the targets
    bool inner = false;
    if (live) {
        const double pnd = nb_epilogue<float, NB_LIST>(d, i, (double)f[0] + (double)fl[0], 0.0,
                                                       (double)f[1] + (double)fl[1], cnt, gcnt);
        inner = pnd > d.c.beta * d.c.n0_pnd;
        if (w16 && cap > 0 && inner) d.diag16[i] = d.c.coef_lap * ((double)f[2] + (double)fl[2]) + d.c.kappa;
    }
    const int ic = inner ? cap : 0, kin = __reduce_max_sync(~0u, ic), wide = __reduce_add_sync(~0u, ic);
    if (lane == 0) {
        d.sbase[sl] = n16 ? r0 : -1;
        d.skmax[sl] = n16 ? kin : -1 - kin;
        if (narrow && !n16 && wide) atomicAdd(d.istat + 1, wide);
    }
}

// the 32-bit columns of the slices that have 16-bit ones alone
__global__ void k_rows_widen(const __grid_constant__ Dev d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.n) return;
    const int sb = d.sbase[i >> 5], cnt = d.nbr_cnt[i];
    if (sb < 0) return;
    for (int k = 0; k < cnt; ++k) {
        const size_t e = sell_index(i, k, d.K);
        d.nbr[e] = sb + (short)d.nbr16[e];
    }
}

}  // namespace mps
