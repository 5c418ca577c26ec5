// ref_kernels.cu - the reference solver's explicit-schedule kernels, GB300 build, and
// the reference-named C-ABI that a caller of the reference's launcher API binds.
//
// Boundary: radix/SPVSOLVER/MultiGPUSolver/DeviceProcess.h:78-120 (declarations) and
// DeviceProcess.cu:49-409 (launchers).  The reference binds every device array once
// through __constant__ pointer symbols (Constant.h:4-76, filled by
// InitializeDeviceMemConst & co.); here the same binding calls fill one host-side
// RefBind record that every launch passes to its kernel as a __grid_constant__
// parameter (it lands in the same constant bank, without cudaMemcpyToSymbol).
//
// This translation unit is compiled with -fmad=false: the float arithmetic below is
// written in the reference's operation order, so each kernel produces the reference's
// results bit for bit (checked against the oracle, which is itself pinned to the
// reference's kernel code).  Deviations, all on invalid inputs: every kernel checks
// its thread index against the item count (CalcSTLDistance_Kernel does not), cell
// bounds skip keys outside [0, cells) instead of writing out of bounds, and a cell's
// triangle list is filled in ascending triangle id (the reference's atomics give an
// arbitrary order).
#include <cfloat>
#include <stdio.h>

#include <algorithm>
#include <atomic>

#include "mps_common.cuh"
#include "mps_internal.h"
#include "../../include/mps_device_process.h"

namespace mps {

struct RefBind {
    CParameter param;
    CGridBox box;
    int particle_num;
    int max_particle_num;
    int* id;
    Scalar3* pos;
    Scalar3* vel;
    float* pressure;
    float* density;
    float* temperature;
    float* kin_visc;
    float* solid_rate;
    int* type;
    int* out_id;
    Scalar3* out_pos;
    Scalar3* out_vel;
    float* out_pressure;
    float* out_density;
    float* out_temperature;
    float* out_kin_visc;
    float* out_solid_rate;
    int* out_type;
    CTriangle* triangles;
    int triangle_num;
    CTriangleParameters* tri_params;
    CDistance* stl_distance;
    int* stl_id;
    CCell* cells;
    int cell_num;
    int* cell_start;
    int* cell_end;
    int* grid_index;
    DragParameter* drag_params;
    int drag_num;
    Scalar3* drag_acc;
    float* drag_temperature;
    int* magnifier_count;
    CDragTriangle* drag_triangles;
    float* turb_visc;   // c_daParticleTurbulaceViscosity (sorted order)
    float* strain;      // c_daParticleStrainTensorProduct (sorted order)
};

static RefBind g_bind;

// ---------------------------------------------------------------------------
// grid
// ---------------------------------------------------------------------------
// calcHashD (DeviceProcess_Kernel.h:39-50)
__global__ void k_ref_hash(int n, const __grid_constant__ CGridBox box, const Scalar3* __restrict__ pos,
                           int* __restrict__ hash, int* __restrict__ index) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int a, b, c;
    hash[i] = ref_cell(box, pos[i], a, b, c);
    index[i] = i;
}

// reorderDataAndFindCellStartD (DeviceProcess_Kernel.h:54-124): cell bounds from
// key changes along the sorted keys, and the gather of the nine particle arrays.
__global__ void k_ref_reorder(int n, int cells, const int* __restrict__ hash, const int* __restrict__ index,
                              int* __restrict__ cs, int* __restrict__ ce, const __grid_constant__ RefBind b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int h = hash[i];
    const bool ok = h >= 0 && h < cells;
    if (i == 0 || h != hash[i - 1]) {
        if (ok) cs[h] = i;
        if (i > 0) {
            const int hp = hash[i - 1];
            if (hp >= 0 && hp < cells) ce[hp] = i;
        }
    }
    if (i == n - 1 && ok) ce[h] = i + 1;
    const int s = index[i];
    b.pos[i] = b.out_pos[s];
    b.vel[i] = b.out_vel[s];
    b.pressure[i] = b.out_pressure[s];
    b.density[i] = b.out_density[s];
    b.temperature[i] = b.out_temperature[s];
    b.kin_visc[i] = b.out_kin_visc[s];
    b.solid_rate[i] = b.out_solid_rate[s];
    b.type[i] = b.out_type[s];
    b.id[i] = s;
}

// Compaction with the order of CCellSet::CheckParticleOutsideComputeZone
// (CGPUCellSet.cpp:1160-1202): the j-th out-of-zone slot i (j = 1, 2, ...) takes the
// particle at N0 - j while i <= N0 - j; the taken particles are not re-checked.
// Sources are never earlier destinations, so one gather kernel suffices.
__global__ void k_ref_outside_flags(int n, const __grid_constant__ RefBind b, unsigned* __restrict__ flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Scalar3 p = b.out_pos[i];
    flag[i] = in_zone<float>(b.box, p.x, p.y, p.z, b.param.Tolerance) ? 0u : 1u;
}
__global__ void k_ref_compact(int n, const __grid_constant__ RefBind b, const unsigned* __restrict__ flag,
                              const unsigned* __restrict__ rank, int* __restrict__ removed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !flag[i]) return;
    const int j = (int)rank[i] + 1;
    if (i > n - j) return;
    atomicAdd(removed, 1);
    const int s = n - j;
    if (s == i) return;
    b.out_pos[i] = b.out_pos[s];
    b.out_vel[i] = b.out_vel[s];
    b.out_pressure[i] = b.out_pressure[s];
    b.out_density[i] = b.out_density[s];
    b.out_temperature[i] = b.out_temperature[s];
    b.out_kin_visc[i] = b.out_kin_visc[s];
    b.out_solid_rate[i] = b.out_solid_rate[s];
    b.out_type[i] = b.out_type[s];
    b.out_id[i] = b.out_id[s];
}

// ---------------------------------------------------------------------------
// walls
// ---------------------------------------------------------------------------
// SegmentRatio / CalcDistanceVectorLine / CalcNormalDistance / CalcDistance(triangle)
// (Utility_Inline.h:56-232), reference arithmetic.
__device__ __forceinline__ float ref_segment_ratio(const Scalar3& p1, const Scalar3& p2, const Scalar3& p3) {
    const Scalar3 d = s3sub(p2, p1);
    float den = d.x * d.x + d.y * d.y + d.z * d.z;
    if (den == 0.0f) den = (float)1e-5;
    return (p3.x - p1.x) * (p2.x - p1.x) + (p3.y - p1.y) * (p2.y - p1.y) + (p3.z - p1.z) * (p2.z - p1.z) / den;
}
__device__ __forceinline__ Scalar3 ref_line(const Scalar3& l0, const Scalar3& l1, const Scalar3& p) {
    const float u = ref_segment_ratio(l0, l1, p);
    Scalar3 dv = s3(0, 0, 0);
    if (u >= 0 && u <= 1) {
        const Scalar3 v = s3sub(l1, l0);
        dv = s3sub(p, s3(l0.x + u * v.x, l0.y + u * v.y, l0.z + u * v.z));
    }
    if (u < 0) dv = s3sub(l1, p);
    if (u > 1) dv = s3sub(l0, p);
    return dv;
}
// CalcDistance(triangle): what depends on the triangle alone, then a point's distance.
// The reference's centroid divides in double, (float)((double)s / 3.0); s / 3.0f is the
// same float: the quotient of a float by 3 lies at least 2^-26 of itself away from every
// midpoint of two floats, so rounding to double first never decides (GB300 has few FP64
// units).
struct RefTri {
    Scalar3 a, b, c, n, e0, e1;   // vertices, normal, edges a-c and a-b
    float nc, sd, d00, d01, d11, inv;
};
__device__ __forceinline__ RefTri ref_tri(const CTriangle& T) {
    RefTri r;
    r.a = T.Vertex[0];
    r.b = T.Vertex[1];
    r.c = T.Vertex[2];
    r.n = T.Normal;
    Scalar3 m;
    m.x = (r.a.x + r.b.x + r.c.x) / 3.0f;
    m.y = (r.a.y + r.b.y + r.c.y) / 3.0f;
    m.z = (r.a.z + r.b.z + r.c.z) / 3.0f;
    r.nc = r.n.x * m.x + r.n.y * m.y + r.n.z * m.z;
    r.sd = ref_sqrt(r.n.x * r.n.x + r.n.y * r.n.y + r.n.z * r.n.z);
    r.e0 = s3sub(r.c, r.a);
    r.e1 = s3sub(r.b, r.a);
    r.d00 = ref_dot(r.e0, r.e0);
    r.d01 = ref_dot(r.e0, r.e1);
    r.d11 = ref_dot(r.e1, r.e1);
    r.inv = 1.0f / (r.d00 * r.d11 - r.d01 * r.d01);
    return r;
}
__device__ __forceinline__ float ref_tri_distance(const RefTri& T, const Scalar3& p, Scalar3& dir) {
    const Scalar3 n = T.n;
    Scalar3 dv = s3(0, 0, 0);
    if (T.sd != 0.0f) {
        const float coef = ((n.x * p.x + n.y * p.y + n.z * p.z) - T.nc) / T.sd;
        dv = s3(coef / T.sd * n.x, coef / T.sd * n.y, coef / T.sd * n.z);
    }
    const Scalar3 P = s3(p.x - dv.x, p.y - dv.y, p.z - dv.z);
    const Scalar3 v2 = s3sub(P, T.a);
    const float d02 = ref_dot(T.e0, v2), d12 = ref_dot(T.e1, v2);
    const float u = (T.d11 * d02 - T.d01 * d12) * T.inv;
    const float v = (T.d00 * d12 - T.d01 * d02) * T.inv;
    // the reference's three edge tests, of which the last one that holds decides
    const bool bc = u >= 0 && v >= 0 && u + v > 1, ab = u < 0, ac = v < 0;
    if (bc || ab || ac) dv = ref_line(ab || ac ? T.a : T.b, ac ? T.c : ab ? T.b : T.c, p);
    dir = dv;
    return ref_mag(dv);
}

// RegisterLine / RegisterTriangle (Utility_Inline.h:1745-1855): walk the three edges
// in cell-size steps, shrink the triangle toward its interior by one cell, repeat.
// visit(cell, ok) is called for every sample point, ok where it lies inside the grid, by
// the G lanes of `group` together: lane l takes steps l, l + G, ... of a line, each step's
// offset summed from cell sizes as the reference's loop sums it.
template <int G, class Visit>
__device__ __forceinline__ void ref_walk_line(const CGridBox& B, Scalar3 v, Scalar3 d, float m, int cells, unsigned group,
                                              int lane, Visit& visit) {
    constexpr int kMost = 100000;   // steps of a line
    float tab = 0.0f;
    for (int q = 0; q < lane && tab <= m; ++q) tab += B.m_CellSize;
    for (int step = lane;; step += G) {
        const bool in = (step == 0 || tab <= m) && step < kMost;
        if (!__any_sync(group, in)) break;
        int cid = -1;
        if (in) {
            const Scalar3 t = s3(v.x + tab * d.x, v.y + tab * d.y, v.z + tab * d.z);
            int i, j, k;
            cid = ref_cell(B, t, i, j, k);
        }
        visit(cid, cid >= 0 && cid < cells);
#pragma unroll
        for (int q = 0; q < G; ++q) tab += B.m_CellSize;
    }
}
template <int G, class Visit>
__device__ void ref_walk_triangle(const CGridBox& B, const CTriangle& T, int cells, unsigned group, int lane, Visit& visit) {
    Scalar3 A = T.Vertex[0], Bv = T.Vertex[1], C = T.Vertex[2];
    const float cs = B.m_CellSize;
    float mbc, mab, mca;
    int guard = 0;
    do {
        const Scalar3 ab = s3sub(Bv, A), ba = s3sub(A, Bv), bc = s3sub(C, Bv), cb = s3sub(Bv, C), ca = s3sub(A, C),
                      ac = s3sub(C, A);
        mbc = ref_mag(bc);
        mab = ref_mag(ab);
        mca = ref_mag(ca);
#pragma unroll 1
        for (int e = 0; e < 3; ++e) {
            const Scalar3 from = e == 0 ? A : e == 1 ? Bv : C, along = e == 0 ? ab : e == 1 ? bc : ca;
            const float m = e == 0 ? mab : e == 1 ? mbc : mca;
            if (m > 0.0f)
                ref_walk_line<G>(B, from, s3(along.x / m, along.y / m, along.z / m), m, cells, group, lane, visit);
        }
        Scalar3 am = s3add(ab, ac), bm = s3add(ba, bc), cm = s3add(ca, cb);
        const float mam = ref_mag(am), mbm = ref_mag(bm), mcm = ref_mag(cm);
        if (mam > 0.0f) {
            am.x /= mam; am.y /= mam; am.z /= mam;
            A.x += am.x * cs; A.y += am.y * cs; A.z += am.z * cs;
        }
        if (mbm > 0.0f) {
            bm.x /= mbm; bm.y /= mbm; bm.z /= mbm;
            Bv.x += bm.x * cs; Bv.y += bm.y * cs; Bv.z += bm.z * cs;
        }
        if (mcm > 0.0f) {
            cm.x /= mcm; cm.y /= mcm; cm.z /= mcm;
            C.x += cm.x * cs; C.y += cm.y * cs; C.z += cm.z * cs;
        }
    } while (mbc >= cs && mab >= cs && mca >= cs && ++guard < 100000);
}

struct CountVisit {
    int n = 0;
    __device__ __forceinline__ void operator()(int, bool ok) { n += ok; }
};
// the visits of a triangle in any order: they are sorted by cell, and a cell takes each
// triangle once
struct StoreVisit {
    int* cell;
    int* tri;
    int t;
    unsigned group, below;
    int k = 0;
    __device__ __forceinline__ void operator()(int c, bool ok) {
        const unsigned m = __ballot_sync(group, ok) & group;
        if (ok) {
            const int at = k + __popc(m & below);
            cell[at] = c;
            tri[at] = t;
        }
        k += __popc(m);
    }
};

// G lanes per triangle
template <int G>
__global__ void __launch_bounds__(kBlock) k_tri_count(int t, const CTriangle* __restrict__ tri,
                                                      const __grid_constant__ CGridBox box, int cells,
                                                      unsigned* __restrict__ count, unsigned* __restrict__ failed) {
    if (blockIdx.x == 0 && threadIdx.x == 0) failed[0] = failed[1] = 0u;   // the sort's error word, the runs' number
    const int i = blockIdx.x * (kBlock / G) + threadIdx.x / G, lane = threadIdx.x % G;
    if (i >= t) return;   // the G lanes of a triangle leave together
    const unsigned group = G == 32 ? ~0u : ((1u << (G % 32)) - 1u) << (threadIdx.x & 31 & ~(G - 1));
    CountVisit v;
    const CTriangle T = tri[i];
    ref_walk_triangle<G>(box, T, cells, group, lane, v);
    for (int o = G / 2; o > 0; o >>= 1) v.n += __shfl_xor_sync(group, v.n, o);
    if (lane == 0) count[i] = (unsigned)v.n;
}
template <int G>
__global__ void __launch_bounds__(kBlock) k_tri_fill(int t, const CTriangle* __restrict__ tri,
                                                     const __grid_constant__ CGridBox box, int cells,
                                                     const unsigned* __restrict__ off, int* __restrict__ vcell,
                                                     int* __restrict__ vtri) {
    const int i = blockIdx.x * (kBlock / G) + threadIdx.x / G, lane = threadIdx.x % G;
    if (i >= t) return;
    StoreVisit v;
    v.group = G == 32 ? ~0u : ((1u << (G % 32)) - 1u) << (threadIdx.x & 31 & ~(G - 1));
    v.below = (1u << (threadIdx.x & 31)) - 1u;
    v.cell = vcell + off[i];
    v.tri = vtri + off[i];
    v.t = i;
    const CTriangle T = tri[i];
    ref_walk_triangle<G>(box, T, cells, v.group, lane, v);
}
// Visits sorted (stably) by cell: where each cell's run of visits begins, in any order, and how
// many runs there are (*runs_n, zero on entry).  After a sort that gave up no cell gets a
// triangle and the host hears of it (*report).
__global__ void __launch_bounds__(kBlock) k_tri_runs(int nv, const int* __restrict__ vcell, int* __restrict__ runs,
                                                     int* __restrict__ runs_n, const unsigned* __restrict__ failed,
                                                     volatile unsigned* report) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (*failed) {
        if (i == 0) *report = 1u;
        return;
    }
    const bool begin = i < nv && (i == 0 || vcell[i] != vcell[i - 1]);
    const unsigned m = __ballot_sync(~0u, begin);
    const int lane = threadIdx.x & 31;
    int at = 0;
    if (m && lane == 0) at = atomicAdd(runs_n, __popc(m));
    at = __shfl_sync(~0u, at, 0);
    if (begin) runs[at + __popc(m & ((1u << lane) - 1u))] = i;
}
// Unique triangle ids per cell, ascending, first 100: a warp per run, 32 visits a round, a
// triangle taken where its visits begin (they ascend) unless the cell held it before.  Cells
// without triangles cost nothing: with a warp per cell of the grid 12 triangles in 8,000,000
// cells took 933 us, 538 with a thread per cell, now 411 (the rest resets the cells).
__global__ void __launch_bounds__(kBlock) k_tri_cells(int nv, const int* __restrict__ runs, const int* __restrict__ runs_n,
                                                      const int* __restrict__ vcell, const int* __restrict__ vtri,
                                                      CCell* __restrict__ out) {
    const int r = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= *runs_n) return;
    const int s = runs[r], c = vcell[s];
    const unsigned held = out[c].m_TriangleNum;
    unsigned cnt = held;
    bool more = true;
    for (int i0 = s; more && cnt < CELLMAXTRIANGLENUM; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i < nv && vcell[i] == c;
        const int t = in ? vtri[i] : -1;
        bool take = in && t != (i > s ? vtri[i - 1] : -1);
        for (unsigned l = 0; take && l < held && l < CELLMAXTRIANGLENUM; ++l) take = out[c].m_TriangleID[l] != t;
        const unsigned m = __ballot_sync(~0u, take);
        const unsigned at = cnt + __popc(m & ((1u << lane) - 1u));
        if (take && at < CELLMAXTRIANGLENUM) out[c].m_TriangleID[at] = t;
        cnt += __popc(m);
        more = __all_sync(~0u, in);
    }
    if (lane == 0) out[c].m_TriangleNum = cnt > CELLMAXTRIANGLENUM && held <= CELLMAXTRIANGLENUM ? CELLMAXTRIANGLENUM : cnt;
}

// ResetTriangleTopology_Kernel (DeviceProcess_Kernel.h:594-602)
__global__ void k_tri_reset(int cells, CCell* __restrict__ cell) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < cells) cell[c].m_TriangleNum = 0;
}

// UpdateTrianglePosition_Kernel (DeviceProcess_Kernel.h:603-621)
__global__ void k_tri_translate(int t, CTriangle* __restrict__ tri, const __grid_constant__ RefBind b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= t) return;
    Scalar3 v = b.tri_params[tri[i].ModelIDNumber].Velocity;
    const float dt = b.param.Dt;
    v.x = v.x * dt; v.y = v.y * dt; v.z = v.z * dt;
    for (int q = 0; q < 3; ++q) tri[i].Vertex[q] = s3add(tri[i].Vertex[q], v);
}

// RotateTrianglePosition_Kernel (DeviceProcess_Kernel.h:622-689)
__global__ void k_tri_rotate(int t, CTriangle* __restrict__ tri, int step, const __grid_constant__ RefBind b) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= t) return;
    CTriangle& T = tri[id];
    const CTriangleParameters tp = b.tri_params[T.ModelIDNumber];
    if (!tp.RotatingOrNot) return;
    const float dt = b.param.Dt;
    if ((step * dt) < tp.RotationStartTime) return;
    float ang = 0.0f;
    const int req = (int)((tp.TimeToReachRPM - tp.RotationStartTime) / dt);
    const float tpass = dt * step;
    if ((tpass < tp.RotationStartTime) || (tp.AngleOfRotationInDegree == 0)) ang = 0.0f;
    else if ((tpass >= tp.RotationStartTime) && (tpass < tp.TimeToReachRPM))
        ang = (tp.AngleOfRotationInDegree / (req + 1)) * (step - (tp.RotationStartTime / dt));
    else ang = tp.AngleOfRotationInDegree;
    if (ang == 0) return;
    for (int q = 0; q < 3; ++q) {
        const float m = ref_dist(tp.SecondPointOfRotation, tp.CenterOfRotation);
        Scalar3 nv = s3(0, 0, 0);
        if (m > 0)
            nv = s3((tp.SecondPointOfRotation.x - tp.CenterOfRotation.x) / m,
                    (tp.SecondPointOfRotation.y - tp.CenterOfRotation.y) / m,
                    (tp.SecondPointOfRotation.z - tp.CenterOfRotation.z) / m);
        const float th = (float)((ang * 3.141592653589793238) / 180.0);
        const float a = tp.CenterOfRotation.x, bb = tp.CenterOfRotation.y, c = tp.CenterOfRotation.z;
        const float u = nv.x, v = nv.y, w = nv.z;
        const float x = T.Vertex[q].x, y = T.Vertex[q].y, z = T.Vertex[q].z;
        const float ct = cosf(th), st = sinf(th);
        T.Vertex[q].x = (a * (v * v + w * w) - (u * (bb * v + c * w - u * x - v * y - w * z))) * (1 - ct) + (x * ct) +
                        (((-c * v) + bb * w - w * y + v * z) * st);
        T.Vertex[q].y = (bb * (u * u + w * w) - (v * (a * u + c * w - u * x - v * y - w * z))) * (1 - ct) + (y * ct) +
                        (((c * u) - a * w + w * x - u * z) * st);
        T.Vertex[q].z = (c * (u * u + v * v) - (w * (a * u + bb * v - u * x - v * y - w * z))) * (1 - ct) + (z * ct) +
                        (((-bb * u) + a * v - v * x + u * y) * st);
    }
}

// ResetWallPosition_Kernel (DeviceProcess_Kernel.h:690-704)
__global__ void k_tri_reset_wall(int t, int step, const CTriangle* __restrict__ orig, const __grid_constant__ RefBind b) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= t) return;
    const CTriangleParameters& tp = b.tri_params[b.triangles[id].ModelIDNumber];
    if (tp.LinearMovableOrNot && tp.LinearResetInterval != 0 && 0 == ((step + 1) % tp.LinearResetInterval))
        b.triangles[id] = orig[id];
}

// Nearest triangle over the 27 cells, (k, j, i) order, first minimum wins: a warp for T
// consecutive particles, lane t holding particle t (`live`: it has a cell).  The cells'
// triangle lists as one sequence, a lane per entry: what depends on the triangle alone is
// computed once for all particles of a cell, each lane keeps its first minimum per
// particle, and the earliest of the warp's minima is the serial loop's (a triangle met
// again changes nothing).  Returns in lane t the triangle (-1: none) and its distance.
//
// Bound by the latency of long lists: particles beside drag spheres meet hundreds of
// entries while most meet none, and a thread per particle ran them one after another, each
// with three FP64 divisions: 535 us for 108,186 particles and 9,216 triangles, DRAM idle.
// A warp for four: 184 us (drag 548 -> 179); 882,080 particles 478 -> 367 (376 -> 314).  Where
// most particles see few triangles a lane per particle goes first (near_short_most).
constexpr int kNearT = 4;
template <bool DRAG>
__device__ __forceinline__ void ref_nearest(const RefBind& b, const Scalar3& p, bool live, CDistance& nd, int& nid) {
    constexpr int T = kNearT;
    const int lane = threadIdx.x & 31;
    int cx = 0, cy = 0, cz = 0;
    if (live) {
        const int cid = ref_cell(b.box, p, cx, cy, cz);
        live = cid >= 0 && cid < b.cell_num;
    }
    Scalar3 q[T];
    float best[T];
    int at[T], id[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        q[t] = s3(__shfl_sync(~0u, p.x, t), __shfl_sync(~0u, p.y, t), __shfl_sync(~0u, p.z, t));
        best[t] = 1e8f;
        at[t] = 0x7fffffff;
        id[t] = -1;
    }
    unsigned todo = __ballot_sync(~0u, live);
#pragma unroll 1
    while (todo) {
        const int l = __ffs(todo) - 1;
        const int gx = __shfl_sync(~0u, cx, l), gy = __shfl_sync(~0u, cy, l), gz = __shfl_sync(~0u, cz, l);
        const unsigned grp = __ballot_sync(~0u, live && cx == gx && cy == gy && cz == gz) & todo;
        todo &= ~grp;
        int m = -1, len = 0;
        if (lane < 27) {
            m = cell_key(b.box.m_GridSize, (int)((unsigned)gx + (unsigned)(lane % 3) - 1u),
                         (int)((unsigned)gy + (unsigned)(lane / 3 % 3) - 1u), (int)((unsigned)gz + (unsigned)(lane / 9) - 1u));
            if (m >= 0 && m < b.cell_num) len = (int)min(b.cells[m].m_TriangleNum, (unsigned)CELLMAXTRIANGLENUM);
        }
        int off = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(~0u, off, o);
            if (lane >= o) off += v;
        }
        const int total = __shfl_sync(~0u, off, 31);
        off -= len;
#pragma unroll 1
        for (int c0 = 0; c0 < total; c0 += 32) {
            const int c = c0 + lane;
            int k = 0;   // the last cell whose list starts at or before c
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const int v = __shfl_sync(~0u, off, k + o);
                if (v <= c) k += o;
            }
            const int cell = __shfl_sync(~0u, m, k), first = __shfl_sync(~0u, off, k);
            if (c < total) {
                const int t = b.cells[cell].m_TriangleID[c - first];
                if (t >= 0 && t < b.triangle_num &&
                    !(DRAG && !b.tri_params[b.triangles[t].ModelIDNumber].isDrag)) {
                    const RefTri tri = ref_tri(b.triangles[t]);
#pragma unroll
                    for (int u = 0; u < T; ++u) {
                        if (!(grp >> u & 1u)) continue;
                        Scalar3 dir;
                        const float d = ref_tri_distance(tri, q[u], dir);
                        if (d < best[u]) {
                            best[u] = d;
                            at[u] = c;
                            id[u] = t;
                        }
                    }
                }
            }
        }
    }
    nd.Magnitude = 1e8f;
    nd.Direction = s3(0, 0, 0);
    nid = -1;
#pragma unroll
    for (int t = 0; t < T; ++t) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float d = __shfl_xor_sync(~0u, best[t], o);
            const int c = __shfl_xor_sync(~0u, at[t], o), i = __shfl_xor_sync(~0u, id[t], o);
            if (d < best[t] || (d == best[t] && c < at[t])) {
                best[t] = d;
                at[t] = c;
                id[t] = i;
            }
        }
        if (lane == t) nid = id[t];
    }
    if (nid != -1) nd.Magnitude = ref_tri_distance(ref_tri(b.triangles[nid]), p, nd.Direction);
}

// A lane per particle: the serial loop itself where its lists hold at most `most` entries in
// all (false: more, nothing done).  The 27 lengths are loaded nine at a time.
template <bool DRAG>
__device__ __forceinline__ bool ref_nearest_short(const RefBind& b, const Scalar3& p, bool live, unsigned most, CDistance& nd,
                                                  int& nid) {
    nd.Magnitude = 1e8f;
    nd.Direction = s3(0, 0, 0);
    nid = -1;
    int cx, cy, cz;
    const int cid = ref_cell(b.box, p, cx, cy, cz);
    if (!live || cid < 0 || cid >= b.cell_num) return true;
    auto key = [&](int c) {
        return cell_key(b.box.m_GridSize, (int)((unsigned)cx + (unsigned)(c % 3) - 1u),
                        (int)((unsigned)cy + (unsigned)(c / 3 % 3) - 1u), (int)((unsigned)cz + (unsigned)(c / 9) - 1u));
    };
    unsigned held = 0, some = 0;
#pragma unroll 9
    for (int c = 0; c < 27; ++c) {
        const int m = key(c);
        const unsigned len = m >= 0 && m < b.cell_num ? min(b.cells[m].m_TriangleNum, (unsigned)CELLMAXTRIANGLENUM) : 0u;
        held += len;
        if (len) some |= 1u << c;
    }
    if (held > most) return false;
    int met0 = -1, met1 = -1;   // triangles met last: one met before is never the nearer one
    while (some) {
        const CCell& cell = b.cells[key(__ffs(some) - 1)];
        some &= some - 1u;
        const int len = (int)min(cell.m_TriangleNum, (unsigned)CELLMAXTRIANGLENUM);
        for (int l = 0; l < len; ++l) {
            const int t = cell.m_TriangleID[l];
            if (t < 0 || t >= b.triangle_num || t == nid || t == met0 || t == met1) continue;
            met1 = met0;
            met0 = t;
            if (DRAG && !b.tri_params[b.triangles[t].ModelIDNumber].isDrag) continue;
            Scalar3 dir;
            const float d = ref_tri_distance(ref_tri(b.triangles[t]), p, dir);
            if (d < nd.Magnitude) {
                nd.Magnitude = d;
                nd.Direction = dir;
                nid = t;
            }
        }
    }
    return true;
}
constexpr int kNearLeft = -2;   // mark of the particles that the lane per particle leaves

// The two launches of a call of which the first does the short lists: the second one may start
// when every CTA of the first has (programmatic dependent launch) and waits for what they wrote.
__device__ __forceinline__ void near_next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void near_wait_for_marks() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// particles of a CTA of four warps: kNearT to a warp, or LEFT marks (a multiple of 32) of which
// the warps share those that are set
template <int LEFT>
constexpr int near_particles() { return LEFT ? LEFT : 4 * kNearT; }
// work(id, mine): a warp's kNearT particles, one in each of its first lanes; LEFT: those with
// the mark alone (mark[id] == kNearLeft)
template <int LEFT, class Work>
__device__ __forceinline__ void near_groups(int n, const int* mark, Work&& work) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, first = blockIdx.x * near_particles<LEFT>();
    if constexpr (!LEFT) {
        const int id = first + warp * kNearT + lane;
        work(id, lane < kNearT && id < n);
    } else {
        __shared__ int list[LEFT];
        near_wait_for_marks();
        int count = 0;
#pragma unroll
        for (int k = 0; k < LEFT / 32; ++k) {   // the same in every warp
            const int id = first + 32 * k + lane;
            const bool on = id < n && mark[id] == kNearLeft;
            const unsigned found = __ballot_sync(~0u, on);
            if (on && warp == k) list[count + __popc(found & ((1u << lane) - 1u))] = id;
            count += __popc(found);
        }
        if (count == 0) return;
        __syncthreads();
        for (int g = warp * kNearT; g < count; g += 4 * kNearT) {
            const bool mine = lane < kNearT && g + lane < count;
            work(mine ? list[g + lane] : 0, mine);
        }
    }
}

// CalcSTLDistance_Kernel (DeviceProcess_Kernel.h:853-919): a warp for kNearT particles, those
// that k_ref_stl_short has left, or all
template <int LEFT>
__global__ void __launch_bounds__(128, 8) k_ref_stl_distance(int n, const __grid_constant__ RefBind b) {
    near_groups<LEFT>(n, b.stl_id, [&](int id, bool mine) {
        CDistance nd;
        int nid;
        ref_nearest<false>(b, mine ? b.pos[id] : s3(0, 0, 0), mine, nd, nid);
        if (!mine) return;
        b.stl_distance[id] = nd;
        b.stl_id[id] = nid;
    });
}
__global__ void __launch_bounds__(128) k_ref_stl_short(int n, unsigned most, const __grid_constant__ RefBind b) {
    near_next_may_start();
    const int id = blockIdx.x * 128 + threadIdx.x;
    if (id >= n) return;
    CDistance nd;
    int nid;
    if (ref_nearest_short<false>(b, b.pos[id], true, most, nd, nid)) b.stl_distance[id] = nd;
    else nid = kNearLeft;
    b.stl_id[id] = nid;
}

// CalcDragEffect_Kernel and mode helpers (DeviceProcess_Kernel.h:125-389), with the
// reference's index use and brace placement (mode 'F' acts outside the region).
__device__ __forceinline__ void ref_drag_finish(const RefBind& b, int id, bool gone, const CDistance& nd, int nid) {
    const CParameter& P = b.param;
    if (b.magnifier_count[id] > 0) b.magnifier_count[id]++;
    if (b.magnifier_count[id] == 10) b.magnifier_count[id] = 0;
    if (gone) {
        b.stl_distance[id] = nd;
        b.stl_id[id] = nid;
    }
    b.drag_acc[id] = s3(0, 0, 0);
    b.drag_temperature[id] = 0;
    b.out_type[id] = TYPE_HEAVY_WEIGHT;
    if (!(nid != -1 && nd.Magnitude != 1e8f)) return;
    const DragParameter dp = b.drag_params[b.tri_params[b.triangles[nid].ModelIDNumber].DragTriangleID];
    if (nd.Magnitude <= dp.CoefficientofInflueneRegion * P.InitialParticleDistance) {
        b.out_type[id] = TYPE_LIGHT_WEIGHT;
        if (dp.DragToken == 'E') {
            if (dp.InputVelocityToken1 == 'V' || dp.InputVelocityToken1 == 'B') {
                float pr = 0.0f;
                const float sv = ref_mag(b.vel[id]);
                pr += dp.VelocityIndex * powf(sv, dp.VelocityExponential);
                const Scalar3 nrm = b.triangles[nid].Normal;
                if (dp.VelocityDragPermiabilityConstant != 0)
                    b.drag_acc[id] = s3((pr * (nrm.x) / dp.VelocityDragPermiabilityConstant),
                                        (pr * (nrm.y) / dp.VelocityDragPermiabilityConstant),
                                        (pr * (nrm.z) / dp.VelocityDragPermiabilityConstant));
            } else if (dp.InputVelocityToken1 == 'T') {
                const float sv = ref_mag(b.vel[id]);
                const float enth = dp.TempIndex * powf(sv, dp.TempExponential);
                const float den = ref_mag(b.vel[id]) * P.Density * P.FruidSpecificHeat;
                if (den != 0)
                    b.drag_temperature[id] = (enth * dp.TempDragPermiabilityConstant * P.Dt * P.ThermalStep) / (den);
                b.out_solid_rate[id] = b.drag_temperature[id];
            }
        } else if (dp.DragToken == 'C') {
            if (dp.InputVelocityToken1 == 'V' || dp.InputVelocityToken1 == 'v') {
                b.out_vel[id] = s3(dp.ConstantVx, dp.ConstantVy, dp.ConstantVz);
                b.vel[id] = s3(dp.ConstantVx, dp.ConstantVy, dp.ConstantVz);
            }
        }
    } else if (dp.DragToken == 'F') {
        if ((dp.InputVelocityToken1 == 'V' || dp.InputVelocityToken1 == 'v') && b.magnifier_count[id] < 1) {
            const float f = dp.VelocityMagnitueFactor;
            b.vel[id].x *= f; b.vel[id].y *= f; b.vel[id].z *= f;
            b.out_vel[id].x *= f; b.out_vel[id].y *= f; b.out_vel[id].z *= f;
        }
    }
}
// as k_ref_stl_distance and k_ref_stl_short
template <int LEFT>
__global__ void __launch_bounds__(128, 8) k_ref_drag(int n, const __grid_constant__ RefBind b) {
    near_groups<LEFT>(n, b.out_type, [&](int id, bool mine) {
        const bool gone = mine && b.out_id[id] < -1;
        CDistance nd;
        int nid;
        ref_nearest<true>(b, mine ? b.pos[id] : s3(0, 0, 0), mine && !gone, nd, nid);
        if (mine) ref_drag_finish(b, id, gone, nd, nid);
    });
}
__global__ void __launch_bounds__(128) k_ref_drag_short(int n, unsigned most, const __grid_constant__ RefBind b) {
    near_next_may_start();
    const int id = blockIdx.x * 128 + threadIdx.x;
    if (id >= n) return;
    const bool gone = b.out_id[id] < -1;
    CDistance nd;
    int nid;
    if (ref_nearest_short<true>(b, b.pos[id], !gone, most, nd, nid)) ref_drag_finish(b, id, gone, nd, nid);
    else b.out_type[id] = kNearLeft;
}

// ---------------------------------------------------------------------------
// particle operators (explicit schedule)
// ---------------------------------------------------------------------------
// Neighbours of a target: the particles of its 27 cells, k outer, j, i inner, a cell's
// in sorted order, closer than re (the temperature operator: at most re); particles whose
// out_id (indexed by sorted position, as in the reference) is negative are skipped.
// Screen: ref_sqrt never returns less than sqrt(x) (1 - 3e-7) (its Newton step from
// below gives y <= 1/sqrt(x), the float roundings cost a few ulps), so a finite squared
// distance >= re^2 (1 + 1e-5) is rejected by the reference's own test and is skipped
// before the square root; the others take the reference's arithmetic unchanged
// (+inf is not screened: the reference's sqrt of it is -0, which it accepts).
__device__ __forceinline__ float ref_screen2(float re) { return re * re * 1.00001f; }

}  // namespace mps
#include "ref_pairs.cuh"
namespace mps {

// Before and after the pair sums of one operator, run by the target's own lane.
// begin: false if the target is done (outside the compute zone, or without a cell where
// the operator needs one); `walk` says whether it has neighbours to sum.
template <class Op>
struct RefOp;

// CalcExplicitly_Kernel (DeviceProcess_Kernel.h:390-582)
template <>
struct RefOp<RpExplicitly> {
    static __device__ __forceinline__ float radius(const CParameter& P) {
        return P.LaplacianInfluenceRadiusCoefficient * P.InitialParticleDistance;
    }
    static __device__ __forceinline__ bool begin(const RefBind& b, int id, RpTarget& t, int& cx, int& cy, int& cz,
                                                 bool& walk) {
        if (!in_zone<float>(b.box, t.pos.x, t.pos.y, t.pos.z, b.param.Tolerance)) {
            const int orig = b.id[id];
            b.out_id[orig] = -1;
            b.out_solid_rate[orig] = 9999;
            return false;
        }
        t.vel = b.vel[id];
        t.s = b.param.bTurbulance ? b.strain[id] : 0.0f;
        const int cid = ref_cell(b.box, t.pos, cx, cy, cz);
        walk = cid >= 0 && cid < b.cell_num;
        return true;
    }
    // coef = (float)(2 Dimension / (double)(lambda n0)), from the host
    static __device__ __forceinline__ void finish(const RefBind& b, int id, const RpTarget& t, const float (&sum)[3],
                                                  const float (&rare)[9], float coef) {
        const CParameter& P = b.param;
        const int orig = b.id[id];
        const Scalar3 tp = t.pos;
        Scalar3 v0 = t.vel;
        Scalar3 lap = s3(sum[0], sum[1], sum[2]);
        const Scalar3 art = s3(rare[0], rare[1], rare[2]), col = s3(rare[3], rare[4], rare[5]);
        const float re = radius(P);
        const float wd = b.stl_distance[id].Magnitude;
        const int tri = b.stl_id[id];
        if (tri >= 0 && tri < b.triangle_num && wd > 0 && wd < re) {
            const float ww = ref_zlap(P.Dimension, wd, P.InitialParticleDistance);
            const Scalar3 v1 = b.tri_params[b.triangles[tri].ModelIDNumber].Velocity;
            lap.x += P.WallFrictionCoeffieicnt * (v1.x - v0.x) * ww;
            lap.y += P.WallFrictionCoeffieicnt * (v1.y - v0.y) * ww;
            lap.z += P.WallFrictionCoeffieicnt * (v1.z - v0.z) * ww;
        }
        lap.x *= coef; lap.y *= coef; lap.z *= coef;
        Scalar3 dragv = s3(0, 0, 0);
        Scalar3 acc = s3add(s3(0, 0, 0), P.GravityConstant);
        if (b.drag_num > 0) dragv = b.drag_acc[id];
        // laminar + turbulent viscosity (:545-552)
        lap = s3mul(lap, P.bTurbulance ? b.kin_visc[id] + b.turb_visc[id] : b.kin_visc[id]);
        acc = s3add(acc, lap);
        v0 = s3sub(s3add(v0, s3mul(acc, P.Dt)), dragv);
        if (P.bTurbulance) {
            // (2/3) is the integer quotient 0 in the reference (:560): the term vanishes
            const Scalar3 tke = s3mul(s3(rare[6], rare[7], rare[8]), (float)(2 / 3));
            v0 = s3sub(v0, s3mul(tke, P.Dt));
        }
        if (P.bExplicitPressure) {
            const float c = (float)(-P.Dimension) / (P.ConstantParticleDensity * P.Density);
            acc = s3add(s3mul(art, c), s3mul(col, (float)0.01));
            v0 = s3add(v0, s3mul(acc, P.Dt));
        }
        if (isfinite(v0.x) && isfinite(v0.y) && isfinite(v0.z)) {
            b.out_pos[orig] = s3(tp.x + P.Dt * v0.x, tp.y + P.Dt * v0.y, tp.z + P.Dt * v0.z);
            b.out_vel[orig] = v0;
        }
    }
};

// CalcTemperatureFactor_Kernel (DeviceProcess_Kernel.h:705-852): conduction over the
// neighbours within the temperature radius (distance <= re), the nearest wall through
// its gradient Z function, the drag heating; each sum counted only above FLT_EPSILON
// in magnitude; clamped; viscosity linear in the temperature (original index)
template <>
struct RefOp<RpTemperature> {
    static __device__ __forceinline__ float radius(const CParameter& P) {
        return P.TemperatureInfluenceRadiusCoefficient * P.InitialParticleDistance;
    }
    static __device__ __forceinline__ bool begin(const RefBind& b, int id, RpTarget& t, int& cx, int& cy, int& cz,
                                                 bool& walk) {
        if (!in_zone<float>(b.box, t.pos.x, t.pos.y, t.pos.z, b.param.Tolerance)) {
            b.out_id[b.id[id]] = -1;
            return false;
        }
        t.s = b.temperature[id];
        const int cid = ref_cell(b.box, t.pos, cx, cy, cz);
        return walk = cid >= 0 && cid < b.cell_num;
    }
    static __device__ __forceinline__ void finish(const RefBind& b, int id, const RpTarget& t, const float (&sum)[1],
                                                  const float (&)[1], float) {
        const CParameter& P = b.param;
        const int orig = b.id[id];
        const float ecoef = P.Dt * 2 * P.Dimension / (P.ConstantParticleDensity * P.Density * P.FruidSpecificHeat);
        const float ret = radius(P), hf = sum[0];
        float tt = t.s, hw = 0.0f;
        const float wd = b.stl_distance[id].Magnitude;
        const int tri = b.stl_id[id];
        if (tri >= 0 && tri < b.triangle_num && wd > 0 && wd < ret) {
            const CTriangleParameters& tq = b.tri_params[b.triangles[tri].ModelIDNumber];
            const float res = tq.WallThermalResistivity;
            const float cond = (2 * P.FruidThermalConductivity * tq.WallThermalConductivity) /
                               (P.FruidThermalConductivity + tq.WallThermalConductivity);
            const float ww = ref_zgrad(P.Dimension, wd, P.InitialParticleDistance);
            const float num = (tq.Temperature - tt) * ww;
            const float den = wd * wd * (1 / cond + res / wd);
            hw = num / den;
        }
        if (b.drag_num > 0) tt += b.drag_temperature[id];
        float comb = 0.0f;
        if (fabsf(hf) > FLT_EPSILON) comb += hf;
        if (fabsf(hw) > FLT_EPSILON) comb += hw;
        tt += (ecoef * (comb));
        if (tt > P.MaxWallTemperature) tt = P.MaxWallTemperature;
        if (tt < P.MinWallTemperature) tt = P.MinWallTemperature;
        b.out_temperature[orig] = tt;
        b.out_kin_visc[orig] = P.ViscosityUpdateParameterA * tt + P.ViscosityUpdateParameterB;
    }
};

// CalcTurbulenceViscosity_Kernel (DeviceProcess_Kernel.h:1273-1476): velocity gradient
// tensor within the gradient radius, strain-rate product, wall-damped Smagorinsky
// viscosity (capped) and turbulent kinetic energy (capped), sorted order.  The
// kernel's vorticity and PND are never read and are left out.
template <>
struct RefOp<RpTurbulence> {
    static __device__ __forceinline__ float radius(const CParameter& P) {
        return P.GradientInfluenceRadiusCoefficient * P.InitialParticleDistance;
    }
    static __device__ __forceinline__ bool begin(const RefBind& b, int id, RpTarget& t, int& cx, int& cy, int& cz,
                                                 bool& walk) {
        if (!in_zone<float>(b.box, t.pos.x, t.pos.y, t.pos.z, b.param.Tolerance)) {
            b.turb_visc[id] = 0.0f;
            b.out_id[b.id[id]] = -1;
            return false;
        }
        t.vel = b.vel[id];
        const int cid = ref_cell(b.box, t.pos, cx, cy, cz);
        if (cid < 0 || cid >= b.cell_num) {
            b.pressure[id] = 0.0f;
            return false;
        }
        return walk = true;
    }
    static __device__ __forceinline__ void finish(const RefBind& b, int id, const RpTarget&, const float (&sum)[9],
                                                  const float (&)[1], float) {
        const CParameter& P = b.param;
        Scalar3 X = s3(sum[0], sum[1], sum[2]), Y = s3(sum[3], sum[4], sum[5]), Z = s3(sum[6], sum[7], sum[8]), D;
        const float re = radius(P);
        const float g = P.Dimension / P.ConstantParticleDensity;
        X.x = g * X.x; X.y = g * X.y; X.z = g * X.z;
        Y.x = g * Y.x; Y.y = g * Y.y; Y.z = g * Y.z;
        Z.x = g * Z.x; Z.y = g * Z.y; Z.z = g * Z.z;
        D.x = (float)(0.5 * (X.y + Y.x));
        D.y = (float)(0.5 * (X.z + Z.x));
        D.z = (float)(0.5 * (Y.z + Z.y));
        const float strain = X.x * X.x + Y.y * Y.y + Z.z * Z.z + 2 * D.x * D.x + 2 * D.y * D.y + 2 * D.z * D.z;
        const float riw = b.stl_distance[id].Magnitude;
        const float ratio = -(riw / re);
        const float damp = 1 - expf(ratio);
        const float smag = P.SmagorinskyConstant * damp;
        const float coef = (smag * P.FilterWidth) * (smag * P.FilterWidth);
        float tv = 0;
        if (strain > 0) tv = coef * sqrtf(2 * strain);
        if (tv > P.TurbulanViscosityRatio) tv = P.TurbulanViscosityRatio;
        b.turb_visc[id] = tv;
        const float tkc = 2 * P.Cnue * P.InitialParticleDistance * P.InitialParticleDistance / P.Cepsilon;
        float tke = strain * tkc;
        if (tke > P.TurbulanceIntensity) tke = P.TurbulanceIntensity;
        b.strain[id] = tke;
    }
};

// CalcExplicitPressure_Kernel (DeviceProcess_Kernel.h:921-1054)
template <>
struct RefOp<RpPressure> {
    static __device__ __forceinline__ float radius(const CParameter& P) {
        return P.GradientInfluenceRadiusCoefficient * P.InitialParticleDistance;
    }
    static __device__ __forceinline__ bool begin(const RefBind& b, int id, RpTarget& t, int& cx, int& cy, int& cz,
                                                 bool& walk) {
        if (!in_zone<float>(b.box, t.pos.x, t.pos.y, t.pos.z, b.param.Tolerance)) {
            b.out_id[b.id[id]] = -1;
            b.pressure[id] = 0.0f;
            return false;
        }
        const int cid = ref_cell(b.box, t.pos, cx, cy, cz);
        if (cid < 0 || cid >= b.cell_num) {
            b.pressure[id] = 0.0f;
            return false;
        }
        return walk = true;
    }
    static __device__ __forceinline__ void finish(const RefBind& b, int id, const RpTarget&, const float (&sum)[1],
                                                  const float (&)[1], float) {
        const CParameter& P = b.param;
        const int orig = b.id[id];
        const float re = radius(P);
        const float coef = P.SonicVelocity * P.SonicVelocity * P.Density / P.ConstantParticleDensity;
        float dens = sum[0];
        const float riw = b.stl_distance[id].Magnitude;
        float ww = 0.0f;
        if (b.stl_id[id] >= 0 && b.stl_id[id] < b.triangle_num && riw >= 0 && riw <= re)
            ww = ref_zgrad(P.Dimension, riw, P.InitialParticleDistance);
        dens += ww;
        if (isfinite(dens)) b.out_density[orig] = dens;
        float pr = 0.0f;
        if (dens > P.ConstantParticleDensity * P.FreeSurfaceThreshold) pr = coef * (dens - P.ConstantParticleDensity);
        if (isfinite(pr)) {
            b.out_pressure[orig] = pr;
            b.pressure[id] = pr;
        }
    }
};

// CalcExplicitPressureGradient_Kernel (DeviceProcess_Kernel.h:1056-1271), without
// the negative-pressure branch.
template <>
struct RefOp<RpGradient> {
    static __device__ __forceinline__ float radius(const CParameter& P) {
        return P.GradientInfluenceRadiusCoefficient * P.InitialParticleDistance;
    }
    static __device__ __forceinline__ bool begin(const RefBind& b, int id, RpTarget& t, int& cx, int& cy, int& cz,
                                                 bool& walk) {
        if (!in_zone<float>(b.box, t.pos.x, t.pos.y, t.pos.z, b.param.Tolerance)) {
            b.out_id[b.id[id]] = -1;
            return false;
        }
        t.s = b.pressure[id];
        const int cid = ref_cell(b.box, t.pos, cx, cy, cz);
        return walk = cid >= 0 && cid < b.cell_num;
    }
    static __device__ __forceinline__ void finish(const RefBind& b, int id, const RpTarget& t, const float (&sum)[3],
                                                  const float (&)[1], float) {
        const CParameter& P = b.param;
        const int orig = b.id[id];
        const Scalar3 tp = t.pos;
        const float re = radius(P), tpress = t.s;
        Scalar3 gf = s3(sum[0], sum[1], sum[2]), gw = s3(0, 0, 0);
        const float c1 = 2 * P.Dimension / (P.ConstantParticleDensity);
        const float c2 = P.Density / (P.Dt * P.Dt);
        const float c3 = -P.Dt / P.Density;
        gf.x *= c1; gf.y *= c1; gf.z *= c1;
        const CDistance riw = b.stl_distance[id];
        if (b.stl_id[id] >= 0 && b.stl_id[id] < b.triangle_num) {
            if (riw.Magnitude > 0 && riw.Magnitude <= re) {
                const float ww = ref_z(c_zgrad3, 21, riw.Magnitude, P.InitialParticleDistance);
                const float wc = (float)((((0.5 * (double)c1) * (double)ww) * (double)tpress) /
                                         (double)(riw.Magnitude * riw.Magnitude));
                gw = s3(wc * (-riw.Direction.x), wc * (-riw.Direction.y), wc * (-riw.Direction.z));
            }
            if (riw.Magnitude > 0 && riw.Magnitude <= P.InitialParticleDistance * P.OffSet) {
                const float dr = (P.InitialParticleDistance * P.OffSet - riw.Magnitude);
                const float mc = c2 * dr / riw.Magnitude;
                gw.x += mc * (-riw.Direction.x);
                gw.y += mc * (-riw.Direction.y);
                gw.z += mc * (-riw.Direction.z);
            }
        }
        const Scalar3 g = s3add(s3add(gf, gw), s3(0, 0, 0));
        Scalar3 iv = s3(c3 * g.x, c3 * g.y, c3 * g.z);
        if (isfinite(iv.x) && isfinite(iv.y) && isfinite(iv.z)) {
            const Scalar3 v = b.vel[id];
            Scalar3 ov = s3(v.x + iv.x, v.y + iv.y, v.z + iv.z);
            // CorrectVelocity (Utility_Inline.h:2369-2396)
            const float cmax = P.InitialParticleDistance * P.CourantNumber / P.Dt;
            const float a = ref_sqrt(ov.x * ov.x + ov.y * ov.y + ov.z * ov.z);
            if (a > cmax) ov = s3(cmax * ov.x / a, cmax * ov.y / a, cmax * ov.z / a);
            b.out_vel[orig] = ov;
            iv = s3(ov.x - v.x, ov.y - v.y, ov.z - v.z);
            b.out_pos[orig] = s3(tp.x + iv.x * P.Dt, tp.y + iv.y * P.Dt, tp.z + iv.z * P.Dt);
        }
    }
};

// Two launches share a large call: one of k_ref_pairs and k_ref_slices takes it in dense fluid,
// k_ref_walk_sparse after it in sparse fluid, and the other one of the two has nothing to do
// (rp_sparse).  k_ref_walk_sparse may start once every CTA of the first has (programmatic dependent
// launch: neither reads what the other writes), and every thread of it ends after the
// first launch has, so what follows in the stream follows both.
__device__ __forceinline__ void ref_beside_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void ref_beside_end() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// One operator over targets 0 .. n-1, T per warp; with four, a warp takes `per` groups one after
// another, its CTA's next to each other (rp_per)
template <class Op, int T>
__global__ void __launch_bounds__(kRpWarps * 32, T == 2 ? 6 : Op::NX > 0 || Op::NS > 3 ? 5 : 7) k_ref_pairs(int n, float coef, float minus_zero, int sparse, int per,
                                                               const __grid_constant__ RefBind b) {
    using W = RpWarp<Op, T>;
    __shared__ __align__(16) float sm[kRpWarps * W::kFloats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ref_beside_start();
    if (sparse > 0 && rp_sparse(b, n, sparse)) return;
    auto group = [&](int first) {
        const int id = first + lane;
        RpTarget t{};
        int cx = 0, cy = 0, cz = 0;
        bool walk = false, fin = false;
        if (lane < T && id < n) {
            t.pos = b.pos[id];
            fin = RefOp<Op>::begin(b, id, t, cx, cy, cz, walk);
        }
        W w(b, sm + warp * W::kFloats, RefOp<Op>::radius(b.param), minus_zero, first, t);
        w.run(b, walk && fin, cx, cy, cz);
        float sum[Op::NS], rare[W::NXR];
#pragma unroll
        for (int c = 0; c < Op::NS; ++c) sum[c] = w.sum(c);
        if constexpr (Op::NX > 0) {
#pragma unroll
            for (int c = 0; c < Op::NX; ++c) rare[c] = w.rare_sum(c);
        }
        if (fin) RefOp<Op>::finish(b, id, t, sum, rare, coef);
    };
    if constexpr (T == 4) {
#pragma unroll 1
        for (int r = 0; r < per; ++r) {
            const int first = ((blockIdx.x * per + r) * kRpWarps + warp) * T;
            if (first >= n) return;
            group(first);
            __syncwarp();
        }
    } else {
        const int first = (blockIdx.x * kRpWarps + warp) * T;
        if (first < n) group(first);
    }
}

// a lane per target
template <class Op>
__device__ __forceinline__ void ref_walk(const RefBind& b, int id, float coef, int2* run) {
    RpTarget t{};
    int cx = 0, cy = 0, cz = 0;
    bool walk = false;
    t.pos = b.pos[id];
    if (!RefOp<Op>::begin(b, id, t, cx, cy, cz, walk)) return;
    float sum[Op::NS], rare[RpShape<Op>::NXR];
    rp_walk_sums<Op>(b, t, id, walk, cx, cy, cz, RefOp<Op>::radius(b.param), run, 128, sum, rare);
    RefOp<Op>::finish(b, id, t, sum, rare, coef);
}
template <class Op>
__global__ void __launch_bounds__(128) k_ref_walk(int n, float coef, const __grid_constant__ RefBind b) {
    __shared__ int2 run[9][128];
    const int id = blockIdx.x * 128 + threadIdx.x;
    if (id < n) ref_walk<Op>(b, id, coef, &run[0][threadIdx.x]);
}
// ... if the kernel beside it leaves them
template <class Op>
__global__ void __launch_bounds__(128) k_ref_walk_sparse(int n, float coef, int sparse, const __grid_constant__ RefBind b) {
    __shared__ int2 run[9][128];
    // one share: as a condition instead of a loop the same work took 890 us instead of 792
    // (pressure, 882,000 particles, 40 % of them in dense fluid)
    if (rp_sparse(b, n, sparse))
        for (int id = blockIdx.x * 128 + threadIdx.x; id < n; id += gridDim.x * 128)
            ref_walk<Op>(b, id, coef, &run[0][threadIdx.x]);
    ref_beside_end();
}

// 32 targets per warp, operators without rarer pairs
template <class Op>
constexpr int rs_warps() { return Op::NS == 1 ? 4 : 2; }
template <class Op>
__global__ void __launch_bounds__(rs_warps<Op>() * 32) k_ref_slices(int n, float minus_zero, int sparse,
                                                                  const __grid_constant__ RefBind b) {
    using W = RpSlice<Op>;
    __shared__ __align__(16) float sm[rs_warps<Op>() * W::kFloats];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = (blockIdx.x * rs_warps<Op>() + warp) * 32;
    ref_beside_start();
    if ((sparse > 0 && rp_sparse(b, n, sparse)) || first >= n) return;
    const int id = first + lane;
    RpTarget t{};
    int cx = 0, cy = 0, cz = 0;
    bool walk = false, fin = false;
    if (id < n) {
        t.pos = b.pos[id];
        fin = RefOp<Op>::begin(b, id, t, cx, cy, cz, walk);
    }
    W w(sm + warp * W::kFloats, RefOp<Op>::radius(b.param), minus_zero, first, t);
    w.run(b, walk && fin, cx, cy, cz);
    float sum[Op::NS];
    const float none[1] = {0.0f};
#pragma unroll
    for (int c = 0; c < Op::NS; ++c) sum[c] = w.sum(c);
    if (fin) RefOp<Op>::finish(b, id, t, sum, none, 0.0f);
}

inline int grid_of(int n) { return div_up(n, kBlock); }

// From here on a warp takes 32 targets of the pressure, its gradient and the temperature (us,
// k_ref_pairs / k_ref_slices): pressure 58 / 60 at 32,768 particles, 104 / 64 at 64,000,
// 1,160 / 437 at 884,736; gradient 130 / 101 and 1,406 / 884; temperature 112 / 89 and
// 1,248 / 642.  The predictor accepts seven times as many pairs and empties its lists too
// often (3,120 / 3,514 at 884,736); the turbulence has nine sums.
constexpr int kRefSlices = 40000;

// From here on a call asks first whether the fluid is sparse and leaves it to k_ref_walk if so.
// The kernels that share candidates between targets have little to share there, and a warp
// per few targets is 8 to 32 times fewer targets at a time (us, without and with k_ref_walk,
// 0.03 particles per cube of the particle distance): pressure 1,262 / 173 at 882,000
// particles, 198 / 33 at 50,000, 50 / 30 at 19,000, 38 / 32 at 10,000; turbulence 2,353 / 245 at
// 882,000, predictor 311 / 69 at 110,000.  In dense fluid the question and the second launch
// cost 1 to 4 % (pressure 77.7 / 79.5 at 103,823, gradient 151 / 153, turbulence 2,215 / 2,269 at
// 884,736); at 15,625 they would cost 8 % of the pressure.
constexpr int kRefSplit = 16384;
// Particles per cell below which k_ref_walk is the faster one.  Measured on random fluid of
// 0.004 to 1 per cube of the distance (64 such cubes are a cell), us at the densities on both
// sides of the line, kernel that shares / k_ref_walk: pressure (slices) 0.15: 581 / 386, 0.3:
// 383 / 626 at 882,000; eight targets per warp 0.06: 65 / 42, 0.15: 48 / 71 at 30,000;
// turbulence (four per warp) 0.5: 2,015 / 1,570, 1.0: 2,882 / 2,839 at 882,000; predictor 0.1:
// 96 / 95 at 30,000 and 0.2: 257 / 210, 0.3: 280 / 282 at 110,000.
template <class Op>
int rp_few(int n, bool slices, bool pairs2) {
    if (slices) return 15;
    if (std::is_same<Op, RpTurbulence>::value && !pairs2) return 40;
    if (n < 40000) return 7;
    return std::is_same<Op, RpExplicitly>::value && n >= 64000 ? 16 : 10;
}

// Four targets per warp are so many CTAs that starting them to find sparse fluid took a tenth of
// the call: a CTA takes several groups while 40 CTAs per SM (eight rounds of five) are left.
// us at 882,000 particles, one group / about twelve rounds / six / three: turbulence at 0.01 per
// cube 201 / 158 / 153 / 151, at 1.0 2,906 / 2,896 / 2,932 / 3,012; at 300,000 76 / 67 / 62 / 60 and
// 979 / 983 / 1,001 / 1,024.
inline int rp_per(int groups) { return std::max(1, groups / (152 * 40)); }

// Beside the launch before it.  With one wave of CTAs that take several shares each it left the
// GPU idle at the end (us, a wave / a CTA per share at 882,000 particles: pressure at 0.15 per
// cube 428 / 386, gradient with 40 % of the particles in dense fluid 1,411 / 1,252); in dense
// fluid, where all it does is ask, the two are alike (558).
template <class Op>
cudaError_t ref_walk_beside(cudaStream_t st, int n, float coef, int sparse) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)div_up(n, 128));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return MPS_COUNT_LAUNCH cudaLaunchKernelEx(&cfg, k_ref_walk_sparse<Op>, n, coef, sparse, (const RefBind)g_bind);
}

// Targets per warp of an operator: kMany share each round's candidates; below `few` of
// them that leaves too few warps per SM and two per warp finish sooner.  Measured in us,
// two against kMany, on a jittered block: pressure 50 / 54 at 15,625 particles, 72 / 54
// at 32,768; turbulence (9 sums, 4 per warp) 90 / 107 at 32,768, 297 / 296 at 103,823.
template <class Op, int kMany>
cudaError_t ref_op_launch(cudaStream_t st, int n, int few, float coef = 0.0f) {
    constexpr bool kSlices = std::is_same<Op, RpPressure>::value || std::is_same<Op, RpGradient>::value ||
                             std::is_same<Op, RpTemperature>::value;
    // 0: not asked, since the call is small or all cells of the grid hold that many on average
    int sparse = n < kRefSplit ? 0 : rp_few<Op>(n, kSlices && n >= kRefSlices, n < few);
    if ((long long)n >= (long long)sparse * g_bind.cell_num) sparse = 0;
    if (n < few) {
        MPS_COUNT_LAUNCH k_ref_pairs<Op, 2><<<div_up(n, kRpWarps * 2), kRpWarps * 32, 0, st>>>(n, coef, -0.0f, sparse, 1, g_bind);
    } else if (kSlices && n >= kRefSlices) {
        if constexpr (kSlices) {
            constexpr int W = rs_warps<Op>();
            MPS_COUNT_LAUNCH k_ref_slices<Op><<<div_up(n, W * 32), W * 32, 0, st>>>(n, -0.0f, sparse, g_bind);
        }
    } else {
        const int groups = div_up(n, kRpWarps * kMany), per = kMany == 4 && sparse ? rp_per(groups) : 1;
        MPS_COUNT_LAUNCH k_ref_pairs<Op, kMany><<<div_up(groups, per), kRpWarps * 32, 0, st>>>(n, coef, -0.0f, sparse, per, g_bind);
    }
    const cudaError_t e = cudaGetLastError();
    return e || sparse == 0 ? e : ref_walk_beside<Op>(st, n, coef, sparse);
}
// Below it a triangle is walked by 32 lanes (few triangles are large ones), else by 8 (us, a
// registration with 32 / 8: 12 large triangles 162 / 209, 576 of a cylinder 95 / 105, 2,048 94 / 102,
// 4,096 83 / 83, or 118 / 132 over cells half the size, 9,216 101 / 88).
constexpr int kTriFew = 2048;
// Wall distance and drag: most particles of a large set see few triangles or none, and a warp
// per four of them is then most of the time.  With 64,000 particles and 100 for every
// triangle a lane per particle does the short lists first.  us, wall distance then drag, a
// thread per particle (its divisions in FP64) / a warp per four / both in turn: no triangles near
// 882,000 particles 44 / 101 / 29, 110,000 14 / 17 / 8, 16,000 14 / 7 / 10; the line: 9,216 with drag
// spheres among 882,080 (96 to one) 539 / 347 / 350, 4,176 among 513,279 (123 to one) 211 / 136 / 130,
// among 318,675 (76 to one) 240 / 108 / 125.
// Up to how many entries, and how many of the others' marks a CTA of the second launch looks at
// (near_marks): 32 and 32, or 64 and 64 with 200 particles for every triangle, whose lists repeat the few
// triangles around and leave fewer particles (us, thread per particle / 32 / 64): 12 triangles
// around 65,536 38.0, 14.5 / 36.6, 16.5 / 24.7, 12.6, around 1,000,000 88.8, 50.6 / 84.7, 57.6 /
// 63.5, 45.3; 4,096 around 882,080 (215 to one) 176.5, 57.4 / 159.9, 65.6 / 147.8, 52.5; the 123 to
// one above 211, 158 / 130, 90 / 194, 144; 9,216 among 1,117,134 (121 to one) 613, 548 / 374, 326 /
// 425, 376.
// From 600,000 particles on 50 for every triangle are enough: the lanes fill the GPU, so a list
// costs what it holds and not its latency, from 2,000,000 on up to 128 entries (thread per particle /
// warps / 32 / 128: a cylinder of 16,128 triangles around 882,080 327, 82 / 248, 123 / 231, 78 / 272,
// 72; four cylinders and 512 spheres, 58,624, among 3,178,892 1,330, 780 / 1,425, 1,178 / 1,251, 999 /
// 1,248, 794; 28,096 among 2,116,620 1,364, 1,293 / 1,131, 1,120 / 1,109, 1,114 / 1,190, 1,171; below
// the line, 28,096 among 1,236,510 (44 to one), 1,335, 1,282 / 933, 928 / 985, 987 / 1,094, 1,075).
int near_short_most(int n) {   // 0: no short lists first
    const int t = g_bind.triangle_num;
    if (n >= 600000 && n / 100 < t && n / 50 >= t) return n < 2000000 ? 32 : 128;
    if (n < 64000 || n / 100 < t) return 0;
    return n / 200 < t ? 32 : 64;
}
constexpr int near_marks(int most) { return most == 32 ? 32 : 64; }
template <class Left>
cudaError_t near_left_launch(cudaStream_t st, int n, int most, Left left) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)div_up(n, near_marks(most)));
    cfg.blockDim = dim3(128);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return MPS_COUNT_LAUNCH cudaLaunchKernelEx(&cfg, left, n, (const RefBind)g_bind);
}
constexpr int kRefFew = 20000, kRefFewTurbulence = 100000;
// From here on the predictor, whose radius is the cell size (250 of 1,728 candidates
// accepted), runs a lane per target whatever the density (us, eight targets per warp / a lane
// each, with turbulence): 642 / 707 at 157,464 particles, 876 / 885 at 216,000, 3,096 / 2,993
// at 884,736.
constexpr int kRefLanes = 216000;

CCTStatusType launch_status() { return cuda_status(cudaGetLastError()); }

}  // namespace mps

using namespace mps;

// ===========================================================================
// Reference-named C-ABI (DeviceProcess.h:78-120)
// ===========================================================================
extern "C" {

CCTStatusType InitializeDeviceMemConst(CParameter Parameter, Integer ParticleNum, CTriangle* Triangles,
                                       Integer TriangleNum, CTriangleParameters* TriangleParameters,
                                       Integer MaxParticleNum, CDistance* STLDistance, Integer* StlID, CCell* Cell,
                                       Integer CellNum, Integer* CellStart, Integer* CellEnd,
                                       Integer* GridParticleIndex, CGridBox BoundingBox) {
    g_bind.param = Parameter;
    g_bind.particle_num = ParticleNum;
    g_bind.triangles = Triangles;
    g_bind.triangle_num = TriangleNum;
    g_bind.tri_params = TriangleParameters;
    g_bind.max_particle_num = MaxParticleNum;
    g_bind.stl_distance = STLDistance;
    g_bind.stl_id = StlID;
    g_bind.cells = Cell;
    g_bind.cell_num = CellNum;
    g_bind.cell_start = CellStart;
    g_bind.cell_end = CellEnd;
    g_bind.grid_index = GridParticleIndex;
    g_bind.box = BoundingBox;
    return CCT_NOERR;
}

CCTStatusType InitializeDeviceConstOutPutParticles(Integer* OutputParticleID, Scalar3* OutputParticlePosition,
                                                   Scalar3* OutputParticleVelocity, Scalar* OutputParticlePressure,
                                                   Scalar* OutputParticleDensity, Scalar* OutputParticleTemperature,
                                                   Scalar* OutputParticleKineticViscosity,
                                                   Scalar* OutputParticleSolidPhaseRate,
                                                   ParticleType* OutputParticleType) {
    g_bind.out_id = OutputParticleID;
    g_bind.out_pos = OutputParticlePosition;
    g_bind.out_vel = OutputParticleVelocity;
    g_bind.out_pressure = OutputParticlePressure;
    g_bind.out_density = OutputParticleDensity;
    g_bind.out_temperature = OutputParticleTemperature;
    g_bind.out_kin_visc = OutputParticleKineticViscosity;
    g_bind.out_solid_rate = OutputParticleSolidPhaseRate;
    g_bind.out_type = (int*)OutputParticleType;
    return CCT_NOERR;
}

CCTStatusType InitializeDeviceConstInputParticles(Integer* InputParticleID, Scalar3* InputParticlePosition,
                                                  Scalar3* InputParticleVelocity, Scalar* InputParticlePressure,
                                                  Scalar* InputParticleDensity, Scalar* InputParticleTemperature,
                                                  Scalar* InputParticleKineticViscosity,
                                                  Scalar* InputParticleSolidPhaseRate, ParticleType* InputParticleType,
                                                  Scalar* ParticleTurbulaceViscosity,
                                                  Scalar* ParticleStrainTensorProduct) {
    g_bind.turb_visc = ParticleTurbulaceViscosity;
    g_bind.strain = ParticleStrainTensorProduct;
    g_bind.id = InputParticleID;
    g_bind.pos = InputParticlePosition;
    g_bind.vel = InputParticleVelocity;
    g_bind.pressure = InputParticlePressure;
    g_bind.density = InputParticleDensity;
    g_bind.temperature = InputParticleTemperature;
    g_bind.kin_visc = InputParticleKineticViscosity;
    g_bind.solid_rate = InputParticleSolidPhaseRate;
    g_bind.type = (int*)InputParticleType;
    return CCT_NOERR;
}

CCTStatusType ParticleNumberToConst(Integer ParticleNum) {
    g_bind.particle_num = ParticleNum;
    return CCT_NOERR;
}

CCTStatusType DragParametersToConst(DragParameter* InputDragParameter, Scalar3* InputDragAcc,
                                    Scalar* InputDragTemperature, Integer DragTriangleNum, Integer* MagnifierCount,
                                    CDragTriangle* DragTriangles) {
    g_bind.drag_params = InputDragParameter;
    g_bind.drag_acc = InputDragAcc;
    g_bind.drag_temperature = InputDragTemperature;
    g_bind.drag_num = DragTriangleNum;
    g_bind.magnifier_count = MagnifierCount;
    g_bind.drag_triangles = DragTriangles;
    return CCT_NOERR;
}

CCTStatusType CaculateCellIDandInitializeHash(cudaStream_t& Stream, Integer ParticleNum, Integer CellNum,
                                              int* dGridParticleHash, int* dGridParticleIndex,
                                              Scalar3* particlePosition) {
    (void)CellNum;
    if (ParticleNum <= 0) return CCT_NOERR;
    MPS_COUNT_LAUNCH k_ref_hash<<<grid_of(ParticleNum), kBlock, 0, Stream>>>(ParticleNum, g_bind.box, particlePosition,
                                                             dGridParticleHash, dGridParticleIndex);
    return launch_status();
}

CCTStatusType reorderDataAndFindCellStart(cudaStream_t& Stream, Integer numParticles, Integer numCells,
                                          int* gridParticleHash, int* gridParticleIndex, int* cellStart,
                                          int* cellEnd) {
    if (numParticles <= 0) return CCT_NOERR;
    MPS_CUDA_TRY(cudaMemsetAsync(cellStart, 0xff, sizeof(int) * (size_t)numCells, Stream));
    MPS_CUDA_TRY(cudaMemsetAsync(cellEnd, 0xff, sizeof(int) * (size_t)numCells, Stream));
    MPS_COUNT_LAUNCH k_ref_reorder<<<grid_of(numParticles), kBlock, 0, Stream>>>(numParticles, numCells, gridParticleHash,
                                                                 gridParticleIndex, cellStart, cellEnd, g_bind);
    return launch_status();
}

// tile sums of the multi-CTA scan (NULL when the slot cannot be had: one-CTA scan)
static unsigned* scan_sums(int slot) {
    return (unsigned*)scratch_get(slot, sizeof(unsigned) * scan_tile_sums_capacity());
}

// Words in host memory that the GPU can write: errors, read without a copy once the stream has
// been waited for, and counts that a call copies to the host (a copy to pageable memory
// waits for its stream inside the driver, where other threads' calls then wait too).
// NULL when they cannot be had.
enum { kErrSort = 0, kErrTriangles, kVisits, kRemoved, kHostWords };
static std::atomic<unsigned*> g_errors{nullptr};
static volatile unsigned* host_word(int which) {
    static unsigned* const words = [] {
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(unsigned) * kHostWords, cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            return (unsigned*)nullptr;
        }
        for (int k = 0; k < kHostWords; ++k) ((unsigned*)p)[k] = 0u;
        g_errors.store((unsigned*)p);
        return (unsigned*)p;
    }();
    return words ? words + which : nullptr;
}
// the triangle cells that an earlier RegisterTriangleTopology made are incomplete
static bool triangles_failed() {
    volatile unsigned* const e = g_errors.load(std::memory_order_relaxed);
    if (!e || !e[kErrTriangles]) return false;
    note_message("RegisterTriangleTopology: a grid barrier of its sort ran out, the triangle cells are incomplete");
    return true;
}

// thrust::sort_by_key replacement: stable LSD radix sort on the legacy default
// stream, keys of any int range.
CCTStatusType SortUsingThrust(Integer MaxParticleNum, Integer* daNumberHash, Integer* daNumberIndex) {
    const int n = MaxParticleNum;
    if (n <= 1) return CCT_NOERR;
    const ScratchTurn turn(ScratchTurn::kSort);
    cudaStream_t st = 0;
    void* scr = scratch_get(1, radix_scratch_bytes(n));
    if (!scr) return CCT_MEMERR;
    volatile unsigned* const err = host_word(kErrSort);
    if (!err) return CCT_MEMERR;
    MPS_CUDA_TRY(radix_sort_pairs(n, daNumberHash, daNumberIndex, -1, scr, (unsigned*)err, 1u, st));
    // thrust::sort_by_key with the default policy returns after the sort completed;
    // callers rely on that (they launch the reorder on their own stream next).
    MPS_CUDA_TRY(cudaStreamSynchronize(st));
    if (*err) {
        *err = 0u;
        note_message("SortUsingThrust: a grid barrier of the sort ran out");
        return CCT_CUDAERR;
    }
    return launch_status();
}

CCTStatusType StableSortUsingThrust(Integer MaxParticleNum, Integer* daNumberHash, Integer* daNumberIndex) {
    return SortUsingThrust(MaxParticleNum, daNumberHash, daNumberIndex);
}

CCTStatusType CheckParticleOutsideComputeZone(cudaStream_t& Stream, Integer* ParticleNum) {
    const int n = *ParticleNum;
    if (n <= 0) return CCT_NOERR;
    const ScratchTurn turn(ScratchTurn::kOutside, Stream);
    unsigned* flag = (unsigned*)scratch_get(2, sizeof(unsigned) * ((size_t)n + 4));
    unsigned* rank = (unsigned*)scratch_get(3, sizeof(unsigned) * ((size_t)n + 4));
    volatile unsigned* const gone = host_word(kRemoved);
    if (!flag || !rank || !gone) return CCT_MEMERR;
    int* removed = (int*)(rank + n);
    MPS_CUDA_TRY(cudaMemsetAsync(removed, 0, sizeof(int), Stream));
    MPS_COUNT_LAUNCH k_ref_outside_flags<<<grid_of(n), kBlock, 0, Stream>>>(n, g_bind, flag);
    MPS_CUDA_TRY(cudaMemcpyAsync(rank, flag, sizeof(unsigned) * (size_t)n, cudaMemcpyDeviceToDevice, Stream));
    MPS_CUDA_TRY(scan_exclusive(rank, n, nullptr, Stream, scan_sums(9)));
    MPS_COUNT_LAUNCH k_ref_compact<<<grid_of(n), kBlock, 0, Stream>>>(n, g_bind, flag, rank, removed);
    MPS_CUDA_TRY(cudaMemcpyAsync((void*)gone, removed, sizeof(int), cudaMemcpyDeviceToHost, Stream));
    MPS_CUDA_TRY(cudaStreamSynchronize(Stream));
    const int r = (int)*gone;
    *ParticleNum = n - r;
    g_bind.particle_num = n - r;
    return launch_status();
}

CCTStatusType ResetTriangleTopology(cudaStream_t& Stream, Integer CellNum, CCell* aCell) {
    if (CellNum <= 0) return CCT_NOERR;
    MPS_COUNT_LAUNCH k_tri_reset<<<grid_of(CellNum), kBlock, 0, Stream>>>(CellNum, aCell);
    return launch_status();
}

CCTStatusType RegisterTriangleTopology(cudaStream_t& Stream, CTriangle* daTriangle, Integer TriangleNum, CCell* daCell,
                                       Integer CellNum) {
    const int t = TriangleNum;
    if (t <= 0 || CellNum <= 0) return CCT_NOERR;
    const ScratchTurn turn(ScratchTurn::kTriangles, Stream);
    unsigned* off = (unsigned*)scratch_get(4, sizeof(unsigned) * ((size_t)t + 4));
    if (!off) return CCT_MEMERR;
    unsigned *const total_dev = off + t, *const failed = off + t + 1;
    volatile unsigned* const report = host_word(kErrTriangles);
    if (!report) return CCT_MEMERR;
    const bool few = t < kTriFew;
    if (few)
        MPS_COUNT_LAUNCH k_tri_count<32><<<div_up(t, kBlock / 32), kBlock, 0, Stream>>>(t, daTriangle, g_bind.box, CellNum, off, failed);
    else
        MPS_COUNT_LAUNCH k_tri_count<8><<<div_up(t, kBlock / 8), kBlock, 0, Stream>>>(t, daTriangle, g_bind.box, CellNum, off, failed);
    MPS_CUDA_TRY(scan_exclusive(off, t, total_dev, Stream, scan_sums(8)));
    volatile unsigned* const visits = host_word(kVisits);
    MPS_CUDA_TRY(cudaMemcpyAsync((void*)visits, total_dev, sizeof(unsigned), cudaMemcpyDeviceToHost, Stream));
    MPS_CUDA_TRY(cudaStreamSynchronize(Stream));
    const unsigned nv = *visits;
    if (triangles_failed()) {   // in an earlier call: said once here, in the wall launchers until then
        *report = 0u;
        return CCT_CUDAERR;
    }
    if (nv == 0) return launch_status();
    int* vcell = (int*)scratch_get(5, sizeof(int) * (size_t)nv * 2);
    const int most = std::min((int)nv, CellNum);   // runs
    int* runs = (int*)scratch_get(6, sizeof(int) * (size_t)most);
    void* sscr = scratch_get(7, radix_scratch_bytes((int)nv));
    if (!vcell || !runs || !sscr) return CCT_MEMERR;
    int* vtri = vcell + nv;
    if (few)
        MPS_COUNT_LAUNCH k_tri_fill<32><<<div_up(t, kBlock / 32), kBlock, 0, Stream>>>(t, daTriangle, g_bind.box, CellNum, off, vcell, vtri);
    else
        MPS_COUNT_LAUNCH k_tri_fill<8><<<div_up(t, kBlock / 8), kBlock, 0, Stream>>>(t, daTriangle, g_bind.box, CellNum, off, vcell, vtri);
    MPS_CUDA_TRY(radix_sort_pairs((int)nv, vcell, vtri, radix_bits((unsigned)CellNum), sscr, failed, 1u, Stream));
    int* const runs_n = (int*)failed + 1;
    MPS_COUNT_LAUNCH k_tri_runs<<<grid_of((int)nv), kBlock, 0, Stream>>>((int)nv, vcell, runs, runs_n, failed, report);
    MPS_COUNT_LAUNCH k_tri_cells<<<div_up(most, kBlock / 32), kBlock, 0, Stream>>>((int)nv, runs, runs_n, vcell, vtri, daCell);
    return launch_status();
}

CCTStatusType UpdateTrianglePosition(cudaStream_t& Stream, const Integer TriangleNum, CTriangle* daTriangles) {
    if (TriangleNum <= 0) return CCT_NOERR;
    MPS_COUNT_LAUNCH k_tri_translate<<<grid_of(TriangleNum), kBlock, 0, Stream>>>(TriangleNum, daTriangles, g_bind);
    return launch_status();
}

CCTStatusType RotateTrianglePosition(cudaStream_t& Stream, const Integer TriangleNum, CTriangle* daTriangles,
                                     const Integer analysisStep) {
    if (TriangleNum <= 0) return CCT_NOERR;
    MPS_COUNT_LAUNCH k_tri_rotate<<<grid_of(TriangleNum), kBlock, 0, Stream>>>(TriangleNum, daTriangles, analysisStep, g_bind);
    return launch_status();
}

CCTStatusType ResetWallPosition(cudaStream_t& Stream, const Integer TriangleNum, const Integer AnalysisStep,
                                const CTriangle* daTriangles) {
    if (TriangleNum <= 0) return CCT_NOERR;
    MPS_COUNT_LAUNCH k_tri_reset_wall<<<grid_of(TriangleNum), kBlock, 0, Stream>>>(TriangleNum, AnalysisStep, daTriangles, g_bind);
    return launch_status();
}

CCTStatusType CalcSTLDistance(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    if (triangles_failed()) return CCT_CUDAERR;
    const int n = ComputeParticleNum;
    if (const int most = near_short_most(n)) {
        MPS_COUNT_LAUNCH k_ref_stl_short<<<div_up(n, 128), 128, 0, Stream>>>(n, (unsigned)most, g_bind);
        MPS_CUDA_TRY(near_left_launch(Stream, n, most, near_marks(most) == 32 ? k_ref_stl_distance<32> : k_ref_stl_distance<64>));
    } else {
        MPS_COUNT_LAUNCH k_ref_stl_distance<0><<<div_up(n, near_particles<0>()), 128, 0, Stream>>>(n, g_bind);
    }
    return launch_status();
}

CCTStatusType CalcDragEffect(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    if (triangles_failed()) return CCT_CUDAERR;
    const int n = ComputeParticleNum;
    if (const int most = near_short_most(n)) {
        MPS_COUNT_LAUNCH k_ref_drag_short<<<div_up(n, 128), 128, 0, Stream>>>(n, (unsigned)most, g_bind);
        MPS_CUDA_TRY(near_left_launch(Stream, n, most, near_marks(most) == 32 ? k_ref_drag<32> : k_ref_drag<64>));
    } else {
        MPS_COUNT_LAUNCH k_ref_drag<0><<<div_up(n, near_particles<0>()), 128, 0, Stream>>>(n, g_bind);
    }
    return launch_status();
}

CCTStatusType CalcExplicitly(cudaStream_t& Stream, Integer ParticleNum) {
    if (ParticleNum <= 0) return CCT_NOERR;
    if (g_bind.param.bTurbulance && (!g_bind.turb_visc || !g_bind.strain)) return CCT_PARAMERR;
    const CParameter& P = g_bind.param;
    const float coef = (float)((2.0 * P.Dimension) / (double)(P.LambdaValue * P.ConstantParticleDensity));
    if (ParticleNum >= kRefLanes)
        MPS_COUNT_LAUNCH k_ref_walk<RpExplicitly><<<div_up(ParticleNum, 128), 128, 0, Stream>>>(ParticleNum, coef, g_bind);
    else
        MPS_CUDA_TRY((ref_op_launch<RpExplicitly, 8>(Stream, ParticleNum, kRefFew, coef)));
    return launch_status();
}

CCTStatusType CalcExplicitPressure(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    MPS_CUDA_TRY((ref_op_launch<RpPressure, 8>(Stream, ComputeParticleNum, kRefFew)));
    return launch_status();
}

CCTStatusType CalcExplicitPressureGradient(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    if (g_bind.param.bNegativePressure) return CCT_PARAMERR;
    MPS_CUDA_TRY((ref_op_launch<RpGradient, 8>(Stream, ComputeParticleNum, kRefFew)));
    return launch_status();
}

CCTStatusType CalcTemperatureFactor(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    if (!g_bind.temperature || !g_bind.out_temperature || !g_bind.out_kin_visc) return CCT_PARAMERR;
    MPS_CUDA_TRY((ref_op_launch<RpTemperature, 8>(Stream, ComputeParticleNum, kRefFew)));
    return launch_status();
}

CCTStatusType CalcTurbulenceViscosity(cudaStream_t& Stream, Integer ComputeParticleNum) {
    if (ComputeParticleNum <= 0) return CCT_NOERR;
    if (!g_bind.turb_visc || !g_bind.strain) return CCT_PARAMERR;
    MPS_CUDA_TRY((ref_op_launch<RpTurbulence, 4>(Stream, ComputeParticleNum, kRefFewTurbulence)));
    return launch_status();
}

}  // extern "C"
