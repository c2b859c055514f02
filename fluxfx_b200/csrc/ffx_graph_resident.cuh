// The collider multigrid with the iterate resident on the chip: whole solves
// (a fixed number of V-cycles, or V-cycles to a tolerance) of one domain or of
// many at once, or the coarse part of a V-cycle, in one cooperative launch.
//
// The passes one by one (ffx_project.cu, ffx_level0.cu) cost 4-10 us each on
// levels of 10^3 to 10^6 cells whatever their arithmetic, and a coarsest level
// without a direct solve costs 80 of them; see ffx_resident.cuh for the scheme
// (tiles of rows in shared memory, rims traded as 64-bit words of value and
// exchange number). Here a level's operator is resident too: level 0 as one
// link byte per cell, coarser levels as their edge records. Every domain of a
// launch has its own blocks, its own tail block and its own convergence, so a
// domain that has converged no longer waits for the others.
//
// Every cell is evaluated with the operations of graph_terms and its callers in
// their order (no contraction), so results are bit-identical to the separate
// passes.
//
// Measured, a step with a sphere and a box, separate passes -> resident:
// 96 x 80 x 112 (two V(4,4) cycles) 783 -> 716 us, 96 x 96 x 160 (five) 2226 ->
// 1838 us. A cycle of 96 x 96 x 160 takes 129 us. What bounds it is the latency of
// a sweep and of its exchange: a quarter of the issue slots are used, and a warp
// waits 8 cycles at block barriers (behind the warps that poll) and 2 for loads per
// instruction it issues (profiles/resident_solves.txt); packed FP32 instructions
// (f32x2) changed nothing.
#pragma once
#include "ffx_batch.cuh"
#include "ffx_resident.cuh"

namespace ffx {
namespace gres {

using resident::collect;
using resident::Exchange;
using resident::kDirectCells;
using resident::kRimItems;
using resident::kThreads;
using resident::published;
using resident::put1;
using resident::put4;
using resident::quotient;
using resident::rim_items;
using resident::u64;
using resident::View;
using resident::Waits;
using resident::zero4;

constexpr int kLevels = 10;
constexpr int kMaxTiles = 160;

// A level of a domain: geometry and shared-memory float4 offsets of a tile.
struct Level {
    resident::Level base;     // n, x4, ty, tz, p, q, r, w (level 0), ll
    int ex, ey, ez, rc;       // edge records along x, y (from the row below), z (from the plane below), 1 / diagonal
    const float4* edges;      // (+x, +y, +z, active) of every cell; NULL on level 0
    float cs;                 // factor of the correction prolonged into this level
};

struct Domain {
    int count, dist, gy, gz;           // levels, levels in tiles, tiles
    int first_block, blocks;
    int pre0, post0, pre, post, last;  // sweeps of level 0, of the levels below, of the coarsest one
    float omega;
    int whole;                         // level 0 is the mask's (links); else level 0 is a coarse level
    const uint8_t* links;
    int link_off;                      // float4 offset of the link bytes, rim included
    int vec;                           // rows of level 0 start on 16 bytes
    float* p;                          // batched solves: the iterate and its right-hand side
    const float* rhs;
    const double* inverse;             // dense FP64 inverse of the coarsest level, or NULL
    u64* ws;
    int64_t tail_rhs, tail_p, maxima, control;   // words
    unsigned* epochs;                  // two per block: the next launch's exchanges and decisions count from them
    int exchanges;                     // of a cycle's sweeps, all levels in tiles
    unsigned* timeouts;
    int* alarm;
    int tile_f4, tail_f4;
    double tol;
    int max_cycles;
    BatchState* state;                 // batched: scale and cycle count of the solve
    Level lv[kLevels];                 // tiles: levels 0 .. dist (dist: its pressure only)
    Level tv[kLevels];                 // tail
};

// What changes from launch to launch of one domain's solve.
struct Call {
    float* p;
    const float* rhs;
    int cycles;          // fixed budget, or 0: to the tolerance
    int from_zero;
    double tol;
    int max_cycles;
    int* counters;       // [cycles of this solve, of all solves, decisions]
    int aligned;         // p and rhs start on 16 bytes
    int batched;         // everything from the domains' own records
};

// Cycles of a launch at most.
__device__ __forceinline__ int cycle_limit(const Domain& D, const Call& A) {
    if (!D.whole) return 1;
    return A.cycles > 0 ? A.cycles : (A.batched ? D.max_cycles : A.max_cycles);
}
// What a launch adds to a block's two numbers: as many exchanges (every sweep's, a
// maximum per decision, the scale) and decisions as it may take, not those it took.
// So a wait that gives up, after which blocks may part ways, leaves them with the
// same numbers for the next launch.
__device__ __forceinline__ unsigned exchanges_numbered(const Domain& D, int limit) {
    return 2u + (unsigned)limit * (unsigned)(D.exchanges + 1);
}
__device__ __forceinline__ unsigned decisions_numbered(int limit) { return (unsigned)limit + 1u; }

struct GView {
    View v;
    const float4* EX;
    const float4* EY;
    const float4* EZ;
    const float4* RC;
    const unsigned* links;    // P's order (rim included)
    float cs;
};

__device__ __forceinline__ GView make_gview(const Domain& D, const Level& L, int by, int bz, float4* smem, u64* ws,
                                            bool flip) {
    GView g;
    g.v = resident::make_view(L.base, by, bz, smem, ws, flip);
    g.EX = smem + L.ex;
    g.EY = smem + L.ey;
    g.EZ = smem + L.ez;
    g.RC = smem + L.rc;
    g.links = reinterpret_cast<const unsigned*>(smem + D.link_off);
    g.cs = L.cs;
    return g;
}

// diag of a cell from its link bits, added in graph_terms' order.
__device__ __forceinline__ float link_diag(unsigned bits, const float* w) {
    float d = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (bits >> (2 * a) & 1u) d = d + w[a];
        if (bits >> (2 * a + 1) & 1u) d = d + w[a];
    }
    return d;
}

// 1 / diag for div_rn, whose divisors lie in [2^-30, 2^30].
__device__ __forceinline__ bool in_range(float diag) { return diag >= 0x1p-30f && diag <= 0x1p30f; }
__device__ __forceinline__ float reciprocal(float diag) { return in_range(diag) ? __frcp_rn(diag) : 0.f; }

// c (1 - omega) + ((nb - r) / diag) omega, 0 where there is no weight. The
// quotient is the IEEE one by either route: div_rn with the kept reciprocal y
// (a third of the instructions), or the division where a diagonal of the level
// lies outside div_rn's range (`divide`, the same for the whole block).
__device__ __forceinline__ float4 relaxed(float4 c, float4 nb, float4 r, float4 diag, float4 y, bool divide, float omega,
                                          float omc) {
    float4 q = make_float4(nb.x - r.x, nb.y - r.y, nb.z - r.z, nb.w - r.w);
    if (divide) q = make_float4(q.x / diag.x, q.y / diag.y, q.z / diag.z, q.w / diag.w);
    else q = make_float4(div_rn(q.x, diag.x, y.x), div_rn(q.y, diag.y, y.y), div_rn(q.z, diag.z, y.z), div_rn(q.w, diag.w, y.w));
    return make_float4(diag.x > 0.f ? c.x * omc + q.x * omega : 0.f, diag.y > 0.f ? c.y * omc + q.y * omega : 0.f,
                       diag.z > 0.f ? c.z * omc + q.z * omega : 0.f, diag.w > 0.f ? c.w * omc + q.w * omega : 0.f);
}
__device__ __forceinline__ float residual(float c, float nb, float r, float diag) {
    return diag > 0.f ? (r - nb) + diag * c : 0.f;
}

// The six terms around a float4 in graph_terms' order. On level 0 (LINKS)
// every weight is the axis's: unlinked neighbours inside the domain are solid
// and hold 0, outside there is 0. A weight of an edge record of 0 does the same.
struct Around {
    float4 c, lo, hi, ym, yp;
    float xl, xr;
};
__device__ __forceinline__ float4 sum_links(const Around& t, const float* w) {
    auto one = [&](float xm, float xp, float a, float b, float e, float f) {
        float nb = 0.f + w[0] * xm;
        nb = nb + w[0] * xp;
        nb = nb + w[1] * a;
        nb = nb + w[1] * b;
        nb = nb + w[2] * e;
        return nb + w[2] * f;
    };
    return make_float4(one(t.xl, t.c.y, t.ym.x, t.yp.x, t.lo.x, t.hi.x), one(t.c.x, t.c.z, t.ym.y, t.yp.y, t.lo.y, t.hi.y),
                       one(t.c.y, t.c.w, t.ym.z, t.yp.z, t.lo.z, t.hi.z), one(t.c.z, t.xr, t.ym.w, t.yp.w, t.lo.w, t.hi.w));
}
__device__ __forceinline__ float4 sum_edges(const Around& t, float exl, float4 ex, float4 eyl, float4 ey, float4 ezl,
                                            float4 ez) {
    auto one = [](float wl, float xm, float wr, float xp, float wd, float a, float wu, float b, float wb, float e,
                  float wf, float f) {
        float nb = 0.f + wl * xm;
        nb = nb + wr * xp;
        nb = nb + wd * a;
        nb = nb + wu * b;
        nb = nb + wb * e;
        return nb + wf * f;
    };
    return make_float4(
        one(exl, t.xl, ex.x, t.c.y, eyl.x, t.ym.x, ey.x, t.yp.x, ezl.x, t.lo.x, ez.x, t.hi.x),
        one(ex.x, t.c.x, ex.y, t.c.z, eyl.y, t.ym.y, ey.y, t.yp.y, ezl.y, t.lo.y, ez.y, t.hi.y),
        one(ex.y, t.c.y, ex.z, t.c.w, eyl.z, t.ym.z, ey.z, t.yp.z, ezl.z, t.lo.z, ez.z, t.hi.z),
        one(ex.z, t.c.z, ex.w, t.xr, eyl.w, t.ym.w, ey.w, t.yp.w, ezl.w, t.lo.w, ez.w, t.hi.w));
}

// diag of a float4's cells from their edge records, added in graph_terms' order.
__device__ __forceinline__ float4 record_diag(float exl, float4 ex, float4 eyl, float4 ey, float4 ezl, float4 ez) {
    auto one = [](float a, float b, float c, float d, float e, float f) { return 0.f + a + b + c + d + e + f; };
    return make_float4(one(exl, ex.x, eyl.x, ey.x, ezl.x, ez.x), one(ex.x, ex.y, eyl.y, ey.y, ezl.y, ez.y),
                       one(ex.y, ex.z, eyl.z, ey.z, ezl.z, ez.z), one(ex.z, ex.w, eyl.w, ey.w, ezl.w, ez.w));
}

// The weights of a float4's cells: the diagonal (and its reciprocal), and on a
// coarse level the six edge records.
struct Weights {
    float4 diag, y, ex, eyl, ey, ezl, ez;
    float exl;
};
template <bool LINKS>
__device__ __forceinline__ Weights weights_at(const GView& g, int x, int y, int z, const float2* table) {
    const View& v = g.v;
    Weights w;
    if (LINKS) {
        const unsigned k = g.links[v.at(x, y, z)];
        const float2 a = table[k & 63u], b = table[k >> 8 & 63u], c = table[k >> 16 & 63u], d = table[k >> 24 & 63u];
        w.diag = make_float4(a.x, b.x, c.x, d.x);
        w.y = make_float4(a.y, b.y, c.y, d.y);
    } else {
        const int s = x + v.x4 * (y + v.ty * z), sy = x + v.x4 * (y + (v.ty + 1) * z);      // sy: EY's row y - 1
        w.exl = x > 0 ? reinterpret_cast<const float*>(g.EX)[4 * s - 1] : 0.f;
        w.ex = g.EX[s];
        w.eyl = g.EY[sy];
        w.ey = g.EY[sy + v.x4];
        w.ezl = g.EZ[s];
        w.ez = g.EZ[s + v.flat];
        w.y = g.RC[s];
        w.diag = record_diag(w.exl, w.ex, w.eyl, w.ey, w.ezl, w.ez);
    }
    return w;
}
template <bool LINKS>
__device__ __forceinline__ float4 neighbours(const Around& t, const Weights& w, const GView& g) {
    if (LINKS) return sum_links(t, g.v.w);
    return sum_edges(t, w.exl, w.ex, w.eyl, w.ey, w.ezl, w.ez);
}

// `count` sweeps. A thread owns a run of float4 along z; the cells beside its
// own along x come from the lanes beside it. With two copies of the pressure a
// sweep goes from P to Q and the copies change places; level 0, where there is
// no room for a second, is swept in place. A coarse level whose runs are one
// float4 keeps its weights in registers for all sweeps.
template <bool LINKS>
__device__ __forceinline__ void relax(GView& g, int level, const float2* table, bool divide, bool zero, int count,
                                      float omega, Exchange& ex) {
    View& v = g.v;
    const int tid = threadIdx.x, lane = tid & 31;
    const int groups = min(max(quotient(kThreads, v.inv_flat), 1), v.tz);
    const int run = quotient(v.tz + groups - 1, __frcp_rn((float)groups));
    const int gr = quotient(tid, v.inv_flat), it = tid - gr * v.flat, y = quotient(it, v.inv_x4), x = it - y * v.x4;
    const int z0 = gr * run, mine = gr < groups ? max(min(run, v.tz - z0), 0) : 0;
    const int i0 = v.at(x, y, z0), r0 = x + v.x4 * (y + v.ty * z0);
    int from[kRimItems], dst[kRimItems];
    u64* out_words = nullptr;
    if (ex.on) {
        rim_items(v, from, dst);
        out_words = v.ll + published(v, x, v.y0 + y, v.z0 + z0);
    }
    const int out_step = 4 * v.x4 * v.n[1];
    const int64_t copy = 4 * (int64_t)v.x4 * v.n[1] * v.n[2];
    const bool rim_y = y == 0 || y == v.ty - 1;
    const float omc = 1.f - omega;
    const bool two = !LINKS || v.P != v.Q, keep = !LINKS && run == 1;
    Weights kept = {};
    float4 kept_r = zero4();
    if (keep && mine > 0) {
        kept = weights_at<LINKS>(g, x, y, z0, table);
        kept_r = v.R[r0];
    }
    for (int s = 0; s < count; ++s) {
        const bool blank = zero && s == 0;
        const int64_t half = ex.turn >> level & 1u ? copy : 0;
        float4 lo = zero4(), c = zero4(), top = zero4();
        if (mine > 0 && !blank) {
            lo = v.P[i0 - v.plane];
            c = v.P[i0];
            if (!two) top = v.P[i0 + mine * v.plane];       // read before the plane above is written
        }
        if (!two) __syncthreads();
        for (int j = 0; j < run; ++j) {
            const bool on = j < mine;
            const int i = i0 + j * v.plane;
            float4 o = zero4();
            Around t = {};
            if (!blank) {
                t.xl = __shfl_up_sync(0xffffffffu, c.w, 1);
                t.xr = __shfl_down_sync(0xffffffffu, c.x, 1);
            }
            if (on) {
                const Weights w = keep ? kept : weights_at<LINKS>(g, x, y, z0 + j, table);
                const float4 r = keep ? kept_r : v.R[r0 + j * v.flat];
                float4 nb = zero4();
                t.c = c;
                if (!blank) {
                    const float* row = reinterpret_cast<const float*>(v.P) + 4 * i;
                    if (x == 0) t.xl = 0.f;
                    else if (lane == 0) t.xl = row[-1];
                    if (x + 1 == v.x4) t.xr = 0.f;
                    else if (lane == 31) t.xr = row[4];
                    t.lo = lo;
                    t.hi = !two && j == mine - 1 ? top : v.P[i + v.plane];
                    t.ym = v.P[i - v.x4];
                    t.yp = v.P[i + v.x4];
                    nb = neighbours<LINKS>(t, w, g);
                }
                o = relaxed(c, nb, r, w.diag, w.y, divide, omega, omc);
                if (ex.on && (rim_y || z0 + j == 0 || z0 + j == v.tz - 1)) put4(out_words + half + j * out_step, o, ex.epoch);
                lo = c;
                c = t.hi;
                if (two) v.Q[i] = o;
            }
            if (!two) {
                // a plane is written when every thread has formed its part of it
                __syncthreads();
                if (on) v.P[i] = o;
            }
        }
        if (ex.on) {
            collect(v.ll + half, from, two ? v.Q : v.P, dst, ex.epoch, ex.waits);
            ex.turn ^= 1u << level;
            ++ex.epoch;
        }
        __syncthreads();
        if (two) {
            float4* t = v.P;
            v.P = v.Q;
            v.Q = t;
        }
    }
}

template <bool LINKS>
__device__ __forceinline__ float4 residual4(const GView& g, const float2* table, int x, int y, int z) {
    const View& v = g.v;
    const int i = v.at(x, y, z);
    const float4 c = v.P[i], r = v.R[x + v.x4 * (y + v.ty * z)];
    const float* row = reinterpret_cast<const float*>(v.P) + 4 * i;
    const Weights w = weights_at<LINKS>(g, x, y, z, table);
    const Around t = {c, v.P[i - v.plane], v.P[i + v.plane], v.P[i - v.x4], v.P[i + v.x4],
                      x > 0 ? row[-1] : 0.f, x + 1 < v.x4 ? row[4] : 0.f};
    const float4 nb = neighbours<LINKS>(t, w, g), d = w.diag;
    return make_float4(residual(c.x, nb.x, r.x, d.x), residual(c.y, nb.y, r.y, d.y), residual(c.z, nb.z, r.z, d.z),
                       residual(c.w, nb.w, r.w, d.w));
}

// The eight children's residuals of the two coarse cells over float4 x, added
// in the restriction's order (z, y, x).
template <bool LINKS, class Store>
__device__ __forceinline__ void restrict_pair(const GView& g, const float2* table, int x, int Y, int Z, Store&& store) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 r = residual4<LINKS>(g, table, x, 2 * Y + (k & 1), 2 * Z + (k >> 1));
        a = a + r.x;
        a = a + r.y;
        b = b + r.z;
        b = b + r.w;
    }
    store(2 * x, a / 8.0f);
    if (4 * x + 2 < g.v.n[0]) store(2 * x + 1, b / 8.0f);
}

// P += cs * coarse on the tile and its rim (the coarse rim reaches under it).
// Solid cells of level 0 keep 0; an inactive cell of a coarse level has no
// weight anywhere and is set to 0 by the sweep after this.
template <bool LINKS>
__device__ __forceinline__ void prolong(const GView& g, const GView& c) {
    const View& v = g.v;
    const int all = v.plane * (v.tz + 2);
    for (int s = threadIdx.x; s < all; s += kThreads) {
        int x, y, z;
        v.item(s, x, y, z);
        const int gy = v.y0 + y, gz = v.z0 + z;
        if (gy < 0 || gz < 0 || gy >= v.n[1] || gz >= v.n[2]) continue;
        const float2 q = reinterpret_cast<const float2*>(c.v.P)[2 * c.v.at(0, (gy >> 1) - c.v.y0, (gz >> 1) - c.v.z0) + x];
        float4 p = v.P[s];
        const unsigned k = LINKS ? g.links[s] : 0x40404040u;
        p = make_float4(k & 0x40u ? p.x + g.cs * q.x : 0.f, k & 0x4000u ? p.y + g.cs * q.x : 0.f,
                        k & 0x400000u ? p.z + g.cs * q.y : 0.f, k & 0x40000000u ? p.w + g.cs * q.y : 0.f);
        v.P[s] = p;
    }
    __syncthreads();
}

// A coarse level's edge records of this block's rows into shared memory; true
// when a diagonal among them is out of div_rn's range.
__device__ __forceinline__ bool load_edges(const Level& L, const GView& g, float4* smem) {
    const View& v = g.v;
    float4 *EX = smem + L.ex, *EY = smem + L.ey, *EZ = smem + L.ez, *RC = smem + L.rc;
    const int rows = v.ty + 1, all = v.x4 * rows * (v.tz + 1);      // from row -1 and plane -1
    const float inv = __frcp_rn((float)(v.x4 * rows));
    for (int s = threadIdx.x; s < all; s += kThreads) {
        const int z = quotient(s, inv) - 1, it = s - (z + 1) * v.x4 * rows;
        const int y = quotient(it, v.inv_x4) - 1, x = it - (y + 1) * v.x4;
        const int gy = v.y0 + y, gz = v.z0 + z;
        float4 e[4] = {zero4(), zero4(), zero4(), zero4()};
        if (gy >= 0 && gz >= 0) {
            const float4* src = L.edges + 4 * x + (int64_t)v.n[0] * (gy + (int64_t)v.n[1] * gz);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (4 * x + j < v.n[0]) e[j] = __ldg(src + j);
        }
        if (y >= 0 && z >= 0) EX[x + v.x4 * (y + v.ty * z)] = make_float4(e[0].x, e[1].x, e[2].x, e[3].x);
        if (z >= 0) EY[x + v.x4 * (y + 1 + rows * z)] = make_float4(e[0].y, e[1].y, e[2].y, e[3].y);
        if (y >= 0) EZ[x + v.x4 * (y + v.ty * (z + 1))] = make_float4(e[0].z, e[1].z, e[2].z, e[3].z);
    }
    __syncthreads();
    bool out = false;
    for (int s = threadIdx.x; s < v.flat * v.tz; s += kThreads) {
        int x, y, z;
        v.slot(s, x, y, z);
        const float exl = x > 0 ? reinterpret_cast<const float*>(EX)[4 * s - 1] : 0.f;
        const int sy = x + v.x4 * (y + rows * z);
        const float4 d = record_diag(exl, EX[s], EY[sy], EY[sy + v.x4], EZ[s], EZ[s + v.flat]);
        RC[s] = make_float4(reciprocal(d.x), reciprocal(d.y), reciprocal(d.z), reciprocal(d.w));
        for (float e : {d.x, d.y, d.z, d.w}) out |= e > 0.f && !in_range(e);
    }
    return __syncthreads_or(out);
}

// Coarsest level: FP64 inverse, a row per warp, summed as direct_kernel does.
__device__ __forceinline__ void direct(const GView& g, const double* __restrict__ inverse) {
    const View& v = g.v;
    const int N = v.n[0] * v.n[1] * v.n[2], lane = threadIdx.x & 31;
    const float* R = reinterpret_cast<const float*>(v.R);
    float* P = reinterpret_cast<float*>(v.P);
    const float inv_nx = __frcp_rn((float)v.n[0]), inv_ny = __frcp_rn((float)v.n[1]);
    for (int row = threadIdx.x >> 5; row < N; row += kThreads / 32) {
        const double* m = inverse + (int64_t)row * N;
        double s = 0.0;
        for (int j = lane; j < N; j += 32) {
            const int yz = quotient(j, inv_nx);
            s += __ldg(m + j) * (double)R[j - yz * v.n[0] + 4 * v.x4 * yz];
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) {
            const int yz = quotient(row, inv_nx), z = quotient(yz, inv_ny);
            P[4 * v.at(0, yz - z * v.n[1], z) + row - yz * v.n[0]] = (float)(s / (double)1.0f);
        }
    }
    __syncthreads();
}

// One value from every tile of the domain, its maximum at every one of them.
__device__ __forceinline__ float domain_max(const Domain& D, float mine, int tile, Exchange& ex, unsigned& turn,
                                            float* scratch) {
    mine = warp_max(mine);
    const int tid = threadIdx.x, tiles = D.gy * D.gz;
    if ((tid & 31) == 0) scratch[tid >> 5] = mine;
    __syncthreads();
    if (tid < 32) {
        float m = tid < kThreads / 32 ? scratch[tid] : 0.f;
        m = warp_max(m);
        if (tid == 0) put1(D.ws + D.maxima + (turn & 1u) * kMaxTiles + tile, m, ex.epoch);
    }
    __syncthreads();
    float m = 0.f;
    if (tid < tiles) {
        const u64* from = D.ws + D.maxima + (turn & 1u) * kMaxTiles + tid;
        for (int spin = 0;; ++spin) {
            u64 w;
            asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(from) : "memory");
            if ((unsigned)(w >> 32) == ex.epoch) {
                m = __uint_as_float((unsigned)w);
                break;
            }
            if ((spin & 255) == 255) {
                if (ex.waits.over()) break;
                if (spin >= resident::kSpinLimit) {
                    ex.waits.give_up();
                    break;
                }
            }
        }
    }
    m = warp_max(m);
    if ((tid & 31) == 0) scratch[tid >> 5] = m;
    __syncthreads();
    m = 0.f;
    for (int k = 0; k < kThreads / 32; ++k) m = fmaxf(m, scratch[k]);
    __syncthreads();
    ++turn;
    ++ex.epoch;
    return m;
}

// ------------------------------------------------------------------- roles
__device__ __forceinline__ void run_tail(const Domain& D, const Call& A, float4* smem, const Waits& waits,
                                         int block) {
    const int tid = threadIdx.x;
    Exchange none = {false, 0u, 0u, waits};
    unsigned flip = 0;
    auto view = [&](int k) { return make_gview(D, D.tv[k], 0, 0, smem, nullptr, flip >> k & 1u); };
    const int first = D.dist, last = D.count - 1;
    unsigned divide = 0;
    for (int k = first; k <= last; ++k)
        if (k != last || !D.inverse) divide |= (load_edges(D.tv[k], view(k), smem) ? 1u : 0u) << k;
    const GView top = view(first);
    const int slots = top.v.flat * top.v.tz;
    const unsigned base = D.epochs[2 * block + 1];
    unsigned number = base;
    __shared__ int go;
    for (int c = 0;; ++c) {
        ++number;
        if (tid == 0) {
            // the tiles' decision about this cycle
            go = 0;
            for (int spin = 0;; ++spin) {
                u64 w;
                asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(D.ws + D.control) : "memory");
                if ((unsigned)(w >> 32) == number) {
                    go = (int)(unsigned)w;
                    break;
                }
                if ((spin & 255) == 255 && spin >= resident::kSpinLimit) {
                    waits.give_up();
                    break;
                }
            }
        }
        __syncthreads();
        if (!go) break;
        for (int at = tid; at < slots; at += kThreads * kRimItems) {
            int from[kRimItems], dst[kRimItems];
#pragma unroll
            for (int u = 0; u < kRimItems; ++u) {
                const int s = at + u * kThreads;
                from[u] = s < slots ? 4 * s : -1;
                dst[u] = s;
            }
            collect(D.ws + D.tail_rhs, from, top.v.R, dst, number, waits);
        }
        __syncthreads();
        for (int k = first; k <= last; ++k) {
            GView g = view(k);
            if (k == last) {
                if (D.inverse) {
                    direct(g, D.inverse);
                } else {
                    relax<false>(g, 0, nullptr, divide >> k & 1u, true, D.last, D.omega, none);
                    flip ^= (unsigned)(D.last & 1) << k;
                }
                break;
            }
            relax<false>(g, 0, nullptr, divide >> k & 1u, true, D.pre, D.omega, none);
            flip ^= (unsigned)(D.pre & 1) << k;
            const GView w = view(k + 1);
            float* r = reinterpret_cast<float*>(w.v.R);
            const int hy = w.v.n[1], pairs = g.v.x4 * hy * w.v.n[2];
            const float inv_hy = __frcp_rn((float)hy);
            for (int i = tid; i < pairs; i += kThreads) {
                const int yz = quotient(i, g.v.inv_x4), x = i - yz * g.v.x4, Z = quotient(yz, inv_hy), Y = yz - Z * hy;
                restrict_pair<false>(g, nullptr, x, Y, Z, [&](int X, float q) { r[X + 4 * w.v.x4 * yz] = q; });
            }
            __syncthreads();
        }
        for (int k = last - 1; k >= first; --k) {
            GView g = view(k);
            prolong<false>(g, view(k + 1));
            relax<false>(g, 0, nullptr, divide >> k & 1u, false, D.post, D.omega, none);
            flip ^= (unsigned)(D.post & 1) << k;
        }
        const GView g = view(first);
        for (int s = tid; s < slots; s += kThreads) {
            int x, y, z;
            g.v.slot(s, x, y, z);
            put4(D.ws + D.tail_p + 4 * s, g.v.P[g.v.at(x, y, z)], number);
        }
    }
    __syncthreads();
    if (tid == 0) D.epochs[2 * block + 1] = base + decisions_numbered(cycle_limit(D, A));
}

// LINKS: the domain's level 0 is the mask's grid (a whole solve); else it is a
// coarse level and one V-cycle from zero runs (the coarse part of a cycle).
template <bool LINKS>
__device__ __forceinline__ void run_tile(const Domain& D, const Call& A, float4* smem, float2* table, float* scratch,
                                         const Waits& waits, int tile) {
    const int tid = threadIdx.x;
    const int by = tile % D.gy, bz = tile / D.gy;
    unsigned flip = 0;
    auto view = [&](int k) { return make_gview(D, D.lv[k], by, bz, smem, D.ws, flip >> k & 1u); };
    const unsigned ex_base = D.epochs[2 * tile], base = D.epochs[2 * tile + 1];
    Exchange ex = {true, ex_base + 1u, 0u, waits};
    unsigned number = base, turn = 0;
    float* const P_out = A.batched ? D.p : A.p;
    const float* const rhs = A.batched ? D.rhs : A.rhs;
    const bool from_zero = !LINKS || (!A.batched && A.from_zero);
    const bool to_tolerance = LINKS && A.cycles == 0;
    const int limit = cycle_limit(D, A);
    const double tol = A.batched ? D.tol : A.tol;
    const bool vec = D.vec && A.aligned;
    float scale = 0.f;
    unsigned divide = 0;
    {
        const GView g = view(0);
        const View& v = g.v;
        if (LINKS) {
            bool out = false;
            if (tid < 64) {
                const float d = link_diag((unsigned)tid, v.w);
                table[tid] = make_float2(d, reciprocal(d));
                out = d > 0.f && !in_range(d);
            }
            divide = __syncthreads_or(out) ? 1u : 0u;
            unsigned* links = reinterpret_cast<unsigned*>(smem + D.link_off);
            const int all = v.plane * (v.tz + 2);
            for (int s = tid; s < all; s += kThreads) {
                int x, y, z;
                v.item(s, x, y, z);
                const int gy = v.y0 + y, gz = v.z0 + z;
                unsigned k = 0;
                float4 p = zero4();
                if (gy >= 0 && gz >= 0 && gy < v.n[1] && gz < v.n[2]) {
                    const int64_t at = 4 * x + (int64_t)v.n[0] * (gy + (int64_t)v.n[1] * gz);
                    const int left = v.n[0] - 4 * x;
                    if (vec) {
                        k = __ldg(reinterpret_cast<const unsigned*>(D.links + at));
                        if (!from_zero) p = *reinterpret_cast<const float4*>(P_out + at);
                    } else {
                        float* q = reinterpret_cast<float*>(&p);
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (j < left) {
                                k |= (unsigned)__ldg(D.links + at + j) << (8 * j);
                                if (!from_zero) q[j] = P_out[at + j];
                            }
                    }
                }
                links[s] = k;
                // solid cells weigh nothing and are 0 from the first sweep on
                v.P[s] = make_float4(k & 0x40u ? p.x : 0.f, k & 0x4000u ? p.y : 0.f, k & 0x400000u ? p.z : 0.f,
                                     k & 0x40000000u ? p.w : 0.f);
            }
        }
        for (int s = tid; s < v.flat * v.tz; s += kThreads) {
            int x, y, z;
            v.slot(s, x, y, z);
            const int64_t at = 4 * x + (int64_t)v.n[0] * ((v.y0 + y) + (int64_t)v.n[1] * (v.z0 + z));
            const int left = v.n[0] - 4 * x;
            float4 r = zero4();
            if (vec) {
                r = __ldg(reinterpret_cast<const float4*>(rhs + at));
            } else {
                r.x = __ldg(rhs + at);
                if (left > 1) r.y = __ldg(rhs + at + 1);
                if (left > 2) r.z = __ldg(rhs + at + 2);
                if (left > 3) r.w = __ldg(rhs + at + 3);
            }
            v.R[s] = r;
            scale = fmaxf(scale, fmaxf(fmaxf(finite_abs(r.x), finite_abs(r.y)), fmaxf(finite_abs(r.z), finite_abs(r.w))));
        }
    }
    for (int k = LINKS ? 1 : 0; k < D.dist; ++k) divide |= (load_edges(D.lv[k], view(k), smem) ? 1u : 0u) << k;
    __syncthreads();
    if (to_tolerance) {
        if (A.batched) scale = D.state->scale;
        else scale = domain_max(D, scale, tile, ex, turn, scratch);
    }
    const int low = min(D.dist, D.count - 1);       // the lowest level the tiles prolong from
    const bool tail = D.count > D.dist;
    int c = 0, decisions = 0;
    bool unscaled = false;
    for (;; ++c) {
        bool go = c < limit;
        if (to_tolerance) {
            if (!A.batched && scale == 0.f) {
                // the solve of a zero right-hand side is zero, whatever the start held
                unscaled = true;
                go = false;
            } else if (go) {
                const GView g = view(0);
                float m = 0.f;
                for (int s = tid; s < g.v.flat * g.v.tz; s += kThreads) {
                    int x, y, z;
                    g.v.slot(s, x, y, z);
                    const float4 r = residual4<LINKS>(g, table, x, y, z);
                    m = fmaxf(m, fmaxf(fmaxf(finite_abs(r.x), finite_abs(r.y)), fmaxf(finite_abs(r.z), finite_abs(r.w))));
                }
                m = domain_max(D, m, tile, ex, turn, scratch);
                go = (double)m > tol * (double)scale;
            }
            ++decisions;
        }
        ++number;
        if (tail && tile == 0 && tid == 0) put1(D.ws + D.control, __uint_as_float(go ? 1u : 0u), number);
        if (!go) break;
        for (int k = 0; k < D.dist; ++k) {
            GView g = view(k);
            const bool zero = k > 0 || (c == 0 && from_zero);
            const int sweeps = k == D.count - 1 ? D.last : (k == 0 ? D.pre0 : D.pre);
            if (LINKS && k == 0) relax<true>(g, 0, table, divide & 1u, zero, sweeps, D.omega, ex);
            else relax<false>(g, k, nullptr, divide >> k & 1u, zero, sweeps, D.omega, ex);
            flip ^= (unsigned)(sweeps & 1) << k;
            if (k == D.count - 1) break;
            const resident::Level& C = D.lv[k + 1].base;
            const int hy = g.v.ty / 2, pairs = g.v.x4 * hy * (g.v.tz / 2);
            const float inv_hy = __frcp_rn((float)hy);
            float* r = reinterpret_cast<float*>(smem + C.r);
            for (int i = tid; i < pairs; i += kThreads) {
                const int yz = quotient(i, g.v.inv_x4), x = i - yz * g.v.x4, Z = quotient(yz, inv_hy), Y = yz - Z * hy;
                u64* out = D.ws + D.tail_rhs + 4 * C.x4 * ((g.v.y0 / 2 + Y) + C.n[1] * (g.v.z0 / 2 + Z));
                auto store = [&](int X, float q) {
                    if (k + 1 < D.dist) r[X + 4 * C.x4 * yz] = q;
                    else put1(out + X, q, number);
                };
                if (LINKS && k == 0) restrict_pair<true>(g, table, x, Y, Z, store);
                else restrict_pair<false>(g, nullptr, x, Y, Z, store);
                if (k + 1 == D.dist && x == g.v.x4 - 1)      // padding of the tail's rows
                    for (int X = C.n[0]; X < 4 * C.x4; ++X) put1(out + X, 0.f, number);
            }
            __syncthreads();
        }
        if (tail) {
            const GView g = view(D.dist);
            const View& v = g.v;
            const int all = v.plane * (v.tz + 2);
            for (int at = tid; at < all; at += kThreads * kRimItems) {
                int from[kRimItems], dst[kRimItems];
#pragma unroll
                for (int u = 0; u < kRimItems; ++u) {
                    const int s = at + u * kThreads;
                    int x, y, z;
                    v.item(s, x, y, z);
                    const int gy = v.y0 + y, gz = v.z0 + z;
                    const bool in = s < all && gy >= 0 && gz >= 0 && gy < v.n[1] && gz < v.n[2];
                    from[u] = in ? published(v, x, gy, gz) : -1;
                    dst[u] = s;
                }
                collect(D.ws + D.tail_p, from, v.P, dst, number, waits);
            }
            __syncthreads();
        }
        for (int k = low - 1; k >= 0; --k) {
            GView g = view(k);
            const int sweeps = k == 0 ? D.post0 : D.post;
            if (LINKS && k == 0) {
                prolong<true>(g, view(1));
                relax<true>(g, 0, table, divide & 1u, false, sweeps, D.omega, ex);
            } else {
                prolong<false>(g, view(k + 1));
                relax<false>(g, k, nullptr, divide >> k & 1u, false, sweeps, D.omega, ex);
            }
            flip ^= (unsigned)(sweeps & 1) << k;
        }
    }
    if (c > 0 || unscaled || (from_zero && !A.batched)) {
        const GView g = view(0);
        const View& v = g.v;
        for (int s = tid; s < v.flat * v.tz; s += kThreads) {
            int x, y, z;
            v.slot(s, x, y, z);
            const float4 p = unscaled ? zero4() : v.P[v.at(x, y, z)];
            float* o = P_out + 4 * x + (int64_t)v.n[0] * ((v.y0 + y) + (int64_t)v.n[1] * (v.z0 + z));
            const int left = v.n[0] - 4 * x;
            if (vec) {
                *reinterpret_cast<float4*>(o) = p;
            } else {
                o[0] = p.x;
                if (left > 1) o[1] = p.y;
                if (left > 2) o[2] = p.z;
                if (left > 3) o[3] = p.w;
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        D.epochs[2 * tile] = ex_base + exchanges_numbered(D, limit);
        D.epochs[2 * tile + 1] = base + decisions_numbered(limit);
        if (tile == 0 && to_tolerance) {
            if (A.batched) {
                D.state->cycles = c;
                D.state->done = 1;
            } else {
                A.counters[0] = c;
                A.counters[1] += c;
                A.counters[2] += decisions;
            }
        }
    }
}

template <bool LINKS>
__global__ void __launch_bounds__(kThreads, 1) graph_resident_kernel(const Domain* __restrict__ domains, int count,
                                                                    const __grid_constant__ Call A) {
    extern __shared__ float4 smem[];
    __shared__ Domain D;
    __shared__ float2 table[64];
    __shared__ float scratch[kThreads / 32];
    __shared__ int dead, which;
    const int tid = threadIdx.x;
    if (tid < count) {
        const int first = domains[tid].first_block;
        if ((int)blockIdx.x >= first && (int)blockIdx.x < first + domains[tid].blocks) which = tid;
    }
    if (tid == 0) dead = 0;
    __syncthreads();
    for (int i = tid; i < (int)(sizeof(Domain) / 4); i += kThreads)
        reinterpret_cast<int*>(&D)[i] = __ldg(reinterpret_cast<const int*>(domains + which) + i);
    __syncthreads();
    // coarse parts: a domain that has converged takes no part in the cycle
    if (!LINKS && A.batched && D.state->done) return;
    const int block = (int)blockIdx.x - D.first_block;
    const bool tail = block == D.gy * D.gz;
    const int clear = tail ? D.tail_f4 : D.tile_f4;
    for (int i = tid; i < clear; i += kThreads) smem[i] = zero4();
    __syncthreads();
    const Waits waits = {&dead, D.timeouts, D.alarm};
    if (tail) run_tail(D, A, smem, waits, block);
    else run_tile<LINKS>(D, A, smem, table, scratch, waits, block);
}

}  // namespace gres
}  // namespace ffx
