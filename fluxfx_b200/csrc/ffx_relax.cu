// Weighted-Jacobi relaxation and the geometric V-cycle, several sweeps per
// launch (pressure_jacobi.glsl, mg_residual.glsl, mg_restrict.glsl,
// mg_prolong.glsl, coarse_pressure.glsl; backend/multigrid.py:20-95,
// backend/pressure.py:57-98).
//
// What bounds these solves is not arithmetic or memory but the chain of small
// dependent passes: one launch per sweep costs 3 us on a 32^3 level whose
// arithmetic takes a tenth of that. A grid that fits the SMs' shared memory
// (128^3 and less) is therefore solved in one launch (ffx_resident.cuh). Larger
// grids relax several sweeps per launch: a block stages its tile with a halo of
// one cell per sweep in shared memory and relaxes it there, recomputing the
// halo's shrinking rim instead of exchanging it:
//   * relax_tile_kernel<kSweeps>: T sweeps;
//   * relax_tile_kernel<kDown>:   T sweeps, then residual + 2x2x2 restriction;
//   * relax_tile_kernel<kUp>:     prolongation of the coarse correction, then T sweeps.
// Their levels small enough for one block run in one launch as well.
//
// A sweep evaluates, with nr = -rhs / dt formed once per launch,
//   out = old + (omega / diag) (sum_a w_a (lower + upper) + nr - diag old)
// in FMAs; cells outside the domain and in colliders hold 0, so they add
// nothing to the sum, and diag counts the open neighbours only. (The form
// old (1 - omega) + omega cand with a rounded omega / diag would scale the
// constant mode by the same rounding error in every sweep.)
#include <algorithm>
#include <atomic>

#include "ffx_resident.cuh"

namespace ffx {
namespace {

constexpr int kTileThreads = 512;
constexpr int kSmemLimit = 220 * 1024;
constexpr int kMaxWidth = 128;         // extended tile width in cells

enum Mode { kSweeps = 0, kDown = 1, kUp = 2 };

using resident::byte_of;
using resident::fill_table;
using resident::weighted;
using resident::weights_of;
using resident::zero4;

// Asynchronous copies into shared memory; nothing is read and zeros are
// written where `on` is false.
__device__ __forceinline__ void copy4(float* dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(on ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A box of cells in shared memory: rows of x4 float4, ny rows, nz planes; its
// cell (0, 0, 0) is cell (gx, gy, gz) of a grid of n cells.
struct Box {
    int x4, ny, nz;
    int gx, gy, gz;
    int n[3];
    float w[3];
};

// A thread's share of a box: one float4 column position (x, y) of the planes
// of its group; groups take contiguous runs of planes.
struct Lane {
    int x, y, g, groups;
    bool active;
};

__device__ __forceinline__ Lane make_lane(const Box& b, int tid, int threads) {
    const int plane = b.x4 * b.ny;
    Lane l;
    l.groups = min(max(threads / plane, 1), b.nz);
    l.g = tid / plane;
    const int it = tid - l.g * plane;
    l.y = it / b.x4;
    l.x = it - l.y * b.x4;
    l.active = l.g < l.groups;
    return l;
}

// Table values of the lane's four cells without colliders.
struct Weights {
    float4 k, d;         // omega / diag and diag inside the domain along z
    unsigned edge;       // table entries at its first and last plane
};
__device__ __forceinline__ Weights lane_weights(const Box& b, const Lane& l, const float2* kd) {
    Weights W;
    const int gy = b.gy + l.y, cy = 2 - (gy == 0) - (gy == b.n[1] - 1);
    unsigned inner = 0;
    W.edge = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int gx = b.gx + 4 * l.x + j;
        const unsigned c = (unsigned)(2 - (gx == 0) - (gx == b.n[0] - 1) + 3 * max(cy, 0));
        inner |= (gx < b.n[0] ? c + 18u : 27u) << (8 * j);
        W.edge |= (gx < b.n[0] ? c + 9u : 27u) << (8 * j);
    }
    weights_of(inner, kd, W.k, W.d);
    return W;
}

// One sweep P -> Q over rows [ya, yb) of planes [za, zb). MASK: cls holds each
// cell's table entry. FROM_ZERO: the iterate P is zero and not read.
template <bool MASK, bool FROM_ZERO>
__device__ __forceinline__ void sweep(const Box& b, const Lane& l, const Weights& W, const float4* __restrict__ P,
                                      float4* __restrict__ Q, const float4* __restrict__ R,
                                      const unsigned* __restrict__ cls, const float2* __restrict__ kd, int ya, int yb,
                                      int za, int zb) {
    if (!l.active || l.y < ya || l.y >= yb) return;
    const int run = (zb - za + l.groups - 1) / l.groups;
    const int z0 = za + l.g * run, z1 = min(z0 + run, zb);
    if (z0 >= z1) return;
    const int plane = b.x4 * b.ny;
    int i = l.x + b.x4 * l.y + plane * z0;
    float4 lo = zero4(), c = zero4();
    if (!FROM_ZERO) {
        if (z0 > 0) lo = P[i - plane];
        c = P[i];
    }
    const float wx = b.w[0], wy = b.w[1], wz = b.w[2];
    const int in_row = b.n[0] - (b.gx + 4 * l.x);
    for (int z = z0; z < z1; ++z, i += plane) {
        const float4 r = R[i];
        float4 k = W.k, d = W.d;
        if (MASK) weights_of(cls[i], kd, k, d);
        else if (b.gz + z == 0 || b.gz + z == b.n[2] - 1) weights_of(W.edge, kd, k, d);
        float4 out;
        if (FROM_ZERO) {
            out = make_float4(k.x * r.x, k.y * r.y, k.z * r.z, k.w * r.w);
        } else {
            const float4 hi = z + 1 < b.nz ? P[i + plane] : zero4();
            const float4 ym = l.y > 0 ? P[i - b.x4] : zero4(), yp = l.y + 1 < b.ny ? P[i + b.x4] : zero4();
            const float xl = l.x > 0 ? reinterpret_cast<const float*>(P)[4 * i - 1] : 0.f;
            const float xr = l.x + 1 < b.x4 ? reinterpret_cast<const float*>(P)[4 * i + 4] : 0.f;
            out.x = fmaf(k.x, fmaf(-d.x, c.x, fmaf(wz, lo.x + hi.x, fmaf(wy, ym.x + yp.x, fmaf(wx, xl + c.y, r.x)))),
                         c.x);
            out.y = fmaf(k.y, fmaf(-d.y, c.y, fmaf(wz, lo.y + hi.y, fmaf(wy, ym.y + yp.y, fmaf(wx, c.x + c.z, r.y)))),
                         c.y);
            out.z = fmaf(k.z, fmaf(-d.z, c.z, fmaf(wz, lo.z + hi.z, fmaf(wy, ym.z + yp.z, fmaf(wx, c.y + c.w, r.z)))),
                         c.z);
            out.w = fmaf(k.w, fmaf(-d.w, c.w, fmaf(wz, lo.w + hi.w, fmaf(wy, ym.w + yp.w, fmaf(wx, c.z + xr, r.w)))),
                         c.w);
            lo = c;
            c = hi;
        }
        Q[i] = weighted<MASK, true>(k, in_row, out);
    }
}

// mg_residual.glsl at box cell (x, y, z): rhs/dt - lap, the differences formed
// before they are weighted, as the shader does.
__device__ __forceinline__ float residual_at(const Box& b, const float* __restrict__ P, const float* __restrict__ R,
                                             int x, int y, int z) {
    const int row = 4 * b.x4, plane = row * b.ny, i = x + row * y + plane * z;
    const int gx = b.gx + x, gy = b.gy + y, gz = b.gz + z;
    const float c = P[i];
    float s = R[i];     // -rhs / dt
    s = fmaf(b.w[0], (gx > 0 ? P[i - 1] - c : 0.f) + (gx + 1 < b.n[0] ? P[i + 1] - c : 0.f), s);
    s = fmaf(b.w[1], (gy > 0 ? P[i - row] - c : 0.f) + (gy + 1 < b.n[1] ? P[i + row] - c : 0.f), s);
    s = fmaf(b.w[2], (gz > 0 ? P[i - plane] - c : 0.f) + (gz + 1 < b.n[2] ? P[i + plane] - c : 0.f), s);
    return -s;
}

// mg_restrict.glsl of the residual: the mean over the eight children whose
// lowest is box cell (x, y, z).
__device__ __forceinline__ float restricted_at(const Box& b, const float* P, const float* R, int x, int y, int z) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += residual_at(b, P, R, x + (k & 1), y + (k >> 1 & 1), z + (k >> 2));
    return v * 0.125f;
}

// mg_prolong.glsl for the four cells of the float4 at box position (x, y, z):
// cell-centred trilinear interpolation of a coarse box C (rows of cw floats,
// ch rows) whose entry (0, 0, 0) is coarse cell (cx, cy, cz) and whose entries
// were staged from clamped coarse indices. The box starts at an even cell.
__device__ __forceinline__ float4 prolonged(const Box& b, const float* __restrict__ C, int cw, int ch, int cx, int cy,
                                            int cz, int x, int y, int z) {
    const int gx = b.gx + 4 * x, gy = b.gy + y, gz = b.gz + z;
    // even cells: 1/4 of the lower and 3/4 of their own coarse cell; odd ones 3/4 and 1/4 of the upper
    const int by = (gy + 1) / 2 - 1 - cy, bz = (gz + 1) / 2 - 1 - cz, bx = gx / 2 - 1 - cx;
    const float fy = gy & 1 ? 0.25f : 0.75f, fz = gz & 1 ? 0.25f : 0.75f;
    const float w00 = (1.f - fy) * (1.f - fz), w10 = fy * (1.f - fz), w01 = (1.f - fy) * fz, w11 = fy * fz;
    const float* r = C + bx + cw * (by + ch * bz);
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        v[j] = fmaf(w11, r[j + cw * (1 + ch)], fmaf(w01, r[j + cw * ch], fmaf(w10, r[j + cw], w00 * r[j])));
    return make_float4(fmaf(0.75f, v[1], 0.25f * v[0]), fmaf(0.25f, v[2], 0.75f * v[1]),
                       fmaf(0.75f, v[2], 0.25f * v[1]), fmaf(0.25f, v[3], 0.75f * v[2]));
}

// ------------------------------------------------------------------ tiles
struct TileParams {
    int n[3], tile[3], ext[3];     // grid, tile interior, extended tile at most (x in cells, a multiple of 4)
    int sweeps, halo, halo_x;      // halo_x: halo rounded up to 4 where x is split
    float w[3], omega, dt;
    const float* p;                // NULL: zero
    const float* rhs;
    float* out;
    const uint8_t* cls;            // MASK: table entries (relax_classes_kernel), rows of up4(nx) bytes
    int vec;                       // rows of p, rhs and out start on 16 bytes
    const float* coarse_in;        // kUp
    float* coarse_out;             // kDown
    int box_cells;                 // floats per shared array
    int q_cells;                   // floats of the second iterate (also holds kUp's coarse box)
};

template <int MODE, bool MASK>
__global__ void __launch_bounds__(kTileThreads) relax_tile_kernel(const __grid_constant__ TileParams A) {
    extern __shared__ float4 smem4[];
    __shared__ float2 kd[28];
    float* sp = reinterpret_cast<float*>(smem4);
    float* sr = sp + A.box_cells;
    float* sq = sr + A.box_cells;
    unsigned* sc = reinterpret_cast<unsigned*>(sq + A.q_cells);
    const int tid = threadIdx.x;
    fill_table(kd, tid, A.w, A.omega);
    // interior [i0, i1) of this block and its extension by the halo, clipped to the grid
    const int bi[3] = {(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z};
    int i0[3], i1[3], e0[3], e1[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        i0[a] = bi[a] * A.tile[a];
        i1[a] = min(i0[a] + A.tile[a], A.n[a]);
        const int h = a == 0 ? A.halo_x : A.halo;
        e0[a] = max(i0[a] - h, 0);
        e1[a] = min(i1[a] + h, A.n[a]);
    }
    Box b;
    b.x4 = (e1[0] - e0[0] + 3) >> 2;
    b.ny = e1[1] - e0[1];
    b.nz = e1[2] - e0[2];
    b.gx = e0[0]; b.gy = e0[1]; b.gz = e0[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) { b.n[a] = A.n[a]; b.w[a] = A.w[a]; }
    const int row = 4 * b.x4, plane = row * b.ny, slots = b.x4 * b.ny * b.nz;
    pdl_enter();
    // stage four cells of a row at a time, all copies in flight at once; cells
    // past the grid's end hold 0
    for (int s = tid; s < slots; s += kTileThreads) {
        const int yz = s / b.x4, x = s - yz * b.x4, z = yz / b.ny, y = yz - z * b.ny;
        const int line = (b.gy + y) + A.n[1] * (b.gz + z);
        const int g = b.gx + 4 * x + A.n[0] * line;
        if (A.vec) {
            copy16(sr + 4 * s, A.rhs + g);
            if (A.p) copy16(sp + 4 * s, A.p + g);
        } else {
            const int left = A.n[0] - (b.gx + 4 * x);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = g + min(j, left - 1);
                copy4(sr + 4 * s + j, A.rhs + k, j < left);
                if (A.p) copy4(sp + 4 * s + j, A.p + k, j < left);
            }
        }
        if (!A.p) reinterpret_cast<float4*>(sp)[s] = zero4();
        if (MASK) copy4(reinterpret_cast<float*>(sc) + s, reinterpret_cast<const float*>(
                            A.cls + b.gx + 4 * x + (int64_t)((A.n[0] + 3) & ~3) * line), true);
    }
    if (MODE == kUp) {
        // the coarse cells under the box, one more on each side, from clamped indices
        const int cn[3] = {A.n[0] / 2, A.n[1] / 2, A.n[2] / 2};
        const int cx = b.gx / 2 - 1, cy = b.gy / 2 - 1, cz = b.gz / 2 - 1;
        const int cw = 2 * b.x4 + 2, ch = b.ny / 2 + 3, cd = b.nz / 2 + 3;
        const int count = cw * ch * cd;
        for (int s = tid; s < count; s += kTileThreads) {
            const int yz = s / cw, x = s - yz * cw, z = yz / ch, y = yz - z * ch;
            copy4(sq + s, A.coarse_in + min(max(cx + x, 0), cn[0] - 1) +
                              cn[0] * (min(max(cy + y, 0), cn[1] - 1) + cn[1] * min(max(cz + z, 0), cn[2] - 1)), true);
        }
        copies_done();
        __syncthreads();
        float4* P = reinterpret_cast<float4*>(sp);
        for (int s = tid; s < slots; s += kTileThreads) {
            const int yz = s / b.x4, x = s - yz * b.x4, z = yz / b.ny, y = yz - z * b.ny;
            const float4 v = prolonged(b, sq, cw, ch, cx, cy, cz, x, y, z);
            float4 p = P[s];
            const int left = b.n[0] - (b.gx + 4 * x);     // cells of this float4 inside the grid
            p.x += v.x;
            if (left > 1) p.y += v.y;
            if (left > 2) p.z += v.z;
            if (left > 3) p.w += v.w;
            P[s] = p;
        }
    } else {
        copies_done();
    }
    // a thread finishes the cells that it staged: -rhs / dt, and the pressure of
    // a solid or isolated cell, which is 0 from the first sweep on
    for (int s = tid; s < slots; s += kTileThreads) {
        float4 r = reinterpret_cast<float4*>(sr)[s];
        if (A.dt != 1.f) r = make_float4(r.x / A.dt, r.y / A.dt, r.z / A.dt, r.w / A.dt);
        reinterpret_cast<float4*>(sr)[s] = make_float4(-r.x, -r.y, -r.z, -r.w);
        if (MASK && A.p) {
            const unsigned t = sc[s];
            float* p = sp + 4 * s;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (byte_of(t, j) == 27u || byte_of(t, j) == 0u) p[j] = 0.f;
        }
    }
    __syncthreads();
    const Lane l = make_lane(b, tid, kTileThreads);
    const Weights W = lane_weights(b, l, kd);
    float* cur = sp;
    float* nxt = sq;
    for (int s = 1; s <= A.sweeps; ++s) {
        // rows and planes still needed: the interior grown by what follows
        const int grow = A.halo - s;
        const int ya = max(i0[1] - grow, 0) - b.gy, yb = min(i1[1] + grow, A.n[1]) - b.gy;
        const int za = max(i0[2] - grow, 0) - b.gz, zb = min(i1[2] + grow, A.n[2]) - b.gz;
        if (s == 1 && A.p == nullptr && MODE != kUp)
            sweep<MASK, true>(b, l, W, (const float4*)cur, (float4*)nxt, (const float4*)sr, sc, kd,
                              ya, yb, za, zb);
        else
            sweep<MASK, false>(b, l, W, (const float4*)cur, (float4*)nxt, (const float4*)sr, sc, kd,
                               ya, yb, za, zb);
        __syncthreads();
        float* t = cur;
        cur = nxt;
        nxt = t;
    }
    // the interior
    {
        const int wx = i1[0] - i0[0], wy = i1[1] - i0[1], wz = i1[2] - i0[2];
        const int ox = i0[0] - b.gx, oy = i0[1] - b.gy, oz = i0[2] - b.gz;
        const int w4 = (wx + 3) >> 2;
        for (int s = tid; s < w4 * wy * wz; s += kTileThreads) {
            const int yz = s / w4, x = 4 * (s - yz * w4), z = yz / wy, y = yz - z * wy;
            float* o = A.out + (i0[0] + x) + A.n[0] * ((i0[1] + y) + A.n[1] * (i0[2] + z));
            const float4 v = *reinterpret_cast<const float4*>(cur + ox + x + row * (oy + y) + plane * (oz + z));
            if (A.vec) {
                *reinterpret_cast<float4*>(o) = v;
            } else {
                o[0] = v.x;
                if (x + 1 < wx) o[1] = v.y;
                if (x + 2 < wx) o[2] = v.z;
                if (x + 3 < wx) o[3] = v.w;
            }
        }
        if (MODE == kDown) {
            const int hx = wx / 2, hy = wy / 2, hz = wz / 2, cnx = A.n[0] / 2, cny = A.n[1] / 2;
            for (int c = tid; c < hx * hy * hz; c += kTileThreads) {
                const int z = c / (hx * hy), y = (c - z * hx * hy) / hx, x = c - hx * (y + hy * z);
                A.coarse_out[(i0[0] / 2 + x) + cnx * ((i0[1] / 2 + y) + cny * (i0[2] / 2 + z))] =
                    restricted_at(b, cur, sr, ox + 2 * x, oy + 2 * y, oz + 2 * z);
            }
        }
    }
}

// Table entry of every cell of a collider mask: cx + 3 cy + 9 cz of its open
// neighbours, 27 for a solid cell (the tests of pressure_jacobi.glsl's masked
// form) and for the padding of each row to a multiple of four.
__global__ void __launch_bounds__(256) relax_classes_kernel(int nx, int ny, int nz, const uint8_t* __restrict__ solid,
                                                           uint8_t* __restrict__ cls) {
    const int pitch = (nx + 3) & ~3;
    int x, y, z;
    if (!cell_coords(pitch, ny, x, y, z)) return;
    uint8_t* out = cls + x + (int64_t)pitch * (y + ny * z);
    const int i = x + nx * (y + ny * z);
    if (x >= nx || __ldg(solid + i)) {
        *out = 27;
        return;
    }
    auto open = [&](bool in, int j) { return in && !__ldg(solid + j) ? 1 : 0; };
    const int cx = open(x > 0, i - 1) + open(x + 1 < nx, i + 1);
    const int cy = open(y > 0, i - nx) + open(y + 1 < ny, i + nx);
    const int cz = open(z > 0, i - nx * ny) + open(z + 1 < nz, i + nx * ny);
    *out = (uint8_t)(cx + 3 * cy + 9 * cz);
}

// ------------------------------------------------------------- host planning
struct Tiling {
    int tile[3], ext[3], halo_x;
    int box_cells, q_cells, smem;
    double cost;          // modelled cycles of the launch
};

int up4(int v) { return (v + 3) & ~3; }

// The tile of a launch of `sweeps` sweeps with a halo of `halo` cells: the one
// with the least modelled time. The model counts, in SM cycles, what a launch
// costs whatever its size (start, first loads), the staging of the extended
// tile and every sweep's shrinking region, times the rounds in which the 148
// SMs take the tiles. Against 2000 tiles of one to four sweeps each, measured over 60
// sweeps, its choice takes 675 us at 301 x 70 x 93 (the best 621, the median 899),
// 4169 at 256^3 (3808, 5615) and 2807 at 192 x 192 x 320 (2681, 4284). Even tile edges
// where the coarse grid has to line up.
bool choose_tile(const int32_t n[3], int sweeps, int halo, int mode, bool mask, Tiling& best) {
    static const int edges[] = {2, 4, 6, 8, 10, 12, 14, 16, 20, 24, 32};
    best.cost = 1e300;
    const int h4 = up4(halo);
    for (int xs = 1; xs <= 64; ++xs) {
        int tx = xs == 1 ? n[0] : up4((n[0] + xs - 1) / xs);
        const int hx = xs == 1 ? 0 : h4;
        if (xs > 1 && (tx < 8 || tx >= n[0])) break;
        const int ex = std::min(up4(tx + 2 * hx), up4(n[0]));
        if (ex > kMaxWidth) continue;
        if (xs > 1 && (n[0] + tx - 1) / tx > 4 && best.cost < 1e300) break;
        for (int ty : edges)
            for (int tz : edges) {
                const int ey = std::min(ty + 2 * halo, (int)n[1]), ez = std::min(tz + 2 * halo, (int)n[2]);
                if (ex / 4 * ey > kTileThreads) continue;
                const int box = ex * ey * ez;
                int q = box;
                if (mode == kUp) q = std::max(q, up4((ex / 2 + 2) * (ey / 2 + 3) * (ez / 2 + 3)));
                const int smem = 4 * (2 * box + q) + (mask ? box : 0);
                if (smem > kSmemLimit) continue;
                const double tiles = (double)((n[0] + tx - 1) / tx) * ((n[1] + ty - 1) / ty) * ((n[2] + tz - 1) / tz);
                const int per_sm = std::max(1, std::min(4, kSmemLimit / (smem + 1024)));
                double work = 0.7 * box + 300.0;
                for (int s = 1; s <= sweeps; ++s) {
                    const int g = halo - s;
                    work += 0.30 * ex * std::min(ty + 2 * g, (int)n[1]) * std::min(tz + 2 * g, (int)n[2]) + 150.0;
                }
                if (mode != kSweeps) work += 0.6 * tx * ty * tz;
                const double rounds = std::ceil(tiles / 148.0);
                // blocks that share an SM overlap each other's waits
                const double waits = 900.0 * std::ceil(rounds / per_sm);
                const double cost = 3500.0 + waits + rounds * work;
                if (cost < best.cost) {
                    best = Tiling{{tx, ty, tz}, {ex, ey, ez}, hx, box, q, smem, cost};
                }
            }
    }
    return best.cost < 1e300;
}

// Raises a kernel's dynamic shared memory limit once per device.
template <class K>
int allow_smem(K kernel, std::atomic<uint64_t>& done) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
    const uint64_t bit = uint64_t(1) << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return FFX_OK;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute");
    done.fetch_or(bit, std::memory_order_release);
    return FFX_OK;
}

template <typename P>
int launch_smem(const char* what, void (*kernel)(P), dim3 grid, int threads, int smem, cudaStream_t st, const P& args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(FFX_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
    }
    return launch_status(what);
}

struct Fields {
    const float* p;
    const float* rhs;
    float* out;
    const uint8_t* cls;
    const float* coarse_in;
    float* coarse_out;
};

template <int MODE, bool MASK>
int launch_tile(const FfxRelaxGrid& g, const FfxRelaxTile& t, const Fields& f, float dt, float omega,
                cudaStream_t st) {
    static std::atomic<uint64_t> ready{0};
    if (int s = allow_smem(relax_tile_kernel<MODE, MASK>, ready)) return s;
    TileParams A = {};
    for (int a = 0; a < 3; ++a) {
        A.n[a] = g.n[a];
        A.tile[a] = t.tile[a];
        A.w[a] = g.inv[a] * g.inv[a];
    }
    A.sweeps = t.sweeps;
    A.halo = t.sweeps + (MODE == kDown ? 1 : 0);
    A.halo_x = t.tile[0] < g.n[0] ? up4(A.halo) : 0;
    const int ex = std::min(up4(t.tile[0] + 2 * A.halo_x), up4(g.n[0]));
    const int ey = std::min(t.tile[1] + 2 * A.halo, g.n[1]), ez = std::min(t.tile[2] + 2 * A.halo, g.n[2]);
    A.box_cells = ex * ey * ez;
    A.q_cells = A.box_cells;
    if (MODE == kUp) A.q_cells = std::max(A.q_cells, up4((ex / 2 + 2) * (ey / 2 + 3) * (ez / 2 + 3)));
    const int smem = 4 * (2 * A.box_cells + A.q_cells) + (MASK ? A.box_cells : 0);
    FFX_REQUIRE(t.tile[0] >= 1 && t.tile[1] >= 1 && t.tile[2] >= 1 && ex <= kMaxWidth &&
                ex / 4 * ey <= kTileThreads && smem <= kSmemLimit &&
                (t.tile[0] == g.n[0] || t.tile[0] % 4 == 0) &&
                (MODE == kSweeps || (t.tile[0] % 2 == 0 && t.tile[1] % 2 == 0 && t.tile[2] % 2 == 0)),
                "relaxation tile out of range");
    A.omega = omega;
    A.dt = dt;
    A.p = f.p;
    A.rhs = f.rhs;
    A.out = f.out;
    A.cls = f.cls;
    const uintptr_t addresses = (uintptr_t)f.p | (uintptr_t)f.rhs | (uintptr_t)f.out;
    A.vec = g.n[0] % 4 == 0 && addresses % 16 == 0;
    A.coarse_in = f.coarse_in;
    A.coarse_out = f.coarse_out;
    const dim3 grid((unsigned)((g.n[0] + t.tile[0] - 1) / t.tile[0]), (unsigned)((g.n[1] + t.tile[1] - 1) / t.tile[1]),
                    (unsigned)((g.n[2] + t.tile[2] - 1) / t.tile[2]));
    return launch_smem("relax_tile_kernel", relax_tile_kernel<MODE, MASK>, grid, kTileThreads, smem, st, A);
}

int cells_of(const int32_t n[3]) { return n[0] * n[1] * n[2]; }

bool grid_valid(const FfxRelaxGrid& g) {
    for (int a = 0; a < 3; ++a)
        if (g.n[a] < 2 || g.n[a] > 4096 || !(g.inv[a] > 0.f)) return false;
    return (int64_t)g.n[0] * g.n[1] * g.n[2] < (int64_t(1) << 31);
}

// The sweeps of one launch that cost least per sweep (`most` at most).
bool plan_sweeps(const int32_t n[3], int most, bool mask, FfxRelaxTile& out) {
    double best = 1e300;
    for (int s = 1; s <= std::min(most, 6); ++s) {
        Tiling t;
        if (!choose_tile(n, s, s, kSweeps, mask, t) || t.cost / s >= best) continue;
        best = t.cost / s;
        out.sweeps = s;
        for (int a = 0; a < 3; ++a) out.tile[a] = t.tile[a];
    }
    return best < 1e300;
}

// The launch that restricts (kDown) or prolongs (kUp) and how many of the
// level's `total` sweeps it does; plain launches do the rest.
bool plan_fused(const int32_t n[3], int total, int mode, const FfxRelaxTile& sweep, FfxRelaxTile& out) {
    Tiling t;
    if (!choose_tile(n, sweep.sweeps, sweep.sweeps, kSweeps, false, t)) return false;
    const double plain = t.cost / sweep.sweeps;
    double best = 1e300;
    for (int s = 1; s <= std::min(total, 6); ++s) {
        if (!choose_tile(n, s, s + (mode == kDown), mode, false, t)) continue;
        const double cost = t.cost + plain * (total - s);
        if (cost >= best) continue;
        best = cost;
        out.sweeps = s;
        for (int a = 0; a < 3; ++a) out.tile[a] = t.tile[a];
    }
    return best < 1e300;
}

// `count` sweeps, the last launch taking what is left (its tile has room for
// fewer sweeps too: the halo only shrinks).
template <bool MASK>
int run_sweeps(const FfxRelaxGrid& g, const FfxRelaxTile& t, const float* rhs, const uint8_t* cls, float dt,
               float omega, int count, bool from_zero, float*& cur, float*& other, cudaStream_t st) {
    for (int done = 0; done < count;) {
        FfxRelaxTile now = t;
        now.sweeps = std::min(t.sweeps, count - done);
        Fields f = {from_zero && done == 0 ? nullptr : cur, rhs, other, cls, nullptr, nullptr};
        if (int s = launch_tile<kSweeps, MASK>(g, now, f, dt, omega, st)) return s;
        std::swap(cur, other);
        done += now.sweeps;
    }
    return FFX_OK;
}

// ---------------------------------------------------------------- resident
using resident::Level;
using resident::Params;

constexpr int kHeaderWords = 128;      // exchange numbers of the blocks, the timeout counter

int64_t slots_of(const int32_t n[3]) { return (int64_t)(up4(n[0]) / 4) * n[1] * n[2]; }

// float4 of shared memory of the levels from `first` on, whole, in one block.
int tail_f4(const FfxRelaxPlan& P, int first) {
    int f4 = 0;
    for (int k = first; k < P.count; ++k) {
        const int32_t* n = P.level[k].grid.n;
        f4 += up4(n[0]) / 4 * (2 * (n[1] + 2) * (n[2] + 2) + n[1] * n[2]);
    }
    return f4;
}

bool tail_level(const int32_t n[3]) {
    return slots_of(n) <= resident::kTailSlots && up4(n[0]) / 4 * n[1] <= resident::kThreads;
}

// float4 of shared memory of a tile of ty x tz rows of the levels below `dist`:
// two copies of each level's pressure, or one of level 0's.
int tile_f4(const FfxRelaxPlan& P, int dist, int ty, int tz, bool one) {
    int f4 = 0;
    for (int k = 0; k <= dist && k < P.count; ++k) {
        const int x4 = up4(P.level[k].grid.n[0]) / 4, y = ty >> k, z = tz >> k;
        f4 += (k == dist || (k == 0 && one) ? 1 : 2) * x4 * (y + 2) * (z + 2) + (k < dist ? x4 * y * z : 0);
    }
    return f4 + (P.classes ? up4(up4(P.level[0].grid.n[0]) / 4 * ty * tz) / 4 : 0);
}

// Whether tiles of ty x tz rows fit with two copies (0) or one (1) of level 0's
// pressure, or not at all (-1).
int tile_fit(const FfxRelaxPlan& P, int dist, int ty, int tz) {
    const int x4 = up4(P.level[0].grid.n[0]) / 4;
    if (x4 * ty > resident::kThreads || x4 * (2 * (ty + tz) + 4) > resident::kThreads * resident::kRimItems) return -1;
    if (16 * tile_f4(P, dist, ty, tz, false) <= resident::kSmem) return 0;
    if (16 * tile_f4(P, dist, ty, tz, true) <= resident::kSmem) return 1;
    return -1;
}

// Tiles of rows for the levels above the tail: as few cells per block as the
// plan's SMs allow, then as small a rim. The weights (a cell 0.9, a rim slot 0.6
// of the same unit) rank tiles well enough: over every tile that fits, the chosen
// one takes 100 sweeps in 121 us at 32^3 (the best 121, the worst 755), 153 at 64^3
// (151, 948), 213 at 75 x 61 x 93 (197, 987), 335 at 128 x 96 x 112 (313, 842) and
// 526 at 127^3 (473, 823), and of V(3,3) cycles it is the best at 64^3, 128 x 96 x
// 112 and 128^3. Tile edges are multiples of 2^levels, so a
// tile restricts into its own coarse tile. False when the grid does not fit.
bool plan_tiles(FfxRelaxPlan& P) {
    const int dist = P.tail;
    const bool tail = dist < P.count;
    const int32_t* n = P.level[0].grid.n;
    const int align = 1 << (tail ? dist : dist - 1), cap = P.sms - (tail ? 1 : 0);
    double best = 1e300;
    for (int ty = align; ty < n[1] + align; ty += align)
        for (int tz = align; tz < n[2] + align; tz += align) {
            const int gy = (n[1] + ty - 1) / ty, gz = (n[2] + tz - 1) / tz;
            if (gy * gz > cap || tile_fit(P, dist, ty, tz) < 0) continue;
            const int x4 = up4(n[0]) / 4;
            const double cost = 0.9 * x4 * ty * tz + 0.6 * x4 * (2 * (ty + tz) + 4);
            if (cost < best) {
                best = cost;
                P.tile[0] = ty;
                P.tile[1] = tz;
            }
        }
    return best < 1e300;
}

int64_t published_words(const FfxRelaxPlan& P) {
    int64_t words = kHeaderWords;
    for (int k = 0; k < P.tail; ++k) words += 2 * 4 * slots_of(P.level[k].grid.n);
    if (P.tail < P.count) words += 2 * 4 * slots_of(P.level[P.tail].grid.n);
    return words;
}

Level make_level(const FfxRelaxGrid& g) {
    Level L = {};
    for (int a = 0; a < 3; ++a) {
        L.n[a] = g.n[a];
        L.w[a] = g.inv[a] * g.inv[a];
    }
    L.x4 = up4(g.n[0]) / 4;
    L.ty = g.n[1];
    L.tz = g.n[2];
    return L;
}

// The levels from `first` on as one block's: the tail entries of `A`.
void tail_layout(const FfxRelaxPlan& P, int first, int shift, Params& A) {
    int off = 0;
    for (int k = first; k < P.count; ++k) {
        Level L = make_level(P.level[k].grid);
        L.p = off;
        off += L.x4 * (L.n[1] + 2) * (L.n[2] + 2);
        L.q = off;
        off += L.x4 * (L.n[1] + 2) * (L.n[2] + 2);
        L.r = off;
        off += L.x4 * L.n[1] * L.n[2];
        A.tv[k - shift] = L;
    }
    A.tail_f4 = off;
    A.work = off;
}

int tail_bytes(const FfxRelaxPlan& P, int first) {
    return 16 * tail_f4(P, first) + (P.basis ? 16 * cells_of(P.level[P.count - 1].grid.n) : 0);
}

template <bool MASK, bool ONE, bool RAGGED>
int launch_resident(const Params& A, int blocks, int smem, cudaStream_t st) {
    static std::atomic<uint64_t> ready{0};
    auto kernel = resident::resident_kernel<MASK, ONE, RAGGED>;
    if (int s = allow_smem(kernel, ready)) return s;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(resident::kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = blocks > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, A);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(FFX_ERR_LAUNCH, "resident_kernel: %s", cudaGetErrorString(e));
    }
    return launch_status("resident_kernel");
}

Params common_params(const FfxRelaxPlan& P, int cycles, float dt) {
    Params A = {};
    A.pre = P.pre;
    A.post = P.post;
    A.last = P.last_sweeps;
    A.cycles = cycles;
    A.omega = P.omega;
    A.dt = dt;
    A.basis = P.basis;
    return A;
}

// Whether rows of the levels from `first` on end in padding.
bool ragged(const FfxRelaxPlan& P, int first) {
    for (int k = first; k < P.count; ++k)
        if (P.level[k].grid.n[0] % 4) return true;
    return false;
}

// The levels from `first` on in one block, from zero unless p_in.
int run_one_block(const FfxRelaxPlan& P, int first, int cycles, float dt, const float* p_in, const float* rhs,
                  float* p_out, cudaStream_t st) {
    Params A = common_params(P, cycles, dt);
    A.count = P.count - first;
    A.from_zero = p_in == nullptr;
    A.p_in = p_in;
    A.rhs = rhs;
    A.p_out = p_out;
    tail_layout(P, first, first, A);
    const int smem = tail_bytes(P, first);
    FFX_REQUIRE(smem <= resident::kSmem && tail_level(P.level[first].grid.n), "relaxation tail out of range");
    return ragged(P, first) ? launch_resident<false, false, true>(A, 1, smem, st)
                            : launch_resident<false, false, false>(A, 1, smem, st);
}

// The whole solve in one cooperative launch.
int run_resident(const FfxRelaxPlan& P, int cycles, float dt, bool from_zero, float* p, cudaStream_t st) {
    Params A = common_params(P, cycles, dt);
    const int dist = P.tail;
    const bool tail = dist < P.count;
    A.count = P.count;
    A.dist = dist;
    A.gy = (P.level[0].grid.n[1] + P.tile[0] - 1) / P.tile[0];
    A.gz = (P.level[0].grid.n[2] + P.tile[1] - 1) / P.tile[1];
    A.from_zero = from_zero;
    A.p_in = p;
    A.p_out = p;
    A.rhs = P.level[0].rhs;
    A.cls = P.classes;
    A.vec = P.level[0].grid.n[0] % 4 == 0 && ((uintptr_t)A.rhs | (uintptr_t)p) % 16 == 0;
    A.ws = reinterpret_cast<resident::u64*>(P.workspace);
    A.epochs = reinterpret_cast<unsigned*>(A.ws);
    A.timeouts = A.epochs + 2 * kHeaderWords - 1;
    A.alarm = P.alarm;
    const int fit = tile_fit(P, dist, P.tile[0], P.tile[1]);
    FFX_REQUIRE(fit >= 0 && A.gy * A.gz < kHeaderWords * 2 - 2, "resident tile out of range");
    const bool one = fit == 1;
    int64_t word = kHeaderWords;
    int off = 0;
    unsigned exchanges = 2;
    for (int k = 0; k <= dist && k < P.count; ++k) {
        Level L = make_level(P.level[k].grid);
        L.ty = P.tile[0] >> k;
        L.tz = P.tile[1] >> k;
        L.p = L.q = off;
        off += L.x4 * (L.ty + 2) * (L.tz + 2);
        if (k < dist) {
            if (k > 0 || !one) {
                L.q = off;
                off += L.x4 * (L.ty + 2) * (L.tz + 2);
            }
            L.r = off;
            off += L.x4 * L.ty * L.tz;
            L.ll = word;
            word += 2 * 4 * slots_of(P.level[k].grid.n);
            exchanges += k == P.count - 1 ? P.last_sweeps : P.pre + P.post + 1;
        }
        A.lv[k] = L;
    }
    A.cls_off = off;
    if (P.classes) off += up4(A.lv[0].x4 * A.lv[0].ty * A.lv[0].tz) / 4;
    A.tile_f4 = off;
    A.epochs_used = exchanges * (unsigned)cycles + 2u;
    int smem = 16 * off;
    if (tail) {
        tail_layout(P, dist, 0, A);
        smem = std::max(smem, tail_bytes(P, dist));
        A.tail_rhs = word;
        A.tail_p = word + 4 * slots_of(P.level[dist].grid.n);
    }
    FFX_REQUIRE(smem <= resident::kSmem, "resident tile out of range");
    const int blocks = A.gy * A.gz + (tail ? 1 : 0);
    if (P.classes) return one ? launch_resident<true, true, false>(A, blocks, smem, st)
                              : launch_resident<true, false, false>(A, blocks, smem, st);
    if (ragged(P, 0)) return one ? launch_resident<false, true, true>(A, blocks, smem, st)
                                 : launch_resident<false, false, true>(A, blocks, smem, st);
    return one ? launch_resident<false, true, false>(A, blocks, smem, st)
               : launch_resident<false, false, false>(A, blocks, smem, st);
}

}  // namespace
}  // namespace ffx

using namespace ffx;

extern "C" {

int ffx_relax_plan(FfxRelaxPlan* P) {
    FFX_REQUIRE(P && P->count >= 1 && P->count <= FFX_RELAX_LEVELS && P->pre >= 1 && P->post >= 1 &&
                P->last_sweeps >= 1 && P->omega > 0.f, "ffx_relax_plan: invalid arguments");
    for (int k = 0; k < P->count; ++k) {
        FFX_REQUIRE(grid_valid(P->level[k].grid), "ffx_relax_plan: level %d is not a grid", k);
        if (k > 0)
            for (int a = 0; a < 3; ++a)
                FFX_REQUIRE(P->level[k - 1].grid.n[a] == 2 * P->level[k].grid.n[a],
                            "ffx_relax_plan: level %d does not halve", k);
    }
    FFX_REQUIRE(!P->basis || (P->count > 1 && cells_of(P->level[P->count - 1].grid.n) <= resident::kDirectCells),
                "ffx_relax_plan: direct solve too large");
    FFX_REQUIRE(!P->classes || P->count == 1, "ffx_relax_plan: classes go with one level");
    // the levels that one block holds; a direct solve is always among them
    P->tail = P->count;
    if (!P->classes)
        while (P->tail > 0 && tail_level(P->level[P->tail - 1].grid.n) &&
               tail_bytes(*P, P->tail - 1) <= resident::kSmem)
            --P->tail;
    FFX_REQUIRE(!P->basis || P->tail < P->count, "ffx_relax_plan: no block holds the coarsest level");
    P->tile[0] = P->tile[1] = 0;
    P->workspace_bytes = 0;
    P->sms = P->sms > 0 ? std::min(P->sms, resident_sms()) : resident_sms();
    if (P->tail == 0) return FFX_OK;
    if (plan_tiles(*P)) {
        P->workspace_bytes = 8 * published_words(*P);
        return FFX_OK;
    }
    for (int k = 0; k < P->tail; ++k) {
        FfxRelaxLevel& L = P->level[k];
        const bool last = k == P->count - 1;
        FFX_REQUIRE(plan_sweeps(L.grid.n, last ? P->last_sweeps : 6, P->classes != nullptr, L.sweep),
                    "ffx_relax_plan: no tile fits level %d", k);
        if (last) continue;
        FFX_REQUIRE(plan_fused(L.grid.n, P->pre, kDown, L.sweep, L.down) &&
                    plan_fused(L.grid.n, P->post, kUp, L.sweep, L.up), "ffx_relax_plan: no tile fits level %d", k);
    }
    return FFX_OK;
}

int ffx_relax_cycles(const FfxRelaxPlan* P, int32_t cycles, float dt, int32_t from_zero, int32_t* swapped,
                     void* stream) {
    FFX_REQUIRE(P && swapped && cycles >= 0 && P->count >= 1 && P->count <= FFX_RELAX_LEVELS && P->tail >= 0 &&
                P->tail <= P->count && P->pre >= 1 && P->post >= 1 && P->last_sweeps >= 1 && P->omega > 0.f &&
                dt > 0.f, "ffx_relax_cycles: invalid arguments");
    const bool fits = P->tail == 0 || P->tile[0] > 0;
    for (int k = 0; k < P->count; ++k) {
        const FfxRelaxLevel& L = P->level[k];
        FFX_REQUIRE(grid_valid(L.grid), "ffx_relax_cycles: level %d is not a grid", k);
        if (k > 0 && fits) continue;
        FFX_REQUIRE(L.p && L.rhs && (fits || (L.q && L.p != L.q)), "ffx_relax_cycles: level %d is incomplete", k);
        if (fits) continue;
        FFX_REQUIRE(k >= P->tail || (L.sweep.sweeps >= 1 &&
                                     (k == P->count - 1 || (L.down.sweeps >= 1 && L.down.sweeps <= P->pre &&
                                                            L.up.sweeps >= 1 && L.up.sweeps <= P->post))),
                    "ffx_relax_cycles: level %d is not planned", k);
    }
    FFX_REQUIRE(!P->classes || (P->count == 1 && (uintptr_t)P->classes % 4 == 0), "ffx_relax_cycles: invalid classes");
    cudaStream_t st = as_stream(stream);
    *swapped = 0;
    if (cycles == 0) return FFX_OK;
    float* p0 = P->level[0].p;
    if (P->tail == 0)
        return run_one_block(*P, 0, cycles, dt, from_zero ? nullptr : p0, P->level[0].rhs, p0, st);
    if (fits) {
        FFX_REQUIRE(P->workspace && (uintptr_t)P->workspace % 16 == 0, "ffx_relax_cycles: workspace missing");
        FFX_REQUIRE(resident_sms() >= P->sms, "ffx_relax_cycles: planned for %d SMs, the device has %d", P->sms,
                    resident_sms());
        return run_resident(*P, cycles, dt, from_zero != 0, p0, st);
    }
    float* cur[FFX_RELAX_LEVELS];
    float* other[FFX_RELAX_LEVELS];
    for (int k = 0; k < P->count; ++k) {
        cur[k] = P->level[k].p;
        other[k] = P->level[k].q;
    }
    const int bottom = std::min(P->tail, P->count - 1);     // levels above it have a coarser one
    for (int c = 0; c < cycles; ++c) {
        for (int k = 0; k < bottom; ++k) {
            const FfxRelaxLevel& L = P->level[k];
            const float step = k == 0 ? dt : 1.f;
            const int before = P->pre - L.down.sweeps;
            bool zero = k > 0 || (c == 0 && from_zero);
            if (before > 0) {
                if (int s = run_sweeps<false>(L.grid, L.sweep, L.rhs, nullptr, step, P->omega, before, zero, cur[k],
                                              other[k], st))
                    return s;
                zero = false;
            }
            Fields f = {zero ? nullptr : cur[k], L.rhs, other[k], nullptr, nullptr, P->level[k + 1].rhs};
            if (int s = launch_tile<kDown, false>(L.grid, L.down, f, step, P->omega, st)) return s;
            std::swap(cur[k], other[k]);
        }
        if (P->tail < P->count) {
            if (int s = run_one_block(*P, P->tail, 1, 1.f, nullptr, P->level[P->tail].rhs, cur[P->tail], st)) return s;
        } else {
            const FfxRelaxLevel& L = P->level[bottom];
            const bool zero = bottom > 0 || (c == 0 && from_zero);
            const float step = bottom == 0 ? dt : 1.f;
            const int s = P->classes ? run_sweeps<true>(L.grid, L.sweep, L.rhs, P->classes, step, P->omega,
                                                        P->last_sweeps, zero, cur[bottom], other[bottom], st)
                                     : run_sweeps<false>(L.grid, L.sweep, L.rhs, nullptr, step, P->omega,
                                                         P->last_sweeps, zero, cur[bottom], other[bottom], st);
            if (s) return s;
        }
        for (int k = bottom - 1; k >= 0; --k) {
            const FfxRelaxLevel& L = P->level[k];
            const float step = k == 0 ? dt : 1.f;
            Fields f = {cur[k], L.rhs, other[k], nullptr, cur[k + 1], nullptr};
            if (int s = launch_tile<kUp, false>(L.grid, L.up, f, step, P->omega, st)) return s;
            std::swap(cur[k], other[k]);
            const int after = P->post - L.up.sweeps;
            if (after > 0)
                if (int s = run_sweeps<false>(L.grid, L.sweep, L.rhs, nullptr, step, P->omega, after, false, cur[k],
                                              other[k], st))
                    return s;
        }
    }
    *swapped = cur[0] != p0;
    return FFX_OK;
}

int ffx_relax_reset(const FfxRelaxPlan* P, void* stream) {
    FFX_REQUIRE(P, "ffx_relax_reset: invalid arguments");
    if (!P->workspace || P->workspace_bytes == 0) return FFX_OK;
    return cuda_status(cudaMemsetAsync(P->workspace, 0, (size_t)P->workspace_bytes, as_stream(stream)),
                       "ffx_relax_reset");
}

int ffx_relax_timeouts(const FfxRelaxPlan* P, int32_t* count, void* stream) {
    FFX_REQUIRE(P && count, "ffx_relax_timeouts: invalid arguments");
    *count = 0;
    if (!P->workspace || P->workspace_bytes == 0) return FFX_OK;
    unsigned v = 0;
    cudaStream_t st = as_stream(stream);
    cudaError_t e = cudaMemcpyAsync(&v, reinterpret_cast<const unsigned*>(P->workspace) + 2 * kHeaderWords - 1, sizeof v,
                                    cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_status(e, "ffx_relax_timeouts");
    *count = (int32_t)v;
    return FFX_OK;
}

int ffx_relax_classes(const int32_t n[3], const uint8_t* solid, uint8_t* classes, void* stream) {
    FFX_REQUIRE(shape_ok(n) && solid && classes, "ffx_relax_classes: invalid arguments");
    relax_classes_kernel<<<cell_grid(up4(n[0]), n[1], n[2]), cell_block(), 0, as_stream(stream)>>>(n[0], n[1], n[2],
                                                                                                   solid, classes);
    return launch_status("relax_classes_kernel");
}

}  // extern "C"
