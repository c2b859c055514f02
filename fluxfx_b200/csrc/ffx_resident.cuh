// Relaxation with the iterate resident on the chip: one cooperative launch
// for a whole solve (all Jacobi sweeps, or all V-cycles) of a grid that fits
// the shared memory of the SMs.
//
// A launch per sweep costs about 3 us however small the level, and fusing T
// sweeps in a tile with a halo of T cells recomputes two to four times the
// cells. Here every block keeps its tile's pressure and
// right-hand side in shared memory for the whole solve and only the rows at
// the tile's rim travel: after a sweep a block publishes them in global memory
// and takes its neighbours' rows from there. A published word is 64 bits, the
// value with the number of the exchange, stored and loaded as one word, so the
// reader polls the data itself and no barrier, fence or flag stands between.
//
//   blocks 0 .. gy gz - 1   tiles of rows (y, z), the full x extent each, of
//                           the levels 0 .. dist - 1;
//   block gy gz             the levels below (at most kTailSlots float4), whole,
//                           where there are any: it waits for the restricted
//                           residual and publishes the correction.
// With dist = 0 one block holds every level and reads and writes global memory.
//
// What bounds a sweep now is the exchange and the latency of a few instructions:
// 1.2 us at 32^3, where a block relaxes 64 float4; a third of the issue slots are
// used, and the warps wait at barriers, behind those that poll
// (profiles/resident_solves.txt).
// Measured, us per sweep, a launch per sweep (T fused sweeps per launch) ->
// resident: 75 x 61 x 93 5.5 (3.5) -> 2.1, 64^3 4.1 (3.4) -> 1.5, 127^3 12 (11)
// -> 5.3; us per V(3,3) cycle: 128^3 250 (143) -> 73, 32^3 95 (40) -> 24.
//
// Blocks wait for one another, so the launch is cooperative (all blocks
// resident at once); every wait is bounded: after kSpinLimit polls a block
// stops waiting, counts a timeout, tells the host (Waits) and runs to its end.
#pragma once
#include "ffx_host.cuh"

namespace ffx {
namespace resident {

constexpr int kThreads = 512;
constexpr int kLevels = 12;
constexpr int kTailSlots = 1024;
constexpr int kRimItems = 4;         // float4 of the rim a thread takes in
constexpr int kDirectCells = 512;
constexpr int kSmem = 220 * 1024;
constexpr int kSpinLimit = 1 << 21;

using u64 = unsigned long long;

struct Level {
    int n[3], x4;
    int ty, tz;          // rows of a tile (the grid's own in the tail)
    int p, q, r;         // shared-memory float4 offsets; q = p where there is one copy of the pressure
    float w[3];
    int64_t ll;          // published rows: words from the start of the workspace
};

struct Params {
    int count, dist, gy, gz;
    int pre, post, last, cycles;
    float omega, dt;
    int from_zero, vec;
    const float* p_in;
    const float* rhs;
    float* p_out;
    const uint8_t* cls;          // masked sweeps: table entries, rows of up4(nx) bytes
    int cls_off;                 // their shared-memory offset (float4)
    const double* basis;
    int work;                    // float4 offset of the direct solve's FP64 arrays (tail)
    u64* ws;
    int64_t tail_rhs, tail_p;    // words
    unsigned* epochs;            // exchange number reached, per block
    unsigned epochs_used;        // exchanges a launch may number
    unsigned* timeouts;
    int* alarm;                  // host memory, or NULL (Waits)
    int tile_f4, tail_f4;        // float4 of shared memory to clear, by role
    Level lv[kLevels];           // tiles: levels 0 .. dist (dist: the tail's level, its pressure only)
    Level tv[kLevels];           // tail: levels dist .. count - 1
};

// diag and omega / diag by open neighbours: entry cx + 3 cy + 9 cz for cx, cy,
// cz open neighbours along the axes; omega / diag is 0 where there are none,
// and in entry 27 (a solid cell or padding).
__device__ __forceinline__ void fill_table(float2* kd, int i, const float* w, float omega) {
    if (i < 0 || i >= 28) return;
    const float diag = i == 27 ? 0.f
                               : (float)(i % 3) * w[0] + (float)(i / 3 % 3) * w[1] + (float)(i / 9) * w[2];
    kd[i] = make_float2(diag > 0.f ? omega / diag : 0.f, diag);
}

__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ unsigned byte_of(unsigned v, int j) { return v >> (8 * j) & 255u; }
__device__ __forceinline__ void weights_of(unsigned codes, const float2* kd, float4& k, float4& d) {
    const float2 a = kd[byte_of(codes, 0)], b = kd[byte_of(codes, 1)], c = kd[byte_of(codes, 2)],
                 e = kd[byte_of(codes, 3)];
    k = make_float4(a.x, b.x, c.x, e.x);
    d = make_float4(a.y, b.y, c.y, e.y);
}

// A sweep's result: 0 in the cells without a weight (colliders, isolated cells,
// padding), whatever stands beside them. Selected, not multiplied: 0 times an
// infinity would carry it through a wall. Without colliders only a row's padding
// has none (`left` cells of the float4 lie in the row), and rows of whole float4
// have no padding (RAGGED false): a projection of 128^3 takes 224 us with the
// weights tested, 223 with the row's end tested, 219 with neither.
template <bool MASK, bool RAGGED>
__device__ __forceinline__ float4 weighted(float4 k, int left, float4 o) {
    if (MASK)
        return make_float4(k.x > 0.f ? o.x : 0.f, k.y > 0.f ? o.y : 0.f, k.z > 0.f ? o.z : 0.f, k.w > 0.f ? o.w : 0.f);
    if (!RAGGED) return o;
    return make_float4(o.x, left > 1 ? o.y : 0.f, left > 2 ? o.z : 0.f, left > 3 ? o.w : 0.f);
}

// n / d for 0 <= n < 2^16 and 1 <= d < 2^12, with inv = 1 / d: (n + 1/2) / d is
// at least 1 / (2 d) from an integer, far more than the rounding.
__device__ __forceinline__ int quotient(int n, float inv) { return __float2int_rd(((float)n + 0.5f) * inv); }

// A block's rows of a level: P (and Q, its second copy) has a rim of one row on
// every side, R none.
struct View {
    int n[3], x4, ty, tz, y0, z0, flat, plane;      // float4 of a plane of R and of P
    float inv_x4, inv_flat, inv_plane;
    float w[3];
    float4* P;
    float4* Q;
    float4* R;
    u64* ll;
    __device__ __forceinline__ int at(int x, int y, int z) const { return x + x4 * (y + 1) + plane * (z + 1); }
    // slot s of R's order, item s of P's order (rim included, from -1)
    __device__ __forceinline__ void slot(int s, int& x, int& y, int& z) const {
        z = quotient(s, inv_flat);
        const int it = s - z * flat;
        y = quotient(it, inv_x4);
        x = it - y * x4;
    }
    __device__ __forceinline__ void item(int s, int& x, int& y, int& z) const {
        z = quotient(s, inv_plane);
        const int it = s - z * plane;
        y = quotient(it, inv_x4);
        x = it - y * x4;
        --y;
        --z;
    }
};

__device__ __forceinline__ View make_view(const Level& L, int by, int bz, float4* smem, u64* ws, bool flip) {
    View v;
#pragma unroll
    for (int a = 0; a < 3; ++a) { v.n[a] = L.n[a]; v.w[a] = L.w[a]; }
    v.x4 = L.x4;
    v.y0 = by * L.ty;
    v.z0 = bz * L.tz;
    v.ty = min(L.ty, L.n[1] - v.y0);
    v.tz = min(L.tz, L.n[2] - v.z0);
    v.flat = L.x4 * v.ty;
    v.plane = L.x4 * (v.ty + 2);
    v.inv_x4 = __frcp_rn((float)v.x4);
    v.inv_flat = __frcp_rn((float)v.flat);
    v.inv_plane = __frcp_rn((float)v.plane);
    v.P = smem + (flip ? L.q : L.p);
    v.Q = smem + (flip ? L.p : L.q);
    v.R = smem + L.r;
    v.ll = ws ? ws + L.ll : nullptr;
    return v;
}

// ------------------------------------------------------- published values
__device__ __forceinline__ u64 pack(float v, unsigned epoch) {
    return (u64)epoch << 32 | (u64)__float_as_uint(v);
}
__device__ __forceinline__ void put4(u64* to, float4 v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(to), "l"(pack(v.x, epoch)),
                 "l"(pack(v.y, epoch))
                 : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(to + 2), "l"(pack(v.z, epoch)),
                 "l"(pack(v.w, epoch))
                 : "memory");
}
__device__ __forceinline__ void put1(u64* to, float v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(to), "l"(pack(v, epoch)) : "memory");
}
__device__ __forceinline__ bool get4(const u64* from, unsigned epoch, float4& v) {
    u64 a, b, c, d;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(from) : "memory");
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "l"(from + 2) : "memory");
    v = make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)b), __uint_as_float((unsigned)c),
                    __uint_as_float((unsigned)d));
    return (unsigned)(a >> 32) == epoch && (unsigned)(b >> 32) == epoch && (unsigned)(c >> 32) == epoch &&
           (unsigned)(d >> 32) == epoch;
}

// The bounded waits of a block: once one has given up the others no longer wait, the
// device's count goes up and the word that the host watches is set.
struct Waits {
    volatile int* dead;
    unsigned* timeouts;
    int* alarm;
    __device__ __forceinline__ bool over() const { return *dead != 0; }
    __device__ __forceinline__ void give_up() const {
        *dead = 1;
        atomicAdd(timeouts, 1u);
        if (alarm) atomicExch_system(alarm, 1);
    }
};

// One bounded poll loop over up to kRimItems float4 of a thread: words
// `base + from[u]` (from[u] < 0: none) into `to + dst[u]`.
__device__ __forceinline__ void collect(const u64* base, const int (&from)[kRimItems], float4* to,
                                        const int (&dst)[kRimItems], unsigned epoch, const Waits& waits) {
    unsigned pending = 0;
#pragma unroll
    for (int u = 0; u < kRimItems; ++u) pending |= from[u] >= 0 ? 1u << u : 0u;
    for (int spin = 0; pending; ++spin) {
#pragma unroll
        for (int u = 0; u < kRimItems; ++u) {
            float4 v;
            if ((pending >> u & 1u) && get4(base + from[u], epoch, v)) {
                to[dst[u]] = v;
                pending &= ~(1u << u);
            }
        }
        if ((spin & 255) == 255 && pending) {
            if (waits.over()) return;
            if (spin >= kSpinLimit) {
                waits.give_up();
                return;
            }
        }
    }
}

// What an exchange of a level's rim needs; `on` is false in the tail.
struct Exchange {
    bool on;
    unsigned epoch;      // of the next exchange
    unsigned turn;       // bit k: which of level k's two published copies comes next
    Waits waits;
};

// Words of row (gy, gz)'s float4 x in a level's published rows.
__device__ __forceinline__ int published(const View& v, int x, int gy, int gz) {
    return 4 * (x + v.x4 * (gy + v.n[1] * gz));
}

// The rows around the tile, corners included (the prolongation reads them, and
// a block that has all eight neighbours' rows of one exchange knows that they
// have read its rows of the exchange before, so two copies suffice).
__device__ __forceinline__ void rim_items(const View& v, int (&from)[kRimItems], int (&dst)[kRimItems]) {
    const int top = v.ty + 2, items = (2 * top + 2 * v.tz) * v.x4;
#pragma unroll
    for (int u = 0; u < kRimItems; ++u) {
        const int i = threadIdx.x + u * kThreads;
        from[u] = -1;
        dst[u] = 0;
        if (i < items) {
            const int row = quotient(i, v.inv_x4), x = i - row * v.x4;
            const int q = row - 2 * top;
            const int z = q >= 0 ? q >> 1 : (row < top ? -1 : v.tz);
            const int y = q >= 0 ? (q & 1 ? v.ty : -1) : (row < top ? row : row - top) - 1;
            const int gy = v.y0 + y, gz = v.z0 + z;
            if (gy >= 0 && gz >= 0 && gy < v.n[1] && gz < v.n[2]) {
                from[u] = published(v, x, gy, gz);
                dst[u] = v.at(x, y, z);
            }
        }
    }
}

// ------------------------------------------------------------------ passes
// `count` weighted Jacobi sweeps:
//   out = old + (omega / diag) (sum_a w_a (lower + upper) + nr - diag old),  nr = -rhs / dt.
// Cells outside the domain and in colliders hold 0, so they add nothing to the
// sum; diag counts the open neighbours. A thread owns a run of float4 along z.
// With two copies of the pressure a sweep goes from P to Q and the copies
// change places (the caller flips the level by count's parity); with one copy
// (ONE) it works in place.
// With an exchange, the rim is current again after every sweep.
template <bool MASK, bool ONE, bool RAGGED>
__device__ __forceinline__ void relax(View& v, int level, const float2* kd, const unsigned* cls, bool zero, int count,
                                      Exchange& ex) {
    const int tid = threadIdx.x;
    const int groups = min(max(quotient(kThreads, v.inv_flat), 1), v.tz);
    const int run = quotient(v.tz + groups - 1, __frcp_rn((float)groups));
    const int g = quotient(tid, v.inv_flat), it = tid - g * v.flat, y = quotient(it, v.inv_x4), x = it - y * v.x4;
    const int z0 = g * run, mine = g < groups ? max(min(run, v.tz - z0), 0) : 0;
    const int i0 = v.at(x, y, z0), r0 = x + v.x4 * (y + v.ty * z0);
    float4 k0 = zero4(), d0 = zero4();
    unsigned edge = 0;
    if (!MASK && mine > 0) {
        const int gy = v.y0 + y, cy = 2 - (gy == 0) - (gy == v.n[1] - 1);
        unsigned inner = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gx = 4 * x + j;
            const unsigned c = (unsigned)(2 - (gx == 0) - (gx == v.n[0] - 1) + 3 * cy);
            inner |= (gx < v.n[0] ? c + 18u : 27u) << (8 * j);
            edge |= (gx < v.n[0] ? c + 9u : 27u) << (8 * j);
        }
        weights_of(inner, kd, k0, d0);
    }
    int from[kRimItems], dst[kRimItems];
    u64* mine_out = nullptr;
    if (ex.on) {
        rim_items(v, from, dst);
        mine_out = v.ll + published(v, x, v.y0 + y, v.z0 + z0);
    }
    const int out_step = 4 * v.x4 * v.n[1];
    const int64_t copy = 4 * (int64_t)v.x4 * v.n[1] * v.n[2];
    const float wx = v.w[0], wy = v.w[1], wz = v.w[2];
    const int in_row = v.n[0] - 4 * x;
    const bool left = x > 0, right = x + 1 < v.x4, rim_y = y == 0 || y == v.ty - 1;
    auto formed = [&](const float4* P, int j, bool blank, float4& lo, float4& c, float4 hi) {
        const int i = i0 + j * v.plane;
        const float4 r = v.R[r0 + j * v.flat];
        float4 k = k0, d = d0;
        if (MASK) {
            weights_of(cls[r0 + j * v.flat], kd, k, d);
        } else {
            const int gz = v.z0 + z0 + j;
            if (gz == 0 || gz == v.n[2] - 1) weights_of(edge, kd, k, d);
        }
        if (blank) return weighted<MASK, RAGGED>(k, in_row, make_float4(k.x * r.x, k.y * r.y, k.z * r.z, k.w * r.w));
        const float4 ym = P[i - v.x4], yp = P[i + v.x4];
        const float* row = reinterpret_cast<const float*>(P) + 4 * i;
        const float xl = left ? row[-1] : 0.f, xr = right ? row[4] : 0.f;
        float4 o;
        o.x = fmaf(wz, lo.x + hi.x, fmaf(wy, ym.x + yp.x, fmaf(wx, xl + c.y, r.x)));
        o.y = fmaf(wz, lo.y + hi.y, fmaf(wy, ym.y + yp.y, fmaf(wx, c.x + c.z, r.y)));
        o.z = fmaf(wz, lo.z + hi.z, fmaf(wy, ym.z + yp.z, fmaf(wx, c.y + c.w, r.z)));
        o.w = fmaf(wz, lo.w + hi.w, fmaf(wy, ym.w + yp.w, fmaf(wx, c.z + xr, r.w)));
        o = make_float4(fmaf(k.x, fmaf(-d.x, c.x, o.x), c.x), fmaf(k.y, fmaf(-d.y, c.y, o.y), c.y),
                        fmaf(k.z, fmaf(-d.z, c.z, o.z), c.z), fmaf(k.w, fmaf(-d.w, c.w, o.w), c.w));
        lo = c;
        c = hi;
        return weighted<MASK, RAGGED>(k, in_row, o);
    };
    for (int s = 0; s < count; ++s) {
        const bool blank = zero && s == 0;
        const int64_t half = ex.turn >> level & 1u ? copy : 0;
        auto publish = [&](int j, float4 o) {
            if (ex.on && (rim_y || z0 + j == 0 || z0 + j == v.tz - 1)) put4(mine_out + half + j * out_step, o, ex.epoch);
        };
        float4 lo = zero4(), c = zero4();
        if (mine > 0 && !blank) {
            lo = v.P[i0 - v.plane];
            c = v.P[i0];
        }
        if (ONE) {
            // a plane at a time: the values above the run are read before anything is
            // written, and a plane is written when every thread has formed its part of it
            const float4 top = mine > 0 && !blank ? v.P[i0 + mine * v.plane] : zero4();
            __syncthreads();
            for (int j = 0; j < run; ++j) {
                float4 o = zero4();
                if (j < mine) {
                    o = formed(v.P, j, blank, lo, c, j == mine - 1 ? top : v.P[i0 + (j + 1) * v.plane]);
                    publish(j, o);
                }
                __syncthreads();
                if (j < mine) v.P[i0 + j * v.plane] = o;
            }
        } else {
            for (int j = 0; j < mine; ++j) {
                const float4 o = formed(v.P, j, blank, lo, c, v.P[i0 + (j + 1) * v.plane]);
                publish(j, o);
                v.Q[i0 + j * v.plane] = o;
            }
        }
        if (ex.on) {
            collect(v.ll + half, from, ONE ? v.P : v.Q, dst, ex.epoch, ex.waits);
            ex.turn ^= 1u << level;
            ++ex.epoch;
        }
        __syncthreads();
        if (!ONE) {
            float4* t = v.P;
            v.P = v.Q;
            v.Q = t;
        }
    }
}

// mg_residual.glsl for a float4 (rhs/dt - lap): the differences are formed
// before they are weighted, as the shader does. Negated.
__device__ __forceinline__ float4 minus_residual(const View& v, int x, int y, int z) {
    const int i = v.at(x, y, z), gy = v.y0 + y, gz = v.z0 + z;
    const float4 c = v.P[i];
    const float4 ym = gy > 0 ? v.P[i - v.x4] : c, yp = gy + 1 < v.n[1] ? v.P[i + v.x4] : c;
    const float4 zm = gz > 0 ? v.P[i - v.plane] : c, zp = gz + 1 < v.n[2] ? v.P[i + v.plane] : c;
    const float* row = reinterpret_cast<const float*>(v.P) + 4 * i;
    const int last = v.n[0] - 4 * x;     // cells from here to the end of the row
    const float xl = x > 0 ? row[-1] : c.x;
    const float e1 = last > 1 ? c.y : c.x, e2 = last > 2 ? c.z : c.y, e3 = last > 3 ? c.w : c.z,
                e4 = last > 4 ? row[4] : c.w;
    const float4 r = v.R[x + v.x4 * (y + v.ty * z)];
    const float wx = v.w[0], wy = v.w[1], wz = v.w[2];
    auto term = [&](float xm, float xp, float a, float b, float e, float f, float m, float s) {
        s = fmaf(wx, (xm - m) + (xp - m), s);
        s = fmaf(wy, (a - m) + (b - m), s);
        return fmaf(wz, (e - m) + (f - m), s);
    };
    return make_float4(term(xl, e1, ym.x, yp.x, zm.x, zp.x, c.x, r.x), term(c.x, e2, ym.y, yp.y, zm.y, zp.y, c.y, r.y),
                       term(c.y, e3, ym.z, yp.z, zm.z, zp.z, c.z, r.z), term(c.z, e4, ym.w, yp.w, zm.w, zp.w, c.w, r.w));
}

// mg_restrict.glsl of the residual: the two coarse cells over float4 x of the
// rows 2Y, 2Y + 1 and planes 2Z, 2Z + 1. store(coarse x, value) of each in the grid.
template <class Store>
__device__ __forceinline__ void restrict_pair(const View& v, int x, int Y, int Z, Store&& store) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 r = minus_residual(v, x, 2 * Y + (k & 1), 2 * Z + (k >> 1));
        a += r.x + r.y;
        b += r.z + r.w;
    }
    store(2 * x, -0.125f * a);
    if (4 * x + 2 < v.n[0]) store(2 * x + 1, -0.125f * b);
}

// mg_prolong.glsl for float4 (x, y, z) of `v` from the coarse rows of `c`:
// cell-centred trilinear interpolation with clamped coarse indices.
__device__ __forceinline__ float4 prolonged(const View& v, const View& c, int x, int y, int z) {
    const int gy = v.y0 + y, gz = v.z0 + z;
    const int by = (gy + 1) / 2 - 1, bz = (gz + 1) / 2 - 1;
    const float fy = gy & 1 ? 0.25f : 0.75f, fz = gz & 1 ? 0.25f : 0.75f;
    const int ya = max(by, 0) - c.y0, yb = min(by + 1, c.n[1] - 1) - c.y0;
    const int za = max(bz, 0) - c.z0, zb = min(bz + 1, c.n[2] - 1) - c.z0;
    const float w00 = (1.f - fy) * (1.f - fz), w10 = fy * (1.f - fz), w01 = (1.f - fy) * fz, w11 = fy * fz;
    const float* P = reinterpret_cast<const float*>(c.P);
    const float *r00 = P + 4 * c.at(0, ya, za), *r10 = P + 4 * c.at(0, yb, za), *r01 = P + 4 * c.at(0, ya, zb),
                *r11 = P + 4 * c.at(0, yb, zb);
    float t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int X = min(max(2 * x - 1 + j, 0), c.n[0] - 1);
        t[j] = fmaf(w11, r11[X], fmaf(w01, r01[X], fmaf(w10, r10[X], w00 * r00[X])));
    }
    const int last = v.n[0] - 4 * x;
    return make_float4(fmaf(0.75f, t[1], 0.25f * t[0]), last > 1 ? fmaf(0.25f, t[2], 0.75f * t[1]) : 0.f,
                       last > 2 ? fmaf(0.75f, t[2], 0.25f * t[1]) : 0.f,
                       last > 3 ? fmaf(0.25f, t[3], 0.75f * t[2]) : 0.f);
}

// P += the prolonged correction, on the tile and on the rim around it (the
// coarse rim reaches under this one, so nothing is exchanged).
__device__ __forceinline__ void prolong(const View& v, const View& c) {
    const int all = v.plane * (v.tz + 2);
    for (int s = threadIdx.x; s < all; s += kThreads) {
        int x, y, z;
        v.item(s, x, y, z);
        const int gy = v.y0 + y, gz = v.z0 + z;
        if (gy < 0 || gz < 0 || gy >= v.n[1] || gz >= v.n[2]) continue;
        const float4 add = prolonged(v, c, x, y, z);
        const float4 p = v.P[s];
        v.P[s] = make_float4(p.x + add.x, p.y + add.y, p.z + add.z, p.w + add.w);
    }
    __syncthreads();
}

// The Neumann pseudoinverse of the coarsest level in its separable cosine
// basis (physics/coarse_pressure.py): three forward contractions, a division
// by the eigenvalues, three back, in FP64. basis: bx (nx x nx, a row per mode),
// by, bz, 1 / eigenvalue per mode (0 for the constant mode). To FP64 rounding
// it is the dense pseudoinverse's product, in 6 n^4 instead of n^6 terms.
__device__ __forceinline__ void separable_solve(const View& v, double* wk, const double* __restrict__ basis) {
    const int tid = threadIdx.x;
    const int nx = v.n[0], ny = v.n[1], nz = v.n[2], N = nx * ny * nz;
    const float* R = reinterpret_cast<const float*>(v.R);
    float* P = reinterpret_cast<float*>(v.P);
    double* a = wk;
    double* c = wk + N;
    const double* bx = basis;
    const double* by = bx + nx * nx;
    const double* bz = by + ny * ny;
    const double* inv = bz + nz * nz;
    const int x = tid % nx, y = tid / nx % ny, z = tid / (nx * ny);
    const bool on = tid < N;
    if (on) a[tid] = -(double)R[x + 4 * v.x4 * (y + ny * z)];     // R holds -rhs / dt
    __syncthreads();
    auto line = [&](const double* from, const double* m, int step, int n, int stride, int base) {
        double s = 0.0;
        for (int j = 0; j < n; ++j) s += __ldg(m + j * step) * from[base + stride * j];
        return s;
    };
    const int lx = nx * (y + ny * z), ly = x + nx * ny * z, lz = x + nx * y;
    if (on) c[tid] = line(a, bx + x * nx, 1, nx, 1, lx);
    __syncthreads();
    if (on) a[tid] = line(c, by + y * ny, 1, ny, nx, ly);
    __syncthreads();
    if (on) c[tid] = line(a, bz + z * nz, 1, nz, nx * ny, lz) * __ldg(inv + tid);
    __syncthreads();
    if (on) a[tid] = line(c, bz + z, nz, nz, nx * ny, lz);
    __syncthreads();
    if (on) c[tid] = line(a, by + y, ny, ny, nx, ly);
    __syncthreads();
    if (on) P[4 * v.at(0, y, z) + x] = (float)line(c, bx + x, nx, nx, 1, lx);
    __syncthreads();
}

// ------------------------------------------------------------------- roles
// A block with whole levels (the tail, or everything when dist = 0).
template <bool RAGGED>
__device__ __forceinline__ void run_tail(const Params& A, float4* smem, float2 (*kd)[28], const Waits& waits,
                                         unsigned base) {
    const int tid = threadIdx.x;
    Exchange none = {false, 0u, 0u, waits};
    unsigned flip = 0;       // bit k: level k's pressure is in its second copy
    auto view = [&](int k) { return make_view(A.tv[k], 0, 0, smem, nullptr, flip >> k & 1u); };
    auto smooth = [&](View& v, int k, bool zero, int count) {
        relax<false, false, RAGGED>(v, 0, kd[k], nullptr, zero, count, none);
        flip ^= (unsigned)(count & 1) << k;
    };
    const int first = A.dist, last = A.count - 1;
    const View top = view(first);
    const int cells = top.n[0] * top.n[1] * top.n[2], slots = top.flat * top.tz;
    if (first == 0) {
        float* R = reinterpret_cast<float*>(top.R);
        float* P = reinterpret_cast<float*>(top.P);
        for (int i = tid; i < cells; i += kThreads) {
            const int yz = i / top.n[0], x = i - yz * top.n[0], z = yz / top.n[1], y = yz - z * top.n[1];
            float q = __ldg(A.rhs + i);
            if (A.dt != 1.f) q = q / A.dt;
            R[x + 4 * top.x4 * yz] = -q;
            if (!A.from_zero) P[4 * top.at(0, y, z) + x] = A.p_in[i];
        }
        __syncthreads();
    }
    for (int c = 0; c < A.cycles; ++c) {
        const unsigned epoch = base + (unsigned)c + 1u;
        if (first > 0) {
            for (int at = tid; at < slots; at += kThreads * kRimItems) {
                int from[kRimItems], dst[kRimItems];
#pragma unroll
                for (int u = 0; u < kRimItems; ++u) {
                    const int s = at + u * kThreads;
                    from[u] = s < slots ? 4 * s : -1;
                    dst[u] = s;
                }
                collect(A.ws + A.tail_rhs, from, top.R, dst, epoch, waits);
            }
            __syncthreads();
        }
        for (int k = first; k <= last; ++k) {
            View v = view(k);
            const bool zero = k > 0 || (c == 0 && A.from_zero);
            if (k == last && A.basis) {
                separable_solve(v, reinterpret_cast<double*>(smem + A.work), A.basis);
                break;
            }
            smooth(v, k, zero, k == last ? A.last : A.pre);
            if (k == last) break;
            const View w = view(k + 1);
            float* r = reinterpret_cast<float*>(w.R);
            const int pairs = v.x4 * w.n[1] * w.n[2];
            const float inv_hy = __frcp_rn((float)w.n[1]);
            for (int i = tid; i < pairs; i += kThreads) {
                const int yz = quotient(i, v.inv_x4), x = i - yz * v.x4, Z = quotient(yz, inv_hy), Y = yz - Z * w.n[1];
                restrict_pair(v, x, Y, Z, [&](int X, float q) { r[X + 4 * w.x4 * yz] = -q; });
            }
            __syncthreads();
        }
        for (int k = last - 1; k >= first; --k) {
            View v = view(k);
            prolong(v, view(k + 1));
            smooth(v, k, false, A.post);
        }
        if (first > 0) {
            const View v = view(first);
            for (int s = tid; s < slots; s += kThreads) {
                int x, y, z;
                v.slot(s, x, y, z);
                put4(A.ws + A.tail_p + 4 * s, v.P[v.at(x, y, z)], epoch);
            }
        }
    }
    if (first == 0) {
        const float* P = reinterpret_cast<const float*>(view(0).P);
        for (int i = tid; i < cells; i += kThreads) {
            const int yz = i / top.n[0], x = i - yz * top.n[0], z = yz / top.n[1], y = yz - z * top.n[1];
            A.p_out[i] = P[4 * top.at(0, y, z) + x];
        }
    }
}

// A block with a tile of the levels 0 .. dist - 1.
template <bool MASK, bool ONE, bool RAGGED>
__device__ __forceinline__ void run_tile(const Params& A, float4* smem, float2 (*kd)[28], const Waits& waits,
                                         unsigned base) {
    const int tid = threadIdx.x;
    const int by = blockIdx.x % A.gy, bz = blockIdx.x / A.gy;
    unsigned flip = 0;
    auto view = [&](int k) { return make_view(A.lv[k], by, bz, smem, A.ws, flip >> k & 1u); };
    Exchange ex = {true, base + 1u, 0u, waits};
    unsigned* cls = reinterpret_cast<unsigned*>(smem + A.cls_off);
    auto smooth = [&](View& v, int k, bool zero, int count) {
        if (k == 0) {
            relax<MASK, ONE, RAGGED>(v, 0, kd[0], cls, zero, count, ex);
            if (!ONE) flip ^= (unsigned)(count & 1);
        } else {
            relax<false, false, RAGGED>(v, k, kd[k], nullptr, zero, count, ex);
            flip ^= (unsigned)(count & 1) << k;
        }
    };
    // this tile of the fields, the pressure with its rim (read before anything is
    // published, so before any block can have finished and written its tile)
    {
        const View v = view(0);
        const int slots = v.flat * v.tz;
        for (int s = tid; s < slots; s += kThreads) {
            int x, y, z;
            v.slot(s, x, y, z);
            const int line = (v.y0 + y) + v.n[1] * (v.z0 + z), left = v.n[0] - 4 * x;
            const float* src = A.rhs + 4 * x + (int64_t)v.n[0] * line;
            float4 r = zero4();
            if (A.vec) {
                r = __ldg(reinterpret_cast<const float4*>(src));
            } else {
                r.x = __ldg(src);
                if (left > 1) r.y = __ldg(src + 1);
                if (left > 2) r.z = __ldg(src + 2);
                if (left > 3) r.w = __ldg(src + 3);
            }
            if (A.dt != 1.f) r = make_float4(r.x / A.dt, r.y / A.dt, r.z / A.dt, r.w / A.dt);
            v.R[s] = make_float4(-r.x, -r.y, -r.z, -r.w);
            if (MASK) cls[s] = __ldg(reinterpret_cast<const unsigned*>(A.cls) + x + (int64_t)v.x4 * line);
        }
        if (!A.from_zero) {
            const int all = v.plane * (v.tz + 2);
            for (int s = tid; s < all; s += kThreads) {
                int x, y, z;
                v.item(s, x, y, z);
                const int gy = v.y0 + y, gz = v.z0 + z;
                if (gy < 0 || gz < 0 || gy >= v.n[1] || gz >= v.n[2]) continue;
                const int line = gy + v.n[1] * gz, left = v.n[0] - 4 * x;
                const float* src = A.p_in + 4 * x + (int64_t)v.n[0] * line;
                float4 p = zero4();
                if (A.vec) {
                    p = *reinterpret_cast<const float4*>(src);
                } else {
                    p.x = src[0];
                    if (left > 1) p.y = src[1];
                    if (left > 2) p.z = src[2];
                    if (left > 3) p.w = src[3];
                }
                if (MASK) {
                    // a solid or isolated cell's pressure is 0 from the first sweep on
                    const unsigned t = __ldg(reinterpret_cast<const unsigned*>(A.cls) + x + (int64_t)v.x4 * line);
                    auto gone = [&](int j) { return byte_of(t, j) == 27u || byte_of(t, j) == 0u; };
                    p = make_float4(gone(0) ? 0.f : p.x, gone(1) ? 0.f : p.y, gone(2) ? 0.f : p.z, gone(3) ? 0.f : p.w);
                }
                v.P[s] = p;
            }
        }
        __syncthreads();
    }
    const int low = min(A.dist, A.count - 1);       // the lowest level the tiles prolong from
    for (int c = 0; c < A.cycles; ++c) {
        const unsigned epoch = base + (unsigned)c + 1u;     // of the words to and from the tail
        for (int k = 0; k < A.dist; ++k) {
            View v = view(k);
            smooth(v, k, k > 0 || (c == 0 && A.from_zero), k == A.count - 1 ? A.last : A.pre);
            if (k == A.count - 1) break;
            const Level& C = A.lv[k + 1];
            const int hy = v.ty / 2, pairs = v.x4 * hy * (v.tz / 2);
            const float inv_hy = __frcp_rn((float)hy);
            float* r = reinterpret_cast<float*>(smem + C.r);
            for (int i = tid; i < pairs; i += kThreads) {
                const int yz = quotient(i, v.inv_x4), x = i - yz * v.x4, Z = quotient(yz, inv_hy), Y = yz - Z * hy;
                if (k + 1 < A.dist) {
                    restrict_pair(v, x, Y, Z, [&](int X, float q) { r[X + 4 * C.x4 * yz] = -q; });
                } else {
                    // to the tail's block, padding included
                    u64* out = A.ws + A.tail_rhs + 4 * C.x4 * ((v.y0 / 2 + Y) + C.n[1] * (v.z0 / 2 + Z));
                    restrict_pair(v, x, Y, Z, [&](int X, float q) { put1(out + X, -q, epoch); });
                    if (x == v.x4 - 1)
                        for (int X = C.n[0]; X < 4 * C.x4; ++X) put1(out + X, 0.f, epoch);
                }
            }
            __syncthreads();
        }
        if (A.count > A.dist) {
            // the correction's rows under this tile, one more on every side
            const View g = view(A.dist);
            const int all = g.plane * (g.tz + 2);
            for (int at = tid; at < all; at += kThreads * kRimItems) {
                int from[kRimItems], dst[kRimItems];
#pragma unroll
                for (int u = 0; u < kRimItems; ++u) {
                    const int s = at + u * kThreads;
                    int x, y, z;
                    g.item(s, x, y, z);
                    const int gy = g.y0 + y, gz = g.z0 + z;
                    const bool in = s < all && gy >= 0 && gz >= 0 && gy < g.n[1] && gz < g.n[2];
                    from[u] = in ? published(g, x, gy, gz) : -1;
                    dst[u] = s;
                }
                collect(A.ws + A.tail_p, from, g.P, dst, epoch, waits);
            }
            __syncthreads();
        }
        for (int k = low - 1; k >= 0; --k) {
            View v = view(k);
            prolong(v, view(k + 1));
            smooth(v, k, false, A.post);
        }
    }
    {
        const View v = view(0);
        const int slots = v.flat * v.tz;
        for (int s = tid; s < slots; s += kThreads) {
            int x, y, z;
            v.slot(s, x, y, z);
            const float4 p = v.P[v.at(x, y, z)];
            float* o = A.p_out + 4 * x + (int64_t)v.n[0] * ((v.y0 + y) + (int64_t)v.n[1] * (v.z0 + z));
            const int left = v.n[0] - 4 * x;
            if (A.vec) {
                *reinterpret_cast<float4*>(o) = p;
            } else {
                o[0] = p.x;
                if (left > 1) o[1] = p.y;
                if (left > 2) o[2] = p.z;
                if (left > 3) o[3] = p.w;
            }
        }
    }
}

// RAGGED: some level's rows are no multiple of four (any, with a mask: its classes tell).
template <bool MASK, bool ONE, bool RAGGED>
__global__ void __launch_bounds__(kThreads, 1) resident_kernel(const __grid_constant__ Params A) {
    extern __shared__ float4 smem[];
    __shared__ float2 kd[kLevels][28];
    __shared__ int dead;
    const int tid = threadIdx.x;
    const bool tail = (int)blockIdx.x == A.gy * A.gz || A.dist == 0;
    if (tid == 0) dead = 0;
    const int clear = tail ? A.tail_f4 : A.tile_f4;
    for (int i = tid; i < clear; i += kThreads) smem[i] = zero4();
    for (int i = tid; i < 32 * A.count; i += kThreads) {
        const int k = i >> 5;
        fill_table(kd[k], i & 31, k < A.dist ? A.lv[k].w : A.tv[k].w, A.omega);
    }
    __syncthreads();
    const unsigned base = A.dist ? A.epochs[blockIdx.x] : 0u;
    const Waits waits = {&dead, A.timeouts, A.alarm};
    if (tail) run_tail<RAGGED>(A, smem, kd, waits, base);
    else run_tile<MASK, ONE, RAGGED>(A, smem, kd, waits, base);
    __syncthreads();
    if (tid == 0 && A.dist) A.epochs[blockIdx.x] = base + A.epochs_used;
}

}  // namespace resident
}  // namespace ffx
