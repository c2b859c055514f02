// Host side of the resident collider multigrid (ffx_graph_resident.cuh): plans
// (which levels, which tiles), descriptors and launches.
#include "ffx_graph_resident.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>

#include "ffx_graph_plan.cuh"

namespace ffx {
namespace gres {
namespace {

int up4(int v) { return (v + 3) & ~3; }
int x4_of(const FfxGraphLevel& g) { return up4(g.nx) / 4; }
int64_t slots_of(const FfxGraphLevel& g) { return (int64_t)x4_of(g) * g.ny * g.nz; }

// float4 of a level with edge records on y x z rows: two pressures with a rim,
// right-hand side, three records and the diagonal's reciprocal.
int edge_f4(int x4, int y, int z) {
    return x4 * (2 * (y + 2) * (z + 2) + 3 * y * z + (y + 1) * z + y * (z + 1));
}

int tail_f4(const Spec& S, int first) {
    int f4 = 0;
    for (int k = first; k < S.count; ++k) {
        const FfxGraphLevel& g = S.level[k];
        f4 += edge_f4(x4_of(g), g.ny, g.nz);
    }
    return f4;
}

// two: level 0 has two copies of its pressure. A plane of an in-place sweep costs
// a block 1100 cycles, a barrier and its latency; a sweep from one copy to the
// other costs the arithmetic. So two wherever they fit.
int tile_f4(const Spec& S, int dist, int ty, int tz, bool two) {
    int f4 = 0;
    for (int k = 0; k <= dist && k < S.count; ++k) {
        const int x4 = x4_of(S.level[k]), y = ty >> k, z = tz >> k, rim = x4 * (y + 2) * (z + 2);
        if (k == dist) f4 += rim;
        else if (k == 0 && S.whole) f4 += (two ? 2 : 1) * rim + x4 * y * z + up4(rim) / 4;
        else f4 += edge_f4(x4, y, z);
    }
    return f4;
}

}  // namespace

bool candidates(const Spec& S, int sms, std::vector<Candidate>& out, int& dist) {
    out.clear();
    if (S.count < 1 || S.count > kLevels || (S.whole && S.count < 2)) return false;
    // the tail: levels that one block holds, never level 0
    dist = S.count;
    while (dist > 1) {
        const FfxGraphLevel& g = S.level[dist - 1];
        if (slots_of(g) > resident::kTailSlots || x4_of(g) * g.ny > kThreads ||
            16 * tail_f4(S, dist - 1) > resident::kSmem)
            break;
        --dist;
    }
    const bool tail = dist < S.count;
    if (S.inverse && !tail) return false;
    const FfxGraphLevel& g = S.level[0];
    const int align = 1 << (tail ? dist : dist - 1), cap = sms - (tail ? 1 : 0), x4 = x4_of(g);
    for (int ty = align; ty < g.ny + align; ty += align)
        for (int tz = align; tz < g.nz + align; tz += align) {
            const int tiles = ((g.ny + ty - 1) / ty) * ((g.nz + tz - 1) / tz);
            if (tiles > cap || tiles > kMaxTiles || x4 * ty > kThreads ||
                x4 * (2 * (ty + tz) + 4) > kThreads * kRimItems || x4 * (ty + 2) >= 4096 ||
                16 * tile_f4(S, dist, ty, tz, false) > resident::kSmem)
                continue;
            // a sweep's work per block: its cells, and its rim's words and addresses. Of all
            // tiles that fit, the least cost was the fastest at 32^3, 64 x 32 x 64, 48 x 96 x
            // 48, 64^3, 96 x 80 x 112 and 96 x 96 x 160 (two V(4,4) cycles: 85 us at 32^3 with
            // the chosen tile, 222 with the worst; 352 and 516 at 96 x 80 x 112)
            out.push_back(Candidate{ty, tz, tiles + (tail ? 1 : 0), 1.0 * x4 * ty * tz + 0.6 * x4 * (2 * (ty + tz) + 4)});
        }
    return !out.empty();
}

bool plan_blocks(const Spec* specs, int count, int sms, std::vector<Candidate>& chosen, std::vector<int>& dist) {
    std::vector<std::vector<Candidate>> all(count);
    chosen.assign(count, Candidate{});
    dist.assign(count, 0);
    int used = 0;
    for (int d = 0; d < count; ++d) {
        if (!candidates(specs[d], sms, all[d], dist[d])) return false;
        // the fewest blocks that hold it, of those the least work
        std::sort(all[d].begin(), all[d].end(), [](const Candidate& a, const Candidate& b) {
            return a.blocks != b.blocks ? a.blocks < b.blocks : a.cost < b.cost;
        });
        chosen[d] = all[d][0];
        used += chosen[d].blocks;
    }
    if (used > sms) return false;
    // then blocks to whichever domain takes longest, while there are any
    for (;;) {
        int worst = 0;
        for (int d = 1; d < count; ++d)
            if (chosen[d].cost > chosen[worst].cost) worst = d;
        const Candidate* next = nullptr;
        for (const Candidate& c : all[worst])
            if (c.cost < chosen[worst].cost && used - chosen[worst].blocks + c.blocks <= sms &&
                (!next || c.blocks < next->blocks || (c.blocks == next->blocks && c.cost < next->cost)))
                next = &c;
        if (!next) return true;
        used += next->blocks - chosen[worst].blocks;
        chosen[worst] = *next;
    }
}

int64_t words_of(const Spec& S, int dist) {
    int64_t words = 2 * kMaxTiles + 2 + kHeader;
    for (int k = 0; k < dist; ++k) words += 2 * 4 * slots_of(S.level[k]);
    if (dist < S.count) words += 2 * 4 * slots_of(S.level[dist]);
    return words;
}

int fill(const Spec& S, int dist, const Candidate& c, int first_block, u64* ws, Domain& D) {
    const FfxGraphLevel& g = S.level[0];
    memset(&D, 0, sizeof D);
    D.count = S.count;
    D.dist = dist;
    D.gy = (g.ny + c.ty - 1) / c.ty;
    D.gz = (g.nz + c.tz - 1) / c.tz;
    D.first_block = first_block;
    D.blocks = D.gy * D.gz + (dist < S.count ? 1 : 0);
    D.pre0 = S.pre0; D.post0 = S.post0; D.pre = S.pre; D.post = S.post; D.last = S.last;
    D.omega = S.omega;
    D.whole = S.whole;
    D.links = g.links;
    D.inverse = S.inverse;
    D.ws = ws;
    // header: two exchange numbers per block, then the timeout count
    D.epochs = reinterpret_cast<unsigned*>(ws);
    D.timeouts = D.epochs + 2 * kHeader - 1;
    int64_t word = kHeader;
    D.maxima = word;
    word += 2 * kMaxTiles;
    D.control = word;
    word += 2;
    auto level = [&](int k, int ty, int tz) {
        Level L = {};
        const FfxGraphLevel& v = S.level[k];
        L.base.n[0] = v.nx; L.base.n[1] = v.ny; L.base.n[2] = v.nz;
        for (int a = 0; a < 3; ++a) L.base.w[a] = v.w[a];
        L.base.x4 = x4_of(v);
        L.base.ty = ty;
        L.base.tz = tz;
        L.edges = reinterpret_cast<const float4*>(v.edges);
        L.cs = v.coarse_scale != 0.f ? v.coarse_scale : 1.f;
        return L;
    };
    auto place_edges = [](Level& L, int y, int z, int& off) {
        const int x4 = L.base.x4;
        L.base.q = off;
        off += x4 * (y + 2) * (z + 2);
        L.base.r = off;
        off += x4 * y * z;
        L.ex = off;
        off += x4 * y * z;
        L.ey = off;
        off += x4 * (y + 1) * z;
        L.ez = off;
        off += x4 * y * (z + 1);
        L.rc = off;
        off += x4 * y * z;
    };
    const bool two = 16 * tile_f4(S, dist, c.ty, c.tz, true) <= resident::kSmem;
    int off = 0;
    for (int k = 0; k <= dist && k < S.count; ++k) {
        const int y = c.ty >> k, z = c.tz >> k;
        Level L = level(k, y, z);
        const int rim = L.base.x4 * (y + 2) * (z + 2);
        L.base.p = L.base.q = off;
        off += rim;
        if (k < dist) {
            D.exchanges += k == S.count - 1 ? S.last : (k == 0 ? S.pre0 + S.post0 : S.pre + S.post);
            L.base.ll = word;
            word += 2 * 4 * slots_of(S.level[k]);
            if (k == 0 && S.whole) {
                if (two) {
                    L.base.q = off;
                    off += rim;
                }
                L.base.r = off;
                off += L.base.x4 * y * z;
                D.link_off = off;
                off += up4(rim) / 4;
            } else {
                place_edges(L, y, z, off);
            }
        }
        D.lv[k] = L;
    }
    D.tile_f4 = off;
    off = 0;
    if (dist < S.count) {
        D.tail_rhs = word;
        word += 4 * slots_of(S.level[dist]);
        D.tail_p = word;
        word += 4 * slots_of(S.level[dist]);
        for (int k = dist; k < S.count; ++k) {
            Level L = level(k, S.level[k].ny, S.level[k].nz);
            L.base.p = off;
            off += L.base.x4 * (L.base.ty + 2) * (L.base.tz + 2);
            place_edges(L, L.base.ty, L.base.tz, off);
            D.tv[k] = L;
        }
    }
    D.tail_f4 = off;
    D.vec = g.nx % 4 == 0 && (!S.whole || (uintptr_t)g.links % 4 == 0);
    return 16 * std::max(D.tile_f4, D.tail_f4);
}

int launch(bool links, const Domain* domains, int count, int blocks, int smem, const Call& A, cudaStream_t st) {
    static std::atomic<uint64_t> ready{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetDevice");
    if (!(ready.load(std::memory_order_acquire) >> (dev & 63) & 1)) {
        e = cudaFuncSetAttribute(graph_resident_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, resident::kSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(graph_resident_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, resident::kSmem);
        if (e != cudaSuccess) return cuda_status(e, "graph_resident_kernel");
        ready.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_release);
    }
    FFX_REQUIRE(blocks <= resident_sms(), "graph_resident_kernel: planned for %d SMs, the device has %d", blocks,
                resident_sms());
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = blocks > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, links ? graph_resident_kernel<true> : graph_resident_kernel<false>, domains, count, A);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(FFX_ERR_LAUNCH, "graph_resident_kernel: %s", cudaGetErrorString(e));
    }
    return launch_status("graph_resident_kernel");
}

}  // namespace gres
}  // namespace ffx

using namespace ffx;

namespace {

constexpr int64_t kDomainBytes = (sizeof(gres::Domain) + 255) / 256 * 256;

// The plan's levels as a Spec; false with a message when they are not a hierarchy.
int spec_of(const FfxGraphPlan* P, gres::Spec& S) {
    FFX_REQUIRE(P && P->count >= 1 && P->count <= FFX_GRAPH_PLAN_LEVELS && P->count <= gres::kLevels && P->pre0 >= 1 &&
                P->post0 >= 1 && P->pre >= 1 && P->post >= 1 && P->last_sweeps >= 1 && P->omega > 0.f,
                "ffx_graph_plan: invalid arguments");
    S = gres::Spec{};
    S.count = P->count;
    S.whole = P->level[0].edges == nullptr;
    S.inverse = P->inverse;
    S.pre0 = P->pre0; S.post0 = P->post0; S.pre = P->pre; S.post = P->post; S.last = P->last_sweeps;
    S.omega = P->omega;
    for (int k = 0; k < P->count; ++k) {
        const FfxGraphLevel& g = P->level[k];
        FFX_REQUIRE(g.nx >= 1 && g.ny >= 1 && g.nz >= 1 && g.nx <= 4096 && g.ny <= 4096 && g.nz <= 4096 &&
                    (k > 0 || !S.whole ? g.edges != nullptr && (uintptr_t)g.edges % 16 == 0 : g.links != nullptr),
                    "ffx_graph_plan: level %d is incomplete", k);
        if (k > 0) {
            const FfxGraphLevel& up = P->level[k - 1];
            FFX_REQUIRE(up.nx == 2 * g.nx && up.ny == 2 * g.ny && up.nz == 2 * g.nz,
                        "ffx_graph_plan: level %d does not halve", k);
        }
        S.level[k] = g;
    }
    return FFX_OK;
}

}  // namespace

extern "C" {

int ffx_graph_plan(FfxGraphPlan* P) {
    gres::Spec S;
    if (int e = spec_of(P, S)) return e;
    P->blocks = P->shared_bytes = 0;
    P->workspace_bytes = 0;
    std::vector<gres::Candidate> c;
    std::vector<int> dist;
    P->sms = P->sms > 0 ? std::min(P->sms, resident_sms()) : resident_sms();
    if (!gres::plan_blocks(&S, 1, P->sms, c, dist)) return FFX_OK;      // it does not fit: blocks stays 0
    P->blocks = c[0].blocks;
    P->tile[0] = c[0].ty;
    P->tile[1] = c[0].tz;
    P->tail = dist[0];
    P->workspace_bytes = kDomainBytes + 8 * gres::words_of(S, dist[0]);
    return FFX_OK;
}

int ffx_graph_plan_upload(FfxGraphPlan* P, void* stream) {
    gres::Spec S;
    if (int e = spec_of(P, S)) return e;
    FFX_REQUIRE(P->blocks > 0 && P->workspace && (uintptr_t)P->workspace % 256 == 0 && P->tail >= 1 &&
                P->tail <= P->count && P->tile[0] >= 1 && P->tile[1] >= 1, "ffx_graph_plan_upload: not a plan that fits");
    gres::Domain D;
    const gres::Candidate c = {P->tile[0], P->tile[1], P->blocks, 0.0};
    char* base = reinterpret_cast<char*>(P->workspace);
    P->shared_bytes = gres::fill(S, P->tail, c, 0, reinterpret_cast<gres::u64*>(base + kDomainBytes), D);
    D.alarm = P->alarm;
    FFX_REQUIRE(D.blocks == P->blocks && P->shared_bytes <= resident::kSmem, "ffx_graph_plan_upload: not a plan that fits");
    cudaStream_t st = as_stream(stream);
    cudaError_t e = cudaMemcpyAsync(base, &D, sizeof D, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return cuda_status(e, "ffx_graph_plan_upload");
}

int ffx_graph_solve(const FfxGraphPlan* P, float* p, const float* rhs, int32_t cycles, int32_t from_zero, double tol,
                    int32_t max_cycles, int32_t* counters, void* stream) {
    FFX_REQUIRE(P && P->blocks > 0 && P->workspace && P->shared_bytes > 0 && p && rhs && p != rhs && cycles >= 0,
                "ffx_graph_solve: invalid arguments");
    const bool whole = P->level[0].edges == nullptr;
    FFX_REQUIRE(cycles > 0 || (whole && tol > 0.0 && max_cycles >= 0 && counters),
                "ffx_graph_solve: a solve to a tolerance needs one, a cycle limit and counters");
    FFX_REQUIRE(whole || (cycles == 1 && from_zero), "ffx_graph_solve: a coarse part is one cycle from zero");
    gres::Call A = {};
    A.p = p;
    A.rhs = rhs;
    A.cycles = cycles;
    A.from_zero = from_zero;
    A.tol = tol;
    A.max_cycles = max_cycles;
    A.counters = counters;
    A.aligned = ((uintptr_t)p | (uintptr_t)rhs) % 16 == 0;
    return gres::launch(whole, reinterpret_cast<const gres::Domain*>(P->workspace), 1, P->blocks, P->shared_bytes, A,
                        as_stream(stream));
}

int ffx_graph_plan_reset(const FfxGraphPlan* P, void* stream) {
    FFX_REQUIRE(P, "ffx_graph_plan_reset: invalid arguments");
    if (!P->workspace || P->blocks == 0) return FFX_OK;
    return cuda_status(cudaMemsetAsync(reinterpret_cast<char*>(P->workspace) + kDomainBytes, 0,
                                       (size_t)(P->workspace_bytes - kDomainBytes), as_stream(stream)),
                       "ffx_graph_plan_reset");
}

int ffx_graph_plan_timeouts(const FfxGraphPlan* P, int32_t* count, void* stream) {
    FFX_REQUIRE(P && count, "ffx_graph_plan_timeouts: invalid arguments");
    *count = 0;
    if (!P->workspace || P->blocks == 0) return FFX_OK;
    unsigned v = 0;
    cudaStream_t st = as_stream(stream);
    const unsigned* at = reinterpret_cast<const unsigned*>(reinterpret_cast<const char*>(P->workspace) + kDomainBytes) +
                         2 * gres::kHeader - 1;
    cudaError_t e = cudaMemcpyAsync(&v, at, sizeof v, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_status(e, "ffx_graph_plan_timeouts");
    *count = (int32_t)v;
    return FFX_OK;
}

}  // extern "C"
