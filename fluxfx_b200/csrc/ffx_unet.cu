// Learned pressure warm start: BF16 implicit-GEMM 3D convolutions (forward,
// data gradient, weight gradient), ReLU backward, Adam, and the loss.
//
// Activations are NDHWC bfloat16 (a voxel's channels are contiguous); a tensor
// is addressed through a view (pointer, elements per voxel, first channel), so
// the decoder's concatenation of the upsampled path and the skip connection is
// one buffer that both producers write into and every consumer reads a channel
// range of, without copies.
//
// Forward convolution as a GEMM: rows = output voxels, columns = output
// channels, reduction k = (tap, input channel), A gathered from the input with
// zero padding (implicit im2col), B = weights [k][cout]. Tiles of 128 x 64 x 16
// per block of four warps, a three-stage cp.async pipeline (zero-fill for
// padding and ragged edges), and BF16 tensor-core MMAs (m16n8k16, FP32
// accumulation, fragments via ldmatrix). The transposed 2^3 stride-2
// convolution (decoder up-sampling, and the data gradient of the stride-2
// down-sampling) maps each output voxel 2q + j to tap j of input voxel q: one
// GEMM per parity class j (blockIdx.z). Weight gradients reduce over voxels:
// dW[k][n] = sum_m A[m][k] G[m][n], split over voxel chunks with FP32 atomics.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "ffx_host.cuh"

namespace ffx {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kBM = 128, kBN = 64, kGemmThreads = 128;
constexpr int kFwdStages = 5;   // ring of the forward GEMM: 42 KB at BN = 64
constexpr int kAStride = 24;    // bf16 per A row in shared memory (16 + 8 pad: 48 B, conflict-free ldmatrix)
constexpr int kBStride = 72;    // bf16 per B row (64 + 8 pad: 144 B)

struct View {
    const bf16* p;
    int pitch, offset;
};

struct Conv {
    int batch, id, ih, iw, od, oh, ow;
    int c1, c2, cin, cout, ks, stride, pad, transposed;
    int taps, units_per_tap, k_units;   // reduction in units of 8 channels
    long long rows;                      // GEMM rows: output voxels, or input voxels per parity class
    View in1, in2;
    const bf16* w;
    const float* bias;
    int relu, accumulate;
    bf16* out;
    int out_pitch, out_offset;
    float* out_f32;
    int out_f32_pitch;
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int size = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(size));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(unsigned r[4], const void* smem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned r[4], const void* smem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x2_trans(unsigned r[2], const void* smem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Position of GEMM row m: the output voxel (convolution) or the input voxel q
// of a parity class (transposed).
struct RowPos {
    int b, z, y, x;
};
__device__ __forceinline__ RowPos decode(long long m, int d, int h, int w) {
    RowPos r;
    r.x = (int)(m % w);
    long long t = m / w;
    r.y = (int)(t % h);
    t /= h;
    r.z = (int)(t % d);
    r.b = (int)(t / d);
    return r;
}

// Address of unit u (8 channels) of GEMM row `pos` in the gathered input, or
// nullptr where the tap falls outside the input (zero padding).
__device__ __forceinline__ const bf16* gather(const Conv& a, const RowPos& pos, int u) {
    const int tap = u / a.units_per_tap;
    const int c = (u - tap * a.units_per_tap) * 8;
    long long vox;
    if (a.transposed) {
        vox = (((long long)pos.b * a.id + pos.z) * a.ih + pos.y) * a.iw + pos.x;
    } else {
        const int ks = a.ks;
        const int dz = tap / (ks * ks), dy = (tap / ks) % ks, dx = tap % ks;
        const int zz = pos.z * a.stride - a.pad + dz, yy = pos.y * a.stride - a.pad + dy,
                  xx = pos.x * a.stride - a.pad + dx;
        if ((unsigned)zz >= (unsigned)a.id || (unsigned)yy >= (unsigned)a.ih || (unsigned)xx >= (unsigned)a.iw)
            return nullptr;
        vox = (((long long)pos.b * a.id + zz) * a.ih + yy) * a.iw + xx;
    }
    if (c < a.c1) return a.in1.p + vox * a.in1.pitch + a.in1.offset + c;
    return a.in2.p + vox * a.in2.pitch + a.in2.offset + (c - a.c1);
}

// The units (8 channels each) of GEMM row `pos` one after another, tap by tap:
// the address of the next, or nullptr where its tap falls outside the input
// (zero padding). The tap's voxel is found once per tap.
struct UnitWalk {
    RowPos pos;
    int tap, c;
    long long vox;      // < 0: outside
    __device__ __forceinline__ UnitWalk(const Conv& a, RowPos p) : pos(p), tap(0), c(0) { place(a); }
    __device__ __forceinline__ void place(const Conv& a) {
        if (a.transposed) {
            vox = (((long long)pos.b * a.id + pos.z) * a.ih + pos.y) * a.iw + pos.x;
            return;
        }
        const int ks = a.ks, dz = tap / (ks * ks), r = tap - dz * ks * ks, dy = r / ks, dx = r - dy * ks;
        const int zz = pos.z * a.stride - a.pad + dz, yy = pos.y * a.stride - a.pad + dy,
                  xx = pos.x * a.stride - a.pad + dx;
        const bool in = (unsigned)zz < (unsigned)a.id && (unsigned)yy < (unsigned)a.ih && (unsigned)xx < (unsigned)a.iw;
        vox = in ? (((long long)pos.b * a.id + zz) * a.ih + yy) * a.iw + xx : -1;
    }
    __device__ __forceinline__ const bf16* next(const Conv& a) {
        const bf16* at = vox < 0 ? nullptr
                         : c < a.c1 ? a.in1.p + vox * a.in1.pitch + a.in1.offset + c
                                    : a.in2.p + vox * a.in2.pitch + a.in2.offset + (c - a.c1);
        c += 8;
        if (c == 8 * a.units_per_tap) {
            c = 0;
            ++tap;
            place(a);
        }
        return at;
    }
};

// Output voxel index of GEMM row m (class j for the transposed form).
__device__ __forceinline__ long long out_voxel(const Conv& a, long long m, int cls) {
    if (!a.transposed) return m;
    const RowPos q = decode(m, a.id, a.ih, a.iw);
    const int z = 2 * q.z + (cls >> 2), y = 2 * q.y + ((cls >> 1) & 1), x = 2 * q.x + (cls & 1);
    return (((long long)q.b * a.od + z) * a.oh + y) * a.ow + x;
}

// ------------------------------------------------------------ forward GEMM
// BN output channels per block (16, 32 or 64, chosen from cout so that narrow
// layers do not multiply padded channels, halved while the grid would leave SMs
// without a block).
//
// Bound by the latency of a k-step: the layers that come here have a few hundred
// to a few thousand rows and 8 to 64 steps. The rows' addresses are walked tap by
// tap instead of divided out per unit, and four steps are in flight. With two
// steps in flight and 64 channels a block whatever the grid, the five layers of a
// guess at 128 x 96 x 64 took 118 us, now 79.
template <int BN>
__global__ void __launch_bounds__(kGemmThreads) conv_fwd_kernel(const __grid_constant__ Conv a) {
    constexpr int BS = BN + 8;   // bf16 per B row in shared memory (8 pad: conflict-free ldmatrix)
    __shared__ __align__(128) bf16 sA[kFwdStages][kBM * kAStride];
    __shared__ __align__(128) bf16 sB[kFwdStages][16 * BS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long m0 = (long long)blockIdx.x * kBM;
    const int n0 = blockIdx.y * BN;
    const int cls = blockIdx.z;
    const bf16* W = a.w + (a.transposed ? (size_t)cls * a.cin * a.cout : 0);
    const long long my_row = m0 + tid;
    const bool row_ok = my_row < a.rows;
    const RowPos pos = row_ok ? (a.transposed ? decode(my_row, a.id, a.ih, a.iw) : decode(my_row, a.od, a.oh, a.ow))
                              : RowPos{0, 0, 0, 0};
    const int k_elems = a.k_units * 8;
    const int nk = (a.k_units + 1) / 2;

    UnitWalk walk(a, pos);
    auto load = [&](int stage, int kstep) {      // steps in order
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int u = kstep * 2 + h;
            const bf16* src = (row_ok && u < a.k_units) ? walk.next(a) : nullptr;
            cp_async16(&sA[stage][tid * kAStride + h * 8], src ? src : a.in1.p, src != nullptr);
        }
        if (tid < 2 * BN) {   // 16 rows x BN / 8 units of 8 channels
            const int kr = tid / (BN / 8), nu = (tid % (BN / 8)) * 8;
            const int k = kstep * 16 + kr, n = n0 + nu;
            const bool ok = k < k_elems && n < a.cout;
            cp_async16(&sB[stage][kr * BS + nu], ok ? W + (size_t)k * a.cout + n : W, ok);
        }
    };

    float acc[2][BN / 8][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < BN / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

#pragma unroll
    for (int s = 0; s < kFwdStages - 1; ++s) {
        if (s < nk) load(s, s);
        cp_async_commit();
    }
    for (int ks = 0; ks < nk; ++ks) {
        cp_async_wait<kFwdStages - 2>();
        __syncthreads();
        const int pf = ks + kFwdStages - 1;
        if (pf < nk) load(pf % kFwdStages, pf);
        cp_async_commit();
        const int st = ks % kFwdStages;
        unsigned af[2][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
            ldmatrix_x4(af[mt], &sA[st][(warp * 32 + mt * 16 + (lane & 15)) * kAStride + (lane >> 4) * 8]);
#pragma unroll
        for (int np = 0; np < BN / 16; ++np) {
            unsigned bf[4];
            ldmatrix_x4_trans(bf, &sB[st][((lane & 7) + ((lane >> 3) & 1) * 8) * BS + np * 16 + (lane >> 4) * 8]);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                mma_bf16(acc[mt][2 * np], af[mt], bf[0], bf[1]);
                mma_bf16(acc[mt][2 * np + 1], af[mt], bf[2], bf[3]);
            }
        }
    }
    cp_async_wait<0>();

    // epilogue: bias, ReLU, optional accumulation, BF16 and/or FP32 stores
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const long long m = m0 + warp * 32 + mt * 16 + (lane >> 2) + half * 8;
            if (m >= a.rows) continue;
            const long long vox = out_voxel(a, m, cls);
#pragma unroll
            for (int nt = 0; nt < BN / 8; ++nt) {
                const int n = n0 + nt * 8 + (lane & 3) * 2;
                if (n >= a.cout) continue;
                float v0 = acc[mt][nt][half * 2], v1 = acc[mt][nt][half * 2 + 1];
                if (a.bias) {
                    v0 += a.bias[n];
                    v1 += a.bias[n + 1];
                }
                if (a.relu) {
                    v0 = fmaxf(v0, 0.f);
                    v1 = fmaxf(v1, 0.f);
                }
                if (a.out) {
                    __nv_bfloat162* o =
                        reinterpret_cast<__nv_bfloat162*>(a.out + vox * a.out_pitch + a.out_offset + n);
                    if (a.accumulate) {
                        const float2 prev = __bfloat1622float2(*o);
                        v0 += prev.x;
                        v1 += prev.y;
                    }
                    *o = __floats2bfloat162_rn(v0, v1);
                }
                if (a.out_f32) {
                    float* o = a.out_f32 + vox * a.out_f32_pitch + n;
                    o[0] = v0;
                    o[1] = v1;
                }
            }
        }
}

// ------------------------------------------------- forward GEMM, tcgen05
// The same implicit GEMM on the 5th-generation tensor cores: one elected
// thread issues tcgen05.mma (kind::f16, M = 128, N = BN, K = 16, BF16 in, FP32
// accumulated in tensor memory) from shared-memory operand descriptors, the
// accumulator tile lives in TMEM for the whole reduction, and the epilogue
// reads it back with tcgen05.ld (one row per thread). Operands are staged by
// cp.async in the canonical no-swizzle core-matrix layouts: A (voxels x k)
// K-major, 8 rows x 16 B per core matrix; B (k x channels) MN-major straight
// from the [k][cout] weights, 8 k-rows x 8 channels per core matrix. A stage
// holds K = 32 (two MMAs); a single mbarrier tracks MMA completion through
// tcgen05.commit. Every wait is bounded: on timeout the kernel records it in
// g_conv_timeouts, stops issuing, and still frees its TMEM.
__device__ int g_conv_timeouts;

constexpr int kTcStages = 3;                     // ring of operand stages (36 KB at BN = 64: six blocks per SM)
constexpr int kTcStageK = 32;                    // two MMA k-steps of 16
constexpr int kTcSpin = 1 << 22;                 // bounded mbarrier polling

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (no swizzle): start, leading- and stride-
// dimension byte offsets (16-byte units), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;                      // version
    return d;                                    // base offset 0, layout type 0 (no swizzle)
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < kTcSpin; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

template <int BN>
constexpr int tc_smem_bytes() { return kTcStages * (2 * kBM * 16 * 2 + 2 * 16 * BN * 2); }

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) conv_fwd_tc_kernel(const __grid_constant__ Conv a) {
    static_assert(BN == 16 || BN == 32 || BN == 64, "BN");
    constexpr int kAStep = kBM * 16 * 2;             // bytes of A per MMA k-step (128 rows x 16 k)
    constexpr int kBStep = 16 * BN * 2;              // bytes of B per MMA k-step (16 k x BN)
    constexpr int kTmemCols = BN < 32 ? 32 : BN;
    extern __shared__ __align__(128) unsigned char tc_smem[];
    unsigned char (*sA)[2 * kAStep] = reinterpret_cast<unsigned char (*)[2 * kAStep]>(tc_smem);
    unsigned char (*sB)[2 * kBStep] =
        reinterpret_cast<unsigned char (*)[2 * kBStep]>(tc_smem + kTcStages * 2 * kAStep);
    __shared__ __align__(8) uint64_t mbar[kTcStages];   // one per stage: its MMAs completed
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long m0 = (long long)blockIdx.x * kBM;
    const int n0 = blockIdx.y * BN;
    const int cls = blockIdx.z;
    const bf16* W = a.w + (a.transposed ? (size_t)cls * a.cin * a.cout : 0);
    const long long my_row = m0 + tid;
    const bool row_ok = my_row < a.rows;
    const RowPos pos = row_ok ? (a.transposed ? decode(my_row, a.id, a.ih, a.iw) : decode(my_row, a.od, a.oh, a.ow))
                              : RowPos{0, 0, 0, 0};
    const int k_elems = a.k_units * 8;
    const int nk = (a.k_units + 3) / 4;              // stages of 4 units (K = 32)

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        abort_flag = 0;
        for (int st = 0; st < kTcStages; ++st)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[st])));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;

    // A: row `tid`, units u (8 channels) of the stage -> core (row/8, chunk)
    // B: k-row r (0..31) x channel chunk h (BN/8) -> MN-major core matrices
    auto load = [&](int stage, int kstep) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int u = kstep * 4 + c;
            const bf16* src = (row_ok && u < a.k_units) ? gather(a, pos, u) : nullptr;
            unsigned char* dst = sA[stage] + (c >> 1) * kAStep + (tid >> 3) * 256 + (c & 1) * 128 + (tid & 7) * 16;
            cp_async16(dst, src ? src : a.in1.p, src != nullptr);
        }
        constexpr int kBLoads = kTcStageK * (BN / 8);       // 16-byte chunks of B per stage
        for (int q = tid; q < kBLoads; q += kGemmThreads) {
            const int r = q / (BN / 8), h = q % (BN / 8);
            const int k = kstep * kTcStageK + r, n = n0 + h * 8;
            const bool ok = k < k_elems && n < a.cout;
            unsigned char* dst = sB[stage] + (r >> 4) * kBStep + h * 256 + ((r & 15) >> 3) * 128 + (r & 7) * 16;
            cp_async16(dst, ok ? W + (size_t)k * a.cout + n : W, ok);
        }
    };
    // kind::f16, D = F32, A = B = BF16, A K-major, B MN-major, N = BN, M = 128
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(kBM >> 4) << 24);

    constexpr int kAhead = 1;                         // stages loaded ahead of the MMAs
#pragma unroll
    for (int st = 0; st < kAhead; ++st) {
        if (st < nk) load(st, st);
        cp_async_commit();
    }
    bool ok = true;
    for (int ks = 0; ks < nk && ok; ++ks) {
        // the prefetch overwrites the stage whose MMAs were issued two iterations ago:
        // wait for that stage's use (kTcStages - kAhead MMA groups may stay in flight)
        const int pf = ks + kAhead;
        const int ps = pf % kTcStages;
        if (pf < nk && pf >= kTcStages) {
            if (!mbar_wait(smem_u32(&mbar[ps]), (uint32_t)(((pf - kTcStages) / kTcStages) & 1))) ok = false;
        }
        if (__syncthreads_or(!ok)) { ok = false; break; }
        if (pf < nk) load(ps, pf);
        cp_async_commit();
        cp_async_wait<kAhead>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int st = ks % kTcStages;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint64_t da = umma_desc(smem_u32(sA[st] + j * kAStep), 128, 256);
                const uint64_t db = umma_desc(smem_u32(sB[st] + j * kBStep), 128, 256);
                const uint32_t acc = (ks > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                    ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(&mbar[st])));
        }
    }
    cp_async_wait<0>();
    // the last commit covers every MMA issued (its stage's barrier, last use)
    const uint32_t last_bar = nk > 0 ? smem_u32(&mbar[(nk - 1) % kTcStages]) : 0u;
    const uint32_t last_parity = nk > 0 ? (uint32_t)(((nk - 1) / kTcStages) & 1) : 0u;
    if (ok && nk > 0 && !mbar_wait(last_bar, last_parity)) ok = false;
    if (!ok && tid == 0) atomicAdd(&g_conv_timeouts, 1);
    if (__syncthreads_or(!ok)) {
        // give MMAs possibly still in flight a bounded grace period before freeing TMEM
        if (nk > 0) mbar_wait(last_bar, last_parity);
    } else {
        asm volatile("tcgen05.fence::after_thread_sync;");
        // epilogue: warp w holds TMEM lanes 32w..32w+31 = rows of the tile
        const long long m = m0 + warp * 32 + lane;
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(taddr + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (m < a.rows) {
                const long long vox = out_voxel(a, m, cls);
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const int n = n0 + c0 + e;
                    if (n >= a.cout) continue;
                    float v0 = __uint_as_float(r[e]), v1 = __uint_as_float(r[e + 1]);
                    if (a.bias) {
                        v0 += a.bias[n];
                        v1 += a.bias[n + 1];
                    }
                    if (a.relu) {
                        v0 = fmaxf(v0, 0.f);
                        v1 = fmaxf(v1, 0.f);
                    }
                    if (a.out) {
                        __nv_bfloat162* o =
                            reinterpret_cast<__nv_bfloat162*>(a.out + vox * a.out_pitch + a.out_offset + n);
                        if (a.accumulate) {
                            const float2 prev = __bfloat1622float2(*o);
                            v0 += prev.x;
                            v1 += prev.y;
                        }
                        *o = __floats2bfloat162_rn(v0, v1);
                    }
                    if (a.out_f32) {
                        float* o = a.out_f32 + vox * a.out_f32_pitch + n;
                        o[0] = v0;
                        o[1] = v1;
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// ------------------------------- 3^3 convolution: TMA halo tile + tcgen05
// Stride-1, pad-1 3x3x3 layers without a gather. A work tile is an output
// block of 8 (x) x 16 (y) x bz (z) voxels and BN output channels; its input
// footprint, a 10 x 18 x (bz + 2) halo tile, comes in by one TMA tensor load
// per 8-channel plane (zero-filled outside the grid, which is the padding).
// In shared memory a plane is laid out [z][y][x][8 channels], 16 bytes per
// voxel, so for every tap (dz, dy, dx) the 128 rows (8 x-voxels x 16 y-rows)
// of the A operand are the canonical no-swizzle K-major core matrices of a
// shifted window: start = the tap's first voxel, 8-row groups one halo row
// (160 B) apart, the two 8-channel halves of K = 16 one plane apart. No data
// moves per tap: a K = 16 channel group costs 27 x bz MMAs (M = 128, N = BN)
// on one staged tile. The weights of a group, pre-packed into the MN-major
// core-matrix image of all 27 taps, arrive by one bulk copy with the planes.
//
// The kernel is persistent and warp-specialised: warp 4 (one thread) issues
// the loads of tile after tile into a ring of stages, warp 5 (one thread)
// issues the MMAs into one of two accumulator sets in tensor memory (bz x BN
// FP32 columns each), and warps 0-3 drain the other set (tcgen05.ld, bias,
// ReLU, accumulation, BF16 or FP32 stores), so a tile's loads, its MMAs and
// the previous tile's epilogue overlap. mbarriers hand over stages (full: the
// loads landed; empty: the stage's MMAs completed, by tcgen05.commit) and
// accumulator sets (acc_full by tcgen05.commit, acc_empty by the four
// epilogue warps). Every wait is bounded and also ends when another role has
// given up (a shared abort flag); the block then counts a timeout in
// g_conv_timeouts, lets its copies and MMAs drain (bounded), frees its tensor
// memory and returns.
constexpr int kTmX = 8, kTmY = 16;                   // output tile in x, y (M = 128)
constexpr int kTmHX = kTmX + 2, kTmHY = kTmY + 2;    // halo tile
constexpr int kTmThreads = 192;                      // warps 0-3 epilogue, 4 loads, 5 MMAs
constexpr int kTmMaxStages = 4;
constexpr int kTmSmemLimit = 200 * 1024;             // dynamic shared memory attribute of the kernels

struct TmaConv {
    CUtensorMap act;          // input: (channel, x, y, z, batch), box (8, 10, 18, bz + 2, 1)
    const bf16* wpack;        // packed weights: [cout / BN][groups][27][BN / 8][16][8]
    int batch, d, h, w;       // grid (input = output)
    int cin, cout, groups;    // groups = ceil(cin / 16) channel groups of K = 16
    int bz, tiles_x, tiles_y, tiles_z, nblocks;
    int tiles;                // work tiles: tiles_x * tiles_y * tiles_z * batch * nblocks
    int stages, planes;       // planes loaded per group (1 when cin == 8)
    uint32_t plane;           // bytes of one plane in shared memory (multiple of 128)
    uint32_t stage;           // bytes of one stage: 2 planes + 27 weight tiles
    uint32_t tx;              // bytes a stage's loads deliver
    uint32_t cols;            // tensor-memory columns allocated (2 accumulator sets)
    const float* bias;
    int relu, accumulate;
    bf16* out;
    int out_pitch, out_offset;
    float* out_f32;
    int out_f32_pitch;
};

struct TmTile {
    int nb, x0, y0, z0, b;
};
__device__ __forceinline__ TmTile tm_tile(const TmaConv& P, int t) {
    TmTile r;
    r.nb = t % P.nblocks;
    t /= P.nblocks;
    r.x0 = (t % P.tiles_x) * kTmX;
    t /= P.tiles_x;
    r.y0 = (t % P.tiles_y) * kTmY;
    t /= P.tiles_y;
    r.z0 = (t % P.tiles_z) * P.bz;
    r.b = t / P.tiles_z;
    return r;
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bounded wait that also gives up once another role has set `abort`.
__device__ __forceinline__ bool tm_wait(uint32_t bar, uint32_t parity, const volatile int* abort) {
    for (int i = 0; i < kTcSpin; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((i & 255) == 255 && *abort) return false;
    }
    return false;
}

// The halo planes of group g (channels 16g .. 16g + 15) and its packed weights.
template <int BN>
__device__ __forceinline__ void tm_issue_loads(const TmaConv& P, uint32_t st, uint32_t bar, int g, const TmTile& T) {
    mbar_expect_tx(bar, P.tx);
    const uint64_t map = reinterpret_cast<uint64_t>(&P.act);
    for (int h = 0; h < P.planes; ++h)
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
            "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
            ::"r"(st + h * P.plane), "l"(map), "r"(16 * g + 8 * h), "r"(T.x0 - 1), "r"(T.y0 - 1), "r"(T.z0 - 1),
              "r"(T.b), "r"(bar)
            : "memory");
    constexpr uint32_t kWBytes = 27u * 32u * BN;
    const bf16* src = P.wpack + ((size_t)T.nb * P.groups + g) * (kWBytes / 2);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(st + 2 * P.plane), "l"(src), "r"(kWBytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tm_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void tm_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// Epilogue of one tile: warp w reads tensor-memory lanes 32w .. 32w + 31 (the
// tile's rows m = 8 y + x) of accumulator set `acc`.
template <int BN>
__device__ __forceinline__ void tm_epilogue(const TmaConv& P, const TmTile& T, uint32_t acc, int warp, int lane) {
    const int m = warp * 32 + lane;
    const int x = T.x0 + (m & 7), y = T.y0 + (m >> 3);
    const uint32_t lane_addr = acc + ((uint32_t)(warp * 32) << 16);
    for (int j = 0; j < P.bz; ++j) {
        const int z = T.z0 + j;
        const bool in = x < P.w && y < P.h && z < P.d;
        const long long vox = (((long long)T.b * P.d + z) * P.h + y) * P.w + x;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(lane_addr + (uint32_t)(j * BN + c0)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (!in) continue;
            const int n = T.nb * BN + c0;
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                v[e] = __uint_as_float(r[e]);
                if (P.bias) v[e] += __ldg(P.bias + n + e);
                if (P.relu) v[e] = fmaxf(v[e], 0.f);
            }
            if (P.out) {
                uint4* o = reinterpret_cast<uint4*>(P.out + vox * P.out_pitch + P.out_offset + n);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (P.accumulate) {
                        const uint4 prev = o[q];
                        const __nv_bfloat162* pv = reinterpret_cast<const __nv_bfloat162*>(&prev);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = __bfloat1622float2(pv[e]);
                            v[8 * q + 2 * e] += f.x;
                            v[8 * q + 2 * e + 1] += f.y;
                        }
                    }
                    uint4 pk;
                    __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
                    for (int e = 0; e < 4; ++e) pp[e] = __floats2bfloat162_rn(v[8 * q + 2 * e], v[8 * q + 2 * e + 1]);
                    o[q] = pk;
                }
            }
            if (P.out_f32) {
                float* o = P.out_f32 + vox * P.out_f32_pitch + n;
#pragma unroll
                for (int e = 0; e < 16; ++e) o[e] = v[e];
            }
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(kTmThreads, 1) conv3_tma_kernel(const __grid_constant__ TmaConv P) {
    static_assert(BN == 16 || BN == 32 || BN == 64, "BN");
    extern __shared__ __align__(128) unsigned char tm_smem[];
    __shared__ __align__(8) uint64_t full[kTmMaxStages], empty[kTmMaxStages], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_word;
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (smem_u32(tm_smem) + 127u) & ~127u;
    const uint32_t acc_cols = (uint32_t)(P.bz * BN);
    const int S = P.stages;

    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(P.cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (P.planes == 1) {
        // cin == 8: the second channel half of K is zero in every stage
        for (int s = 0; s < S; ++s)
            for (uint32_t i = tid * 16; i < P.plane; i += kTmThreads * 16)
                asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(base + s * P.stage + P.plane + i),
                             "r"(0u)
                             : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (tid == 0) {
        abort_word = 0;
        for (int s = 0; s < S; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[s])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&empty[s])));
        }
        for (int a = 0; a < 2; ++a) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&acc_full[a])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(smem_u32(&acc_empty[a])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&drained)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base;

    if (warp == 4) {
        if (lane == 0) {
            // loads: tile after tile, group after group, into the stage ring
            int q = 0;
            for (int t = blockIdx.x; t < P.tiles && !*abort_flag; t += gridDim.x) {
                const TmTile T = tm_tile(P, t);
                for (int g = 0; g < P.groups; ++g, ++q) {
                    const int s = q % S;
                    if (q >= S && !tm_wait(smem_u32(&empty[s]), (uint32_t)(((q / S) - 1) & 1), abort_flag)) {
                        *abort_flag = 1;
                        break;
                    }
                    tm_issue_loads<BN>(P, base + s * P.stage, smem_u32(&full[s]), g, T);
                }
            }
            // the last load of every stage has landed before the block may exit
            for (int k = q > S ? q - S : 0; k < q; ++k) mbar_wait(smem_u32(&full[k % S]), (uint32_t)((k / S) & 1));
        }
    } else if (warp == 5) {
        if (lane == 0) {
            // MMAs: D[set][j] += A(tap, z slice j) x B(tap), 27 taps x bz slices per group
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(BN >> 3) << 17) |
                                   ((uint32_t)(128 >> 4) << 24);
            int q = 0, it = 0;
            for (int t = blockIdx.x; t < P.tiles && !*abort_flag; t += gridDim.x, ++it) {
                const int a = it & 1;
                if (it >= 2 && !tm_wait(smem_u32(&acc_empty[a]), (uint32_t)(((it >> 1) - 1) & 1), abort_flag)) {
                    *abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t d0 = tmem + (uint32_t)a * acc_cols;
                bool ok = true;
                for (int g = 0; g < P.groups; ++g, ++q) {
                    const int s = q % S;
                    if (!tm_wait(smem_u32(&full[s]), (uint32_t)((q / S) & 1), abort_flag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t st = base + s * P.stage;
                    const uint64_t da0 = umma_desc(st, P.plane, kTmHX * 16);
                    const uint64_t db0 = umma_desc(st + 2 * P.plane, 128, 256);
                    for (int j = 0; j < P.bz; ++j) {
                        // descriptor start addresses advance in 16-byte units (no carry: shared memory < 256 KB)
                        const uint64_t daj = da0 + (uint64_t)(j * kTmHY * kTmHX);
#pragma unroll
                        for (int tap = 0; tap < 27; ++tap) {
                            const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
                            tm_mma(d0 + (uint32_t)(j * BN), daj + (uint64_t)((dz * kTmHY + dy) * kTmHX + dx),
                                   db0 + (uint64_t)(tap * 2 * BN), idesc, (g > 0 || tap > 0) ? 1u : 0u);
                        }
                    }
                    tm_commit(smem_u32(&empty[s]));
                }
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                tm_commit(smem_u32(&acc_full[a]));
            }
            // every MMA issued has completed before tensor memory is freed
            tm_commit(smem_u32(&drained));
            mbar_wait(smem_u32(&drained), 0);
        }
    } else {
        // epilogue warps 0-3
        int it = 0;
        for (int t = blockIdx.x; t < P.tiles; t += gridDim.x, ++it) {
            const int a = it & 1;
            const bool ok = !*abort_flag && tm_wait(smem_u32(&acc_full[a]), (uint32_t)((it >> 1) & 1), abort_flag);
            if (!__all_sync(0xffffffffu, ok)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            tm_epilogue<BN>(P, tm_tile(P, t), tmem + (uint32_t)a * acc_cols, warp, lane);
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[a])) : "memory");
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (tid == 0 && abort_word) atomicAdd(&g_conv_timeouts, 1);
    if (warp == 5)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.cols));
}

// ------------------------------- narrow per-voxel convolutions (CUDA cores)
// 1^3 convolutions and transposed 2^3 stride-2 convolutions with 8 or 16
// output channels: each output voxel is one dot product of its input (parent)
// voxel's channels with the weights of its tap, and a tensor-core tile of 128
// voxels x 16 channels would be mostly idle. The input channels come in 16-byte
// groups, the weights as FP32 from shared memory; FP32 fused multiply-adds in
// channel order (two output channels to an instruction), then the bias, ReLU,
// accumulation and BF16 / FP32 stores of the implicit-GEMM epilogue.
constexpr int kDirectThreads = 256;
constexpr int kDirectMaxWeights = 12288;   // taps x cin x cout FP32 values (48 KB)

template <int COUT>
__device__ __forceinline__ void store_direct(const Conv& a, long long o, float (&acc)[COUT]) {
#pragma unroll
    for (int n = 0; n < COUT; ++n) {
        if (a.bias) acc[n] += __ldg(a.bias + n);
        if (a.relu) acc[n] = fmaxf(acc[n], 0.f);
    }
    if (a.out) {
        uint4* dst = reinterpret_cast<uint4*>(a.out + o * a.out_pitch + a.out_offset);
#pragma unroll
        for (int g = 0; g < COUT / 8; ++g) {
            if (a.accumulate) {
                const uint4 prev = dst[g];
                const __nv_bfloat162* pv = reinterpret_cast<const __nv_bfloat162*>(&prev);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(pv[e]);
                    acc[8 * g + 2 * e] += f.x;
                    acc[8 * g + 2 * e + 1] += f.y;
                }
            }
            uint4 pk;
            __nv_bfloat162* pp = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int e = 0; e < 4; ++e) pp[e] = __floats2bfloat162_rn(acc[8 * g + 2 * e], acc[8 * g + 2 * e + 1]);
            dst[g] = pk;
        }
    }
    if (a.out_f32) {
        float* dst = a.out_f32 + o * a.out_f32_pitch;
#pragma unroll
        for (int n = 0; n < COUT; ++n) dst[n] = acc[n];
    }
}

// acc[pair] += x w[pair] over the channels of one voxel for NT taps whose weights
// lie `step` floats apart.
template <int COUT, int NT>
__device__ __forceinline__ void dot_direct(const bf16* x, int cin, const float* W, int step, float (&out)[NT][COUT]) {
    unsigned long long acc[NT][COUT / 2];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int n = 0; n < COUT / 2; ++n) acc[t][n] = 0ull;
    for (int c8 = 0; c8 < cin; c8 += 8) {
        const uint4 raw = *reinterpret_cast<const uint4*>(x + c8);
        const unsigned h[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const unsigned bits = e & 1 ? h[e / 2] & 0xffff0000u : h[e / 2] << 16;      // BF16 -> FP32
            const unsigned long long f = (unsigned long long)bits << 32 | bits;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const ulonglong2* w = reinterpret_cast<const ulonglong2*>(W + t * step + (c8 + e) * COUT);
#pragma unroll
                for (int n = 0; n < COUT / 4; ++n) {
                    const ulonglong2 v = w[n];
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][2 * n]) : "l"(f), "l"(v.x));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][2 * n + 1]) : "l"(f), "l"(v.y));
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int n = 0; n < COUT / 2; ++n) {
            out[t][2 * n] = __uint_as_float((unsigned)acc[t][n]);
            out[t][2 * n + 1] = __uint_as_float((unsigned)(acc[t][n] >> 32));
        }
}

// 1^3: a thread per voxel.
template <int COUT>
__global__ void __launch_bounds__(kDirectThreads) conv_direct_kernel(const __grid_constant__ Conv a) {
    extern __shared__ __align__(16) float ws[];          // [cin][COUT]
    for (int i = threadIdx.x; i < a.cin * COUT; i += kDirectThreads) ws[i] = __bfloat162float(a.w[i]);
    __syncthreads();
    const long long o = (long long)blockIdx.x * kDirectThreads + threadIdx.x;
    if (o >= (long long)a.batch * a.od * a.oh * a.ow) return;
    float acc[1][COUT];
    dot_direct<COUT, 1>(a.in1.p + o * a.in1.pitch + a.in1.offset, a.cin, ws, 0, acc);
    store_direct<COUT>(a, o, acc[0]);
}

// Transposed: a thread per input voxel and (z, y) tap, the output voxels of both
// x taps; blockIdx.y is the (z, y) tap, so a block's threads read the same
// weights (one shared-memory word for a warp) and each input value serves two
// outputs. A thread per output voxel, its tap by its parity, was bound by those
// reads: 32 -> 16 channels at 128 x 96 x 64 59 us, now 40.
template <int COUT>
__global__ void __launch_bounds__(kDirectThreads) conv_up_kernel(const __grid_constant__ Conv a) {
    extern __shared__ __align__(16) float ws[];          // [2][cin][COUT]
    const int zy = blockIdx.y, step = a.cin * COUT;
    const bf16* w = a.w + (size_t)(2 * zy) * step;
    for (int i = threadIdx.x; i < 2 * step; i += kDirectThreads) ws[i] = __bfloat162float(w[i]);
    __syncthreads();
    const long long q = (long long)blockIdx.x * kDirectThreads + threadIdx.x;
    if (q >= a.rows) return;
    RowPos p;
    if (a.rows < (1ll << 31)) {
        const unsigned m = (unsigned)q, w1 = m / (unsigned)a.iw, h1 = w1 / (unsigned)a.ih, d1 = h1 / (unsigned)a.id;
        p = RowPos{(int)d1, (int)(h1 - d1 * a.id), (int)(w1 - h1 * a.ih), (int)(m - w1 * a.iw)};
    } else {
        p = decode(q, a.id, a.ih, a.iw);
    }
    float acc[2][COUT];
    dot_direct<COUT, 2>(a.in1.p + q * a.in1.pitch + a.in1.offset, a.cin, ws, step, acc);
    const long long o = (((long long)p.b * a.od + 2 * p.z + (zy >> 1)) * a.oh + 2 * p.y + (zy & 1)) * a.ow + 2 * p.x;
    store_direct<COUT>(a, o, acc[0]);
    store_direct<COUT>(a, o + 1, acc[1]);
}

// Packed weights of the TMA convolution: w[k = tap * cin + c][cout] ->
// [cout / BN][groups][27][BN / 8][16][8] (channels >= cin zero), the
// MN-major core-matrix image a stage copies into shared memory as it is.
__global__ void conv3_pack_kernel(const bf16* __restrict__ w, int cin, int cout, int bn, int groups,
                                  bf16* __restrict__ packed) {
    const long long n = (long long)(cout / bn) * groups * 27 * bn * 16;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int e = (int)(i % 8);
    long long r = i / 8;
    const int row = (int)(r % 16);
    r /= 16;
    const int j = (int)(r % (bn / 8));
    r /= bn / 8;
    const int tap = (int)(r % 27);
    r /= 27;
    const int g = (int)(r % groups);
    const int nb = (int)(r / groups);
    const int c = 16 * g + row, co = nb * bn + 8 * j + e;
    packed[i] = c < cin ? w[((long long)tap * cin + c) * cout + co] : __float2bfloat16(0.f);
}

// ------------------------------------------------------ weight gradient GEMM
// dW[k][n] += sum over the block's voxel chunk of A[m][k] G[m][n]; A^T
// fragments come from the [m][k] tile through ldmatrix.trans.
//
// What bounds it is the chain of MMAs into one accumulator: a chunk of 8192
// voxels is 512 of them in a row, whatever the tile. So the tile is narrow (64
// input by 16 or 32 output channels; a warp has 16 of the former and half of
// the latter), a step is one or two MMAs long, and a layer of one chunk still
// fills the SMs (64 -> 64 channels: 54 blocks). A stage is 64 voxels and three
// are in flight, so a step never waits for its gathers, and a gather costs
// a dozen instructions: its tap is fixed per thread and its voxel's position
// moves by carries, not divisions. Every accumulator sums its voxels in the
// order of the 16-voxel steps, so a chunk's sums do not depend on the tile.
// With a 128 x 64 tile, three 16-voxel stages and 64-bit divisions per gather a
// step took 1.4 us and a layer 730 us.
constexpr int kWgVox = 64, kWgK = 64, kWgStages = 4, kWgThreads = 256;

struct Wgrad {
    Conv a;
    const bf16* g;
    int g_pitch;
    float* dw;
    int chunk;
    int w, h, d;               // the GEMM row's grid (output voxels, or input voxels per parity class)
    int step_x, step_y, step_z;   // kWgVox rows further, in that grid
    int nt, kind;              // output channels of a block (16 or 32), WgKind
    int blocks_k, blocks_n, blocks_z;
};

// Position of a GEMM row that moves on by kWgVox rows at a time.
struct Walk {
    int x, y, z, b;
    __device__ __forceinline__ void start(const Wgrad& P, int m) {
        const int r = m / P.w, t = r / P.h;
        x = m - r * P.w;
        y = r - t * P.h;
        b = t / P.d;
        z = t - b * P.d;
    }
    __device__ __forceinline__ void advance(const Wgrad& P) {
        x += P.step_x;
        y += P.step_y;
        z += P.step_z;
        if (x >= P.w) { x -= P.w; ++y; }
        if (y >= P.h) { y -= P.h; ++z; }
        while (z >= P.d) { z -= P.d; ++b; }
    }
};

// How a GEMM row's input voxel follows from it: the same voxel shifted by the
// tap (padded stride-1 convolutions: the address moves on by a constant), the
// strided convolution's, or the row itself (transposed: the gradient's voxel
// is the strided one).
enum WgKind { kWgSame = 0, kWgStrided = 1, kWgTransposed = 2 };

template <int NT, int KIND>
__device__ __forceinline__ void wgrad_block(const Wgrad& P, int block_k, int block_n, int block_z) {
    constexpr int AS = kWgK + 8, GS = NT + 8;      // bf16 per shared row (8 pad: conflict-free ldmatrix)
    constexpr int NW = NT / 2;                     // output channels of a warp
    constexpr int kRows = kWgThreads / 8;          // voxels that the block's gathers cover at once
    extern __shared__ __align__(128) unsigned char wg_smem[];
    bf16* sA = reinterpret_cast<bf16*>(wg_smem);
    bf16* sG = sA + kWgStages * kWgVox * AS;
    const Conv& a = P.a;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k0 = block_k * kWgK, n0 = block_n * NT;
    const int cls = KIND == kWgTransposed ? block_z % 8 : 0;
    const int split = KIND == kWgTransposed ? block_z / 8 : block_z;
    const int mb = split * P.chunk;
    const int rows = (int)min(a.rows - mb, (long long)P.chunk);
    const int stages = (rows + kWgVox - 1) / kWgVox;

    // this thread's input channels (one unit of 8 at one tap) for every voxel it gathers
    const int u = k0 / 8 + (tid & 7);
    const bool unit_ok = u < a.k_units;
    const int tap = KIND == kWgTransposed ? 0 : u / a.units_per_tap;
    const int c = (u - tap * a.units_per_tap) * 8;
    const int dz = tap / (a.ks * a.ks) - a.pad, dy = tap / a.ks % a.ks - a.pad, dx = tap % a.ks - a.pad;
    const bool second = c >= a.c1;
    const bf16* in = second ? a.in2.p + a.in2.offset + (c - a.c1) : a.in1.p + a.in1.offset + c;
    const int pitch = second ? a.in2.pitch : a.in1.pitch;
    // and its gradient channels
    constexpr int kUnits = NT / 8;
    const int g_row = tid / kUnits, g_ch = tid % kUnits * 8;
    const bool g_ok = g_row < kWgVox && n0 + g_ch < a.cout;
    constexpr int kMine = kWgVox / kRows;
    Walk walk[kMine], g_walk;
    const bf16* src[kMine];
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
        const int m = mb + (tid >> 3) + kRows * i;
        walk[i].start(P, m);
        src[i] = in + (m + (KIND == kWgSame ? (dz * P.h + dy) * P.w + dx : 0)) * (long long)pitch;
    }
    g_walk.start(P, mb + g_row);
    const bf16* g_src = P.g + (mb + g_row) * (long long)P.g_pitch + n0 + g_ch;

    int left = rows - (tid >> 3), g_left = rows - g_row;     // rows from this thread's on, at the next stage
    auto load = [&](int slot) {         // stages in order: the walks and addresses move on
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            bool ok = unit_ok && left > kRows * i;
            const bf16* from = src[i];
            if (KIND == kWgSame) {
                ok = ok && (unsigned)(walk[i].x + dx) < (unsigned)P.w && (unsigned)(walk[i].y + dy) < (unsigned)P.h &&
                     (unsigned)(walk[i].z + dz) < (unsigned)P.d;
            } else if (KIND == kWgStrided) {
                const int xx = walk[i].x * a.stride + dx, yy = walk[i].y * a.stride + dy,
                          zz = walk[i].z * a.stride + dz;
                ok = ok && (unsigned)zz < (unsigned)a.id && (unsigned)yy < (unsigned)a.ih &&
                     (unsigned)xx < (unsigned)a.iw;
                from = in + ((((long long)walk[i].b * a.id + zz) * a.ih + yy) * a.iw + xx) * pitch;
            }
            cp_async16(sA + (slot * kWgVox + (tid >> 3) + kRows * i) * AS + (tid & 7) * 8, ok ? from : a.in1.p, ok);
            if (KIND != kWgTransposed) walk[i].advance(P);
            src[i] += (long long)kWgVox * pitch;
        }
        if (g_row < kWgVox) {
            const bool ok = g_ok && g_left > 0;
            const bf16* from = g_src;
            if (KIND == kWgTransposed) {
                from = P.g + n0 + g_ch + ((((long long)g_walk.b * a.od + 2 * g_walk.z + (cls >> 2)) * a.oh +
                                           2 * g_walk.y + (cls >> 1 & 1)) * a.ow + 2 * g_walk.x + (cls & 1)) * P.g_pitch;
                g_walk.advance(P);
            }
            cp_async16(sG + (slot * kWgVox + g_row) * GS + g_ch, ok ? from : P.g, ok);
            g_src += (long long)kWgVox * P.g_pitch;
        }
        left -= kWgVox;
        g_left -= kWgVox;
    };

    float acc[NW / 8][4];
#pragma unroll
    for (int j = 0; j < NW / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;

    const int kw = (warp & 3) * 16, nw = (warp >> 2) * NW;
#pragma unroll
    for (int s = 0; s < kWgStages - 1; ++s) {
        if (s < stages) load(s);
        cp_async_commit();
    }
    int slot = 0, fill = kWgStages - 1;
    for (int s = 0; s < stages; ++s) {
        cp_async_wait<kWgStages - 2>();
        __syncthreads();
        if (s + kWgStages - 1 < stages) load(fill);
        cp_async_commit();
        const bf16* A = sA + slot * kWgVox * AS + ((lane & 7) + ((lane >> 4) << 3)) * AS + kw + ((lane >> 3) & 1) * 8;
        const bf16* G = sG + slot * kWgVox * GS + ((lane & 7) + ((lane >> 3) & 1) * 8) * GS + nw +
                        (NW == 16 ? (lane >> 4) * 8 : 0);
#pragma unroll
        for (int step = 0; step < kWgVox / 16; ++step) {
            // (rows past the chunk's end were staged as zeros and add nothing)
            unsigned af[4];
            ldmatrix_x4_trans(af, A + 16 * step * AS);
            if (NW == 16) {
                unsigned bf[4];
                ldmatrix_x4_trans(bf, G + 16 * step * GS);
                mma_bf16(acc[0], af, bf[0], bf[1]);
                mma_bf16(acc[NW / 8 - 1], af, bf[2], bf[3]);
            } else {
                unsigned bf[2];
                ldmatrix_x2_trans(bf, G + 16 * step * GS);
                mma_bf16(acc[0], af, bf[0], bf[1]);
            }
        }
        slot = slot + 1 == kWgStages ? 0 : slot + 1;
        fill = fill + 1 == kWgStages ? 0 : fill + 1;
    }
    cp_async_wait<0>();
    const int k_elems = a.k_units * 8;
    float* base = P.dw + (size_t)cls * a.cin * a.cout;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int k = k0 + kw + (lane >> 2) + half * 8;
        if (k >= k_elems) continue;
#pragma unroll
        for (int nt = 0; nt < NW / 8; ++nt) {
            const int n = n0 + nw + nt * 8 + (lane & 3) * 2;
            if (n >= a.cout) continue;
            atomicAdd(base + (size_t)k * a.cout + n, acc[nt][half * 2]);
            atomicAdd(base + (size_t)k * a.cout + n + 1, acc[nt][half * 2 + 1]);
        }
    }
}

// The weight gradients of several layers in one launch: they depend on nothing
// but finished activations and gradients, a layer's blocks all take one chain's
// time, and most layers alone leave SMs idle.
struct WgradMany {
    int count;
    int first[FFX_WGRAD_LAYERS + 1];     // first block of each layer
    Wgrad layer[FFX_WGRAD_LAYERS];
};

__global__ void __launch_bounds__(kWgThreads) conv_wgrad_kernel(const __grid_constant__ WgradMany A) {
    int k = 0;
    while (k + 1 < A.count && (int)blockIdx.x >= A.first[k + 1]) ++k;
    const Wgrad& P = A.layer[k];
    int r = (int)blockIdx.x - A.first[k];
    const int bk = r % P.blocks_k;
    r /= P.blocks_k;
    const int bn = r % P.blocks_n, bz = r / P.blocks_n;
    if (P.nt == 16) {
        if (P.kind == kWgSame) wgrad_block<16, kWgSame>(P, bk, bn, bz);
        else if (P.kind == kWgStrided) wgrad_block<16, kWgStrided>(P, bk, bn, bz);
        else wgrad_block<16, kWgTransposed>(P, bk, bn, bz);
    } else {
        if (P.kind == kWgSame) wgrad_block<32, kWgSame>(P, bk, bn, bz);
        else if (P.kind == kWgStrided) wgrad_block<32, kWgStrided>(P, bk, bn, bz);
        else wgrad_block<32, kWgTransposed>(P, bk, bn, bz);
    }
}

// ------------------------------------------------------------ elementwise
// dy *= (y > 0): the ReLU derivative, in place.
__global__ void relu_backward_kernel(long long voxels, int channels, bf16* dy, int dy_pitch, const bf16* y,
                                     int y_pitch, int y_offset) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= voxels * channels) return;
    const long long v = i / channels;
    const int c = (int)(i - v * channels);
    if (!(__bfloat162float(y[v * y_pitch + y_offset + c]) > 0.f)) dy[v * dy_pitch + c] = __float2bfloat16_rn(0.f);
}

// The ReLU derivative of a layer's output gradient, in place, and its bias
// gradient, in one pass over 16-byte groups of 8 channels (a separate scalar
// pass each took 29 + 11 us at 64^3 x 2 x 16 channels; the bytes take 8). A
// thread keeps one group of channels; blocks end with one atomic per channel.
__global__ void __launch_bounds__(256) relu_bias_kernel(long long voxels, int channels, bf16* dy, int dy_pitch,
                                                        const bf16* __restrict__ y, int y_pitch, int y_offset,
                                                        float* db) {
    __shared__ float part[128];
    const int groups = channels / 8, c = threadIdx.x % groups * 8;
    for (int i = threadIdx.x; i < channels; i += blockDim.x) part[i] = 0.f;
    __syncthreads();
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int rows = blockDim.x / groups;
    for (long long v = (long long)blockIdx.x * rows + threadIdx.x / groups; v < voxels;
         v += (long long)gridDim.x * rows) {
        uint4* at = reinterpret_cast<uint4*>(dy + v * dy_pitch + c);
        uint4 g = *at;
        bf16* h = reinterpret_cast<bf16*>(&g);
        if (y) {
            const uint4 o = __ldg(reinterpret_cast<const uint4*>(y + v * y_pitch + y_offset + c));
            const bf16* k = reinterpret_cast<const bf16*>(&o);
#pragma unroll
            for (int e = 0; e < 8; ++e)
                if (!(__bfloat162float(k[e]) > 0.f)) h[e] = __float2bfloat16_rn(0.f);
            *at = g;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] += __bfloat162float(h[e]);
    }
    // lanes of a warp with the same channels (groups is a power of two up to 16)
    for (int o = groups; o < 32; o <<= 1)
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], o);
    if ((threadIdx.x & 31) < groups)
#pragma unroll
        for (int e = 0; e < 8; ++e) atomicAdd(&part[c + e], sum[e]);
    __syncthreads();
    for (int i = threadIdx.x; i < channels; i += blockDim.x) atomicAdd(db + i, part[i]);
}

// db[c] += sum over voxels of g[v][c] (block-local FP32 sums, one atomic per channel and block).
__global__ void bias_grad_kernel(long long voxels, int channels, const bf16* g, int pitch, float* db) {
    __shared__ float part[128];
    for (int c = threadIdx.x; c < channels; c += blockDim.x) part[c] = 0.f;
    __syncthreads();
    const long long per = (voxels + gridDim.x - 1) / gridDim.x;
    const long long vb = blockIdx.x * per, ve = min(voxels, vb + per);
    for (int c = threadIdx.x % channels; c < channels; c += channels) {
        float s = 0.f;
        for (long long v = vb + threadIdx.x / channels; v < ve; v += blockDim.x / channels)
            s += __bfloat162float(g[v * pitch + c]);
        atomicAdd(&part[c], s);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < channels; c += blockDim.x) atomicAdd(db + c, part[c]);
}

// Adam on FP32 master weights, refreshing their BF16 copy.
__global__ void adam_kernel(long long n, float* w, float* m, float* v, const float* g, bf16* w16, float lr, float b1,
                            float b2, float eps, float c1, float c2) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (w16) w16[i] = __float2bfloat16_rn(wi);
}

// Network input: channel 0 = scale * divergence, channel 1 = solid mask,
// channels 2..7 = 0 (the first convolution reads 8 channels).
// out = src * scale; with `max_abs`, scale = 1 / (input_scale * weight) in
// FP64 (0 for a zero input), the factor that undoes the input normalisation.
// adam_kernel for all parameter tensors of a network in one launch (blockIdx.y:
// the tensor): 42 launches of 3 us each were latency only.
struct AdamMany {
    FfxAdamSlot slot[FFX_ADAM_SLOTS];
    float lr, b1, b2, eps, c1, c2;
};
__global__ void __launch_bounds__(256) adam_many_kernel(const __grid_constant__ AdamMany P) {
    const FfxAdamSlot& s = P.slot[blockIdx.y];
    bf16* w16 = (bf16*)s.w_bf16;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < s.n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = s.g[i];
        const float mi = P.b1 * s.m[i] + (1.f - P.b1) * gi;
        const float vi = P.b2 * s.v[i] + (1.f - P.b2) * gi * gi;
        s.m[i] = mi;
        s.v[i] = vi;
        const float wi = s.w[i] - P.lr * (mi / P.c1) / (sqrtf(vi / P.c2) + P.eps);
        s.w[i] = wi;
        if (w16) w16[i] = __float2bfloat16_rn(wi);
    }
}

__global__ void unpack_channel_kernel(long long voxels, const float* __restrict__ src, int pitch, float scale,
                                      const float* max_abs, double weight, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (max_abs) {
        const float m = *max_abs;
        scale = m > 0.f ? (float)(1.0 / ((1.0 / (double)m) * weight)) : 0.f;
    }
    if (i < voxels) out[i] = src[i * pitch] * scale;
}

// Coarse collider mask: a coarse cell is solid when at least `threshold` of its
// eight children are.
__global__ void mask_restrict_kernel(int cx, int cy, int cz, const uint8_t* __restrict__ fine, int threshold,
                                     uint8_t* __restrict__ coarse) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (long long)cx * cy * cz) return;
    const int x = (int)(c % cx), y = (int)((c / cx) % cy), z = (int)(c / ((long long)cx * cy));
    const int fx = 2 * cx, fy = 2 * cy;
    int n = 0;
    for (int dz = 0; dz < 2; ++dz)
        for (int dy = 0; dy < 2; ++dy)
            for (int dx = 0; dx < 2; ++dx)
                n += fine[(2 * x + dx) + (long long)fx * ((2 * y + dy) + (long long)fy * (2 * z + dz))] != 0;
    coarse[c] = n >= threshold ? 1 : 0;
}

// Scale of the network's input from max |div| on the device: 1 / max (0 when
// the field is zero), the FP32 rounding of the FP64 quotient, as a host would
// form it.
__device__ __forceinline__ float input_scale(const float* max_abs) {
    const float m = *max_abs;
    return m > 0.f ? (float)(1.0 / (double)m) : 0.f;
}

__global__ void pack_input_kernel(long long voxels, const float* div, const uint8_t* mask, float scale,
                                  const float* max_abs, bf16* out) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= voxels) return;
    if (max_abs) scale = input_scale(max_abs);
    __align__(16) bf16 c[8];
    c[0] = __float2bfloat16_rn(scale * div[v]);
    c[1] = __float2bfloat16_rn(mask && mask[v] ? 1.f : 0.f);
#pragma unroll
    for (int k = 2; k < 8; ++k) c[k] = __float2bfloat16_rn(0.f);
    *reinterpret_cast<uint4*>(out + v * 8) = *reinterpret_cast<const uint4*>(c);
}

// Loss sum_v (pred - target)^2 / count over fluid voxels and its gradient,
// written into channel 0 of an 8-channel BF16 tensor (the head's input gradient
// is formed from it by the head's data-gradient convolution).
// `fluid`: the count of fluid voxels on the device (fluid_count_kernel), for
// 1 / max(count, 1), or NULL for inv_count.
__global__ void mse_kernel(long long voxels, const float* pred, int pred_pitch, const float* target,
                           const uint8_t* mask, float inv_count, const int* fluid, bf16* grad, double* loss) {
    if (fluid) inv_count = (float)(1.0 / (double)max(*fluid, 1));
    double e = 0.0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < voxels;
         v += (long long)gridDim.x * blockDim.x) {
        const bool open = !(mask && mask[v]);
        const float d = open ? pred[v * pred_pitch] - target[v] : 0.f;
        e += (double)d * d * inv_count;
        __align__(16) bf16 c[8];
        c[0] = __float2bfloat16_rn(2.f * d * inv_count);
#pragma unroll
        for (int k = 1; k < 8; ++k) c[k] = __float2bfloat16_rn(0.f);
        *reinterpret_cast<uint4*>(grad + v * 8) = *reinterpret_cast<const uint4*>(c);
    }
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0 && e != 0.0) atomicAdd(loss, e);
}

// *count += voxels - sum of the mask (its fluid voxels where it holds 0 and 1).
__global__ void fluid_count_kernel(long long voxels, const uint8_t* __restrict__ mask, int* count) {
    int n = 0;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < voxels;
         v += (long long)gridDim.x * blockDim.x)
        n += 1 - (int)mask[v];
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(count, n);
}

// dst[t][co][ci] = src[flip ? taps - 1 - t : t][ci][co]: the weights of the
// data-gradient convolution (transposed per tap; taps reversed for a padded
// convolution whose gradient correlates with the mirrored kernel).
__global__ void weight_transpose_kernel(int taps, int cin, int cout, int flip, const bf16* src, bf16* dst) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long n = (long long)taps * cin * cout;
    if (i >= n) return;
    const int ci = (int)(i % cin);
    const long long r = i / cin;
    const int co = (int)(r % cout);
    const int t = (int)(r / cout);
    const int ts = flip ? taps - 1 - t : t;
    dst[i] = src[((long long)ts * cin + ci) * cout + co];
}

bool view_ok(const FfxTensorView& t, int channels) {
    return t.data && t.pitch >= t.offset + channels && t.pitch % 8 == 0 && t.offset % 8 == 0 &&
           ((uintptr_t)t.data & 15) == 0;
}

int make_conv(const FfxConv* c, Conv& a) {
    FFX_REQUIRE(c && c->batch >= 1 && c->c1 >= 8 && c->c1 % 8 == 0 && c->c2 >= 0 && c->c2 % 8 == 0 &&
                    c->cout >= 8 && c->cout % 8 == 0 && c->weight && ((uintptr_t)c->weight & 15) == 0,
                "ffx_conv: invalid arguments (channels multiples of 8, 16-byte aligned weights)");
    for (int i = 0; i < 3; ++i)
        FFX_REQUIRE(c->in_dims[i] >= 1 && c->out_dims[i] >= 1 && c->in_dims[i] <= 4096 && c->out_dims[i] <= 4096,
                    "ffx_conv: invalid dimensions");
    FFX_REQUIRE(view_ok(c->in1, c->c1) && (c->c2 == 0 || view_ok(c->in2, c->c2)),
                "ffx_conv: input views need 16-byte aligned data, pitch and offset multiples of 8");
    if (c->transposed) {
        FFX_REQUIRE(c->ksize == 2 && c->stride == 2 && c->pad == 0 && c->out_dims[0] == 2 * c->in_dims[0] &&
                        c->out_dims[1] == 2 * c->in_dims[1] && c->out_dims[2] == 2 * c->in_dims[2],
                    "ffx_conv: the transposed form is 2^3 with stride 2 onto a grid twice as large");
    } else {
        FFX_REQUIRE(c->ksize >= 1 && c->ksize <= 3 && c->stride >= 1 && c->stride <= 2 && c->pad >= 0 &&
                        c->pad < c->ksize,
                    "ffx_conv: kernel size 1..3, stride 1..2, pad < kernel size");
        for (int i = 0; i < 3; ++i)
            FFX_REQUIRE(c->out_dims[i] == (c->in_dims[i] + 2 * c->pad - c->ksize) / c->stride + 1,
                        "ffx_conv: output dimensions do not follow from input, kernel, stride and pad");
    }
    if (c->out)
        FFX_REQUIRE(c->out_pitch >= c->out_offset + c->cout && c->out_pitch % 8 == 0 && c->out_offset % 8 == 0 &&
                        ((uintptr_t)c->out & 15) == 0,
                    "ffx_conv: output view");
    if (c->out_f32) FFX_REQUIRE(c->out_f32_pitch >= c->cout && c->out_f32_pitch % 2 == 0, "ffx_conv: FP32 output pitch");
    a.batch = c->batch;
    a.id = c->in_dims[0]; a.ih = c->in_dims[1]; a.iw = c->in_dims[2];
    a.od = c->out_dims[0]; a.oh = c->out_dims[1]; a.ow = c->out_dims[2];
    a.c1 = c->c1; a.c2 = c->c2; a.cin = c->c1 + c->c2; a.cout = c->cout;
    a.ks = c->ksize; a.stride = c->stride; a.pad = c->pad; a.transposed = c->transposed;
    a.taps = c->transposed ? 1 : c->ksize * c->ksize * c->ksize;
    a.units_per_tap = a.cin / 8;
    a.k_units = a.taps * a.units_per_tap;
    const long long in_vox = (long long)a.batch * a.id * a.ih * a.iw;
    a.rows = c->transposed ? in_vox : (long long)a.batch * a.od * a.oh * a.ow;
    FFX_REQUIRE(a.rows < (1LL << 40), "ffx_conv: too many voxels");
    a.in1 = View{(const bf16*)c->in1.data, c->in1.pitch, c->in1.offset};
    a.in2 = View{(const bf16*)(c->c2 ? c->in2.data : c->in1.data), c->c2 ? c->in2.pitch : 8,
                 c->c2 ? c->in2.offset : 0};
    a.w = (const bf16*)c->weight;
    a.bias = c->bias;
    a.relu = c->relu;
    a.accumulate = c->accumulate;
    a.out = (bf16*)c->out;
    a.out_pitch = c->out_pitch;
    a.out_offset = c->out_offset;
    a.out_f32 = c->out_f32;
    a.out_f32_pitch = c->out_f32_pitch;
    return FFX_OK;
}

// ---------------------------------------------- TMA convolution, host side
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver the runtime loaded (no link-time libcuda).
EncodeTiled tensor_map_encoder() {
    static EncodeTiled fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// 3x3x3, stride 1, pad 1, one input view, channels the kernel tiles.
bool tma_eligible(const Conv& a) {
    return !a.transposed && a.ks == 3 && a.stride == 1 && a.pad == 1 && a.c2 == 0 &&
           (a.cin % 16 == 0 || a.cin == 8) && a.cin <= 512 && a.cout % 16 == 0 && a.od == a.id && a.oh == a.ih &&
           a.ow == a.iw;
}
int tma_bn(int cout) { return cout % 64 == 0 ? 64 : (cout % 32 == 0 ? 32 : 16); }
int tma_groups(int cin) { return (cin + 15) / 16; }
long long tma_packed_elems(const Conv& a) { return (long long)tma_groups(a.cin) * 27 * 16 * a.cout; }

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) !=
                                                     cudaSuccess || n <= 0)
            n = 148;
    }
    return n;
}

}  // namespace
}  // namespace ffx

using namespace ffx;

extern "C" {

int ffx_conv_forward(const FfxConv* c, void* stream) {
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    FFX_REQUIRE(a.out || a.out_f32, "ffx_conv_forward: no output");
    int bn = a.cout <= 16 ? 16 : (a.cout <= 32 ? 32 : 64);
    const long long row_blocks = (a.rows + kBM - 1) / kBM * (a.transposed ? 8 : 1);
    while (bn > 16 && row_blocks * ((a.cout + bn - 1) / bn) < sm_count()) bn /= 2;
    const dim3 grid((unsigned)((a.rows + kBM - 1) / kBM), (unsigned)((a.cout + bn - 1) / bn), a.transposed ? 8 : 1);
    FFX_REQUIRE(grid.x < (1u << 31), "ffx_conv_forward: grid too large");
    if (bn == 16) conv_fwd_kernel<16><<<grid, kGemmThreads, 0, as_stream(stream)>>>(a);
    else if (bn == 32) conv_fwd_kernel<32><<<grid, kGemmThreads, 0, as_stream(stream)>>>(a);
    else conv_fwd_kernel<64><<<grid, kGemmThreads, 0, as_stream(stream)>>>(a);
    return launch_status("conv_fwd_kernel");
}

int ffx_conv_forward_tc(const FfxConv* c, void* stream) {
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    FFX_REQUIRE(a.out || a.out_f32, "ffx_conv_forward_tc: no output");
    const int bn = a.cout <= 16 ? 16 : (a.cout <= 32 ? 32 : 64);
    const dim3 grid((unsigned)((a.rows + kBM - 1) / kBM), (unsigned)((a.cout + bn - 1) / bn), a.transposed ? 8 : 1);
    FFX_REQUIRE(grid.x < (1u << 31), "ffx_conv_forward_tc: grid too large");
    static bool configured = false;     // dynamic shared memory above 48 KB, once per process
    if (!configured) {
        cudaFuncSetAttribute(conv_fwd_tc_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<16>());
        cudaFuncSetAttribute(conv_fwd_tc_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<32>());
        cudaFuncSetAttribute(conv_fwd_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_smem_bytes<64>());
        configured = true;
    }
    cudaStream_t st = as_stream(stream);
    if (bn == 16) conv_fwd_tc_kernel<16><<<grid, kGemmThreads, tc_smem_bytes<16>(), st>>>(a);
    else if (bn == 32) conv_fwd_tc_kernel<32><<<grid, kGemmThreads, tc_smem_bytes<32>(), st>>>(a);
    else conv_fwd_tc_kernel<64><<<grid, kGemmThreads, tc_smem_bytes<64>(), st>>>(a);
    return launch_status("conv_fwd_tc_kernel");
}

int ffx_conv_packed_bytes(const FfxConv* c, int64_t* bytes) {
    FFX_REQUIRE(bytes, "ffx_conv_packed_bytes: invalid arguments");
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    *bytes = tma_eligible(a) ? tma_packed_elems(a) * 2 : 0;
    return FFX_OK;
}

int ffx_conv_pack_weights(const FfxConv* c, void* packed, void* stream) {
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    FFX_REQUIRE(tma_eligible(a), "ffx_conv_pack_weights: not a 3x3x3 stride-1 pad-1 convolution the TMA kernel tiles");
    FFX_REQUIRE(packed && ((uintptr_t)packed & 15) == 0, "ffx_conv_pack_weights: packed buffer (16-byte aligned)");
    const long long n = tma_packed_elems(a);
    conv3_pack_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(a.w, a.cin, a.cout, tma_bn(a.cout),
                                                                        tma_groups(a.cin), (bf16*)packed);
    return launch_status("conv3_pack_kernel");
}

int ffx_conv_forward_tma(const FfxConv* c, const void* packed, void* stream) {
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    if (!tma_eligible(a)) {
        // 1^3 and transposed 2^3 layers with 8 or 16 output channels: the per-voxel kernel;
        // the remaining shapes: the mma.sync implicit GEMM
        const bool one = !a.transposed && a.ks == 1 && a.stride == 1 && a.pad == 0;
        if ((one || a.transposed) && (a.cout == 8 || a.cout == 16) && a.c2 == 0 &&
            (a.transposed ? 8 : 1) * a.cin * a.cout <= kDirectMaxWeights && (a.out || a.out_f32)) {
            const long long vox = (long long)a.batch * a.od * a.oh * a.ow;
            if (a.transposed) {
                const size_t smem = sizeof(float) * 2 * (size_t)a.cin * a.cout;
                const dim3 grid((unsigned)((a.rows + kDirectThreads - 1) / kDirectThreads), 4);
                if (a.cout == 8) conv_up_kernel<8><<<grid, kDirectThreads, smem, as_stream(stream)>>>(a);
                else conv_up_kernel<16><<<grid, kDirectThreads, smem, as_stream(stream)>>>(a);
                return launch_status("conv_up_kernel");
            }
            const size_t smem = sizeof(float) * (size_t)a.cin * a.cout;
            const unsigned blocks = (unsigned)((vox + kDirectThreads - 1) / kDirectThreads);
            if (a.cout == 8) conv_direct_kernel<8><<<blocks, kDirectThreads, smem, as_stream(stream)>>>(a);
            else conv_direct_kernel<16><<<blocks, kDirectThreads, smem, as_stream(stream)>>>(a);
            return launch_status("conv_direct_kernel");
        }
        return ffx_conv_forward(c, stream);
    }
    FFX_REQUIRE(a.out || a.out_f32, "ffx_conv_forward_tma: no output");
    FFX_REQUIRE(packed && ((uintptr_t)packed & 15) == 0,
                "ffx_conv_forward_tma: packed weights (ffx_conv_pack_weights, 16-byte aligned)");
    FFX_REQUIRE(!a.out_f32 || a.out_f32_pitch >= a.cout, "ffx_conv_forward_tma: FP32 output pitch");
    EncodeTiled encode = tensor_map_encoder();
    FFX_REQUIRE(encode, "ffx_conv_forward_tma: cuTensorMapEncodeTiled is not available from the driver");
    const int bn = tma_bn(a.cout);
    TmaConv P;
    std::memset(&P, 0, sizeof(P));
    P.wpack = (const bf16*)packed;
    P.batch = a.batch;
    P.d = a.id; P.h = a.ih; P.w = a.iw;
    P.cin = a.cin; P.cout = a.cout; P.groups = tma_groups(a.cin);
    P.planes = a.cin == 8 ? 1 : 2;
    P.tiles_x = (a.iw + kTmX - 1) / kTmX;
    P.tiles_y = (a.ih + kTmY - 1) / kTmY;
    // deepest tile (z slices sharing one halo) that still gives every SM two tiles
    const long long nblocks = a.cout / bn;
    const long long want = 2LL * sm_count();
    P.bz = 1;
    for (int bz = 4; bz >= 1; bz >>= 1) {
        const long long blocks = (long long)P.tiles_x * P.tiles_y * ((a.id + bz - 1) / bz) * a.batch * nblocks;
        if (blocks >= want || bz == 1) { P.bz = bz; break; }
    }
    P.tiles_z = (a.id + P.bz - 1) / P.bz;
    P.nblocks = (int)nblocks;
    const long long tiles = (long long)P.tiles_x * P.tiles_y * P.tiles_z * a.batch * nblocks;
    FFX_REQUIRE(tiles < (1LL << 31), "ffx_conv_forward_tma: too many tiles");
    P.tiles = (int)tiles;
    const uint32_t box_bytes = 8u * kTmHX * kTmHY * (uint32_t)(P.bz + 2) * 2u;
    P.plane = (box_bytes + 127u) & ~127u;
    P.stage = 2 * P.plane + 27u * 32u * (uint32_t)bn;
    P.tx = (uint32_t)P.planes * box_bytes + 27u * 32u * (uint32_t)bn;
    // as many stages as fit (the ring runs across tiles), at most four
    P.stages = std::min(kTmMaxStages, (int)((kTmSmemLimit - 128u) / P.stage));
    FFX_REQUIRE(P.stages >= 1, "ffx_conv_forward_tma: a stage does not fit in shared memory");
    const size_t smem = (size_t)P.stages * P.stage + 128;
    const uint32_t need = 2u * (uint32_t)P.bz * (uint32_t)bn;    // two accumulator sets
    P.cols = need <= 32 ? 32u : (need <= 64 ? 64u : (need <= 128 ? 128u : (need <= 256 ? 256u : 512u)));
    FFX_REQUIRE(need <= 512, "ffx_conv_forward_tma: accumulators exceed tensor memory");
    // persistent: one block per SM (the stage ring fills its shared memory)
    const long long blocks = std::min<long long>(tiles, sm_count());
    P.bias = a.bias;
    P.relu = a.relu;
    P.accumulate = a.accumulate;
    P.out = a.out;
    P.out_pitch = a.out_pitch;
    P.out_offset = a.out_offset;
    P.out_f32 = a.out_f32;
    P.out_f32_pitch = a.out_f32_pitch;
    // input activations as a (channel, x, y, z, batch) tensor, zero outside
    const cuuint64_t pitch = (cuuint64_t)a.in1.pitch * 2;
    const cuuint64_t dims[5] = {(cuuint64_t)a.cin, (cuuint64_t)a.iw, (cuuint64_t)a.ih, (cuuint64_t)a.id,
                                (cuuint64_t)a.batch};
    const cuuint64_t strides[4] = {pitch, pitch * a.iw, pitch * a.iw * a.ih, pitch * a.iw * a.ih * a.id};
    const cuuint32_t box[5] = {8, kTmHX, kTmHY, (cuuint32_t)(P.bz + 2), 1};
    const cuuint32_t estride[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(&P.act, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, (void*)(a.in1.p + a.in1.offset), dims,
                              strides, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    FFX_REQUIRE(r == CUDA_SUCCESS, "ffx_conv_forward_tma: cuTensorMapEncodeTiled rejected the input view");
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(conv3_tma_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTmSmemLimit);
        cudaFuncSetAttribute(conv3_tma_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTmSmemLimit);
        cudaFuncSetAttribute(conv3_tma_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTmSmemLimit);
        configured = true;
    }
    const dim3 grid((unsigned)blocks, 1, 1);
    cudaStream_t st = as_stream(stream);
    if (bn == 16) conv3_tma_kernel<16><<<grid, kTmThreads, smem, st>>>(P);
    else if (bn == 32) conv3_tma_kernel<32><<<grid, kTmThreads, smem, st>>>(P);
    else conv3_tma_kernel<64><<<grid, kTmThreads, smem, st>>>(P);
    return launch_status("conv3_tma_kernel");
}

int ffx_conv_timeouts(int32_t* out, int32_t reset) {
    FFX_REQUIRE(out, "ffx_conv_timeouts: invalid arguments");
    int e = cuda_status(cudaMemcpyFromSymbol(out, g_conv_timeouts, sizeof(int32_t)), "ffx_conv_timeouts: read");
    if (e) return e;
    if (reset) {
        const int32_t zero = 0;
        e = cuda_status(cudaMemcpyToSymbol(g_conv_timeouts, &zero, sizeof(int32_t)), "ffx_conv_timeouts: reset");
    }
    return e;
}

static int make_wgrad(const FfxConv* c, const void* grad, int32_t grad_pitch, float* dweight, Wgrad& P) {
    Conv a;
    int e = make_conv(c, a);
    if (e) return e;
    FFX_REQUIRE(grad && dweight && grad_pitch >= c->cout && grad_pitch % 8 == 0 && ((uintptr_t)grad & 15) == 0,
                "ffx_conv_weight_grad: invalid gradient view");
    const long long chunk = 8192;
    const long long splits = (a.rows + chunk - 1) / chunk;
    FFX_REQUIRE(splits * (a.transposed ? 8 : 1) < 65536 && a.rows < (1ll << 31),
                "ffx_conv_weight_grad: too many voxels for one launch");
    P = {};
    P.a = a;
    P.g = (const bf16*)grad;
    P.g_pitch = grad_pitch;
    P.dw = dweight;
    P.chunk = (int)chunk;
    P.w = a.transposed ? a.iw : a.ow;
    P.h = a.transposed ? a.ih : a.oh;
    P.d = a.transposed ? a.id : a.od;
    P.step_x = kWgVox % P.w;
    P.step_y = kWgVox / P.w % P.h;
    P.step_z = kWgVox / P.w / P.h;
    P.nt = a.cout <= 16 ? 16 : 32;      // 16 output channels a block where the layer has no more
    const bool same = a.stride == 1 && a.id == a.od && a.ih == a.oh && a.iw == a.ow;
    P.kind = a.transposed ? kWgTransposed : (same ? kWgSame : kWgStrided);
    P.blocks_k = (a.k_units * 8 + kWgK - 1) / kWgK;
    P.blocks_n = (a.cout + P.nt - 1) / P.nt;
    P.blocks_z = (int)(splits * (a.transposed ? 8 : 1));
    return FFX_OK;
}

int ffx_conv_weight_grad_many(int32_t count, const FfxWeightGrad* layers, void* stream) {
    FFX_REQUIRE(count >= 1 && count <= FFX_WGRAD_LAYERS && layers, "ffx_conv_weight_grad_many: invalid arguments");
    WgradMany A;
    A.count = count;
    A.first[0] = 0;
    long long blocks = 0;
    for (int k = 0; k < count; ++k) {
        Wgrad& P = A.layer[k];
        if (int e = make_wgrad(&layers[k].conv, layers[k].grad, layers[k].grad_pitch, layers[k].dweight, P)) return e;
        blocks += (long long)P.blocks_k * P.blocks_n * P.blocks_z;
        FFX_REQUIRE(blocks < (1ll << 31), "ffx_conv_weight_grad_many: too many blocks for one launch");
        A.first[k + 1] = (int)blocks;
    }
    constexpr int smem = kWgStages * kWgVox * (kWgK + 8 + 32 + 8) * (int)sizeof(bf16);
    static std::atomic<uint64_t> ready{0};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess && !(ready.load(std::memory_order_acquire) >> (dev & 63) & 1)) {
        err = cudaFuncSetAttribute(conv_wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err == cudaSuccess) ready.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_release);
    }
    if (err != cudaSuccess) return cuda_status(err, "ffx_conv_weight_grad_many");
    conv_wgrad_kernel<<<(unsigned)blocks, kWgThreads, smem, as_stream(stream)>>>(A);
    return launch_status("conv_wgrad_kernel");
}

int ffx_conv_weight_grad(const FfxConv* c, const void* grad, int32_t grad_pitch, float* dweight, void* stream) {
    FFX_REQUIRE(c, "ffx_conv_weight_grad: invalid arguments");
    const FfxWeightGrad one = {*c, grad, grad_pitch, dweight};
    return ffx_conv_weight_grad_many(1, &one, stream);
}

int ffx_relu_backward(int64_t voxels, int32_t channels, void* dy, int32_t dy_pitch, const void* y, int32_t y_pitch,
                      int32_t y_offset, void* stream) {
    FFX_REQUIRE(voxels >= 1 && channels >= 1 && dy && y && dy_pitch >= channels && y_pitch >= y_offset + channels,
                "ffx_relu_backward: invalid arguments");
    const long long n = voxels * channels;
    relu_backward_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(voxels, channels, (bf16*)dy, dy_pitch,
                                                                             (const bf16*)y, y_pitch, y_offset);
    return launch_status("relu_backward_kernel");
}

int ffx_bias_grad(int64_t voxels, int32_t channels, const void* g, int32_t pitch, float* dbias, void* stream) {
    FFX_REQUIRE(voxels >= 1 && channels >= 1 && channels <= 128 && 256 % channels == 0 && g && dbias &&
                    pitch >= channels,
                "ffx_bias_grad: invalid arguments (channels divide 256, at most 128)");
    const long long blocks = std::min<long long>(1184, (voxels + 255) / 256);
    bias_grad_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(voxels, channels, (const bf16*)g, pitch, dbias);
    return launch_status("bias_grad_kernel");
}

int ffx_adam(int64_t n, float* w, float* m, float* v, const float* g, void* w_bf16, float lr, float beta1,
             float beta2, float eps, int32_t step, void* stream) {
    FFX_REQUIRE(n >= 1 && w && m && v && g && step >= 1 && lr > 0.f, "ffx_adam: invalid arguments");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    adam_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(n, w, m, v, g, (bf16*)w_bf16, lr, beta1, beta2,
                                                                    eps, c1, c2);
    return launch_status("adam_kernel");
}

int ffx_adam_many(int32_t count, const FfxAdamSlot* slots, float lr, float beta1, float beta2, float eps, int32_t step,
                  void* stream) {
    FFX_REQUIRE(count >= 1 && count <= FFX_ADAM_SLOTS && slots && step >= 1 && lr > 0.f,
                "ffx_adam_many: invalid arguments");
    AdamMany P;
    int64_t most = 1;
    for (int k = 0; k < count; ++k) {
        const FfxAdamSlot& s = slots[k];
        FFX_REQUIRE(s.n >= 1 && s.w && s.m && s.v && s.g, "ffx_adam_many: slot %d is incomplete", k);
        P.slot[k] = s;
        most = std::max<int64_t>(most, s.n);
    }
    P.lr = lr;
    P.b1 = beta1;
    P.b2 = beta2;
    P.eps = eps;
    P.c1 = 1.f - powf(beta1, (float)step);
    P.c2 = 1.f - powf(beta2, (float)step);
    const dim3 grid((unsigned)std::min<int64_t>(blocks_for(most, 256), 148), (unsigned)count);
    adam_many_kernel<<<grid, 256, 0, as_stream(stream)>>>(P);
    return launch_status("adam_many_kernel");
}

int ffx_relu_bias_backward(int64_t voxels, int32_t channels, void* dy, int32_t dy_pitch, const void* y, int32_t y_pitch,
                           int32_t y_offset, float* dbias, void* stream) {
    FFX_REQUIRE(voxels >= 1 && channels >= 8 && channels <= 128 && (channels & (channels - 1)) == 0 && dy && dbias &&
                dy_pitch >= channels && dy_pitch % 8 == 0 && ((uintptr_t)dy & 15) == 0,
                "ffx_relu_bias_backward: invalid arguments (channels: a power of two in [8, 128])");
    FFX_REQUIRE(!y || (y_pitch >= y_offset + channels && y_offset >= 0 && y_pitch % 8 == 0 && y_offset % 8 == 0 &&
                       ((uintptr_t)y & 15) == 0), "ffx_relu_bias_backward: invalid activation view");
    const long long rows = 256 / (channels / 8);
    const unsigned blocks = (unsigned)std::min<long long>((voxels + rows - 1) / rows, 148 * 4);
    relu_bias_kernel<<<blocks, 256, 0, as_stream(stream)>>>(voxels, channels, (bf16*)dy, dy_pitch, (const bf16*)y,
                                                            y_pitch, y_offset, dbias);
    return launch_status("relu_bias_kernel");
}

int ffx_weight_transpose(int32_t taps, int32_t cin, int32_t cout, int32_t flip, const void* src, void* dst,
                         void* stream) {
    FFX_REQUIRE(taps >= 1 && cin >= 1 && cout >= 1 && src && dst && src != dst, "ffx_weight_transpose: invalid arguments");
    const long long n = (long long)taps * cin * cout;
    weight_transpose_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(taps, cin, cout, flip, (const bf16*)src,
                                                                                (bf16*)dst);
    return launch_status("weight_transpose_kernel");
}

int ffx_pack_input(int64_t voxels, const float* div, const uint8_t* mask, float scale, void* out, void* stream) {
    FFX_REQUIRE(voxels >= 1 && div && out && ((uintptr_t)out & 15) == 0, "ffx_pack_input: invalid arguments");
    pack_input_kernel<<<blocks_for(voxels, 256), 256, 0, as_stream(stream)>>>(voxels, div, mask, scale, nullptr,
                                                                            (bf16*)out);
    return launch_status("pack_input_kernel");
}

int ffx_pack_input_scaled(int64_t voxels, const float* div, const uint8_t* mask, const float* max_abs, void* out,
                          void* stream) {
    FFX_REQUIRE(voxels >= 1 && div && max_abs && out && ((uintptr_t)out & 15) == 0,
                "ffx_pack_input_scaled: invalid arguments");
    pack_input_kernel<<<blocks_for(voxels, 256), 256, 0, as_stream(stream)>>>(voxels, div, mask, 0.f, max_abs,
                                                                            (bf16*)out);
    return launch_status("pack_input_kernel");
}

int ffx_mask_restrict(const int32_t coarse_n[3], const uint8_t* fine, int32_t threshold, uint8_t* coarse,
                      void* stream) {
    FFX_REQUIRE(coarse_n && coarse_n[0] >= 1 && coarse_n[1] >= 1 && coarse_n[2] >= 1 && fine && coarse &&
                threshold >= 1 && threshold <= 8 &&
                (int64_t)coarse_n[0] * coarse_n[1] * coarse_n[2] * 8 < (int64_t(1) << 40),
                "ffx_mask_restrict: invalid arguments");
    const int64_t n = (int64_t)coarse_n[0] * coarse_n[1] * coarse_n[2];
    mask_restrict_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(coarse_n[0], coarse_n[1], coarse_n[2],
                                                                            fine, threshold, coarse);
    return launch_status("mask_restrict_kernel");
}

int ffx_unpack_channel(int64_t voxels, const float* src, int32_t pitch, float scale, float* out, void* stream) {
    FFX_REQUIRE(voxels >= 1 && src && out && pitch >= 1, "ffx_unpack_channel: invalid arguments");
    unpack_channel_kernel<<<blocks_for(voxels, 256), 256, 0, as_stream(stream)>>>(voxels, src, pitch, scale, nullptr,
                                                                                0.0, out);
    return launch_status("unpack_channel_kernel");
}

int ffx_unpack_channel_scaled(int64_t voxels, const float* src, int32_t pitch, const float* max_abs, double weight,
                              float* out, void* stream) {
    FFX_REQUIRE(voxels >= 1 && src && max_abs && out && pitch >= 1, "ffx_unpack_channel_scaled: invalid arguments");
    unpack_channel_kernel<<<blocks_for(voxels, 256), 256, 0, as_stream(stream)>>>(voxels, src, pitch, 0.f, max_abs,
                                                                                weight, out);
    return launch_status("unpack_channel_kernel");
}

int ffx_mse_grad(int64_t voxels, const float* pred, int32_t pred_pitch, const float* target, const uint8_t* mask,
                 float inv_count, void* grad, double* loss, void* stream) {
    FFX_REQUIRE(voxels >= 1 && pred && target && grad && loss && pred_pitch >= 1 && ((uintptr_t)grad & 15) == 0,
                "ffx_mse_grad: invalid arguments");
    const unsigned blocks = (unsigned)std::min<long long>(blocks_for(voxels, 256), 148 * 8);
    mse_kernel<<<blocks, 256, 0, as_stream(stream)>>>(voxels, pred, pred_pitch, target, mask, inv_count, nullptr,
                                                      (bf16*)grad, loss);
    return launch_status("mse_kernel");
}

int ffx_mse_grad_masked(int64_t voxels, const float* pred, int32_t pred_pitch, const float* target, const uint8_t* mask,
                        int32_t* fluid, void* grad, double* loss, void* stream) {
    FFX_REQUIRE(voxels >= 1 && voxels < (int64_t(1) << 31) && pred && target && mask && fluid && grad && loss &&
                pred_pitch >= 1 && ((uintptr_t)grad & 15) == 0, "ffx_mse_grad_masked: invalid arguments");
    const unsigned blocks = (unsigned)std::min<long long>(blocks_for(voxels, 256), 148 * 8);
    fluid_count_kernel<<<blocks, 256, 0, as_stream(stream)>>>(voxels, mask, fluid);
    int e = launch_status("fluid_count_kernel");
    if (e) return e;
    mse_kernel<<<blocks, 256, 0, as_stream(stream)>>>(voxels, pred, pred_pitch, target, mask, 0.f, fluid, (bf16*)grad,
                                                      loss);
    return launch_status("mse_kernel");
}

}  // extern "C"
