// boids_mlp.cu -- the sweep surrogate's network on the tensor cores.
//
// A multilayer perceptron in -> hidden -> hidden -> out with ReLU, BF16
// weights and activations and FP32 accumulation, trained with Adam on the
// mean squared error.  It maps a flock's rule parameters to its order
// statistics after a run (the ensemble's boids_ensemble_stats), so that a
// parameter sweep can be screened before the plain simulation re-runs the
// candidates it selects.  No counterpart in the reference.
//
// The forward pass's hidden-to-hidden product (rows x 256 by 256 x 256, the
// network's one square product) runs on the 5th-generation tensor cores:
// k_mlp_hidden_tc stages a 128-row tile of the activations and the whole
// weight matrix in shared memory in the canonical K-major layout, one thread
// issues tcgen05.mma (M 128, N 256, K 16) into an FP32 accumulator in tensor
// memory, and the epilogue reads it back with tcgen05.ld, adds the bias and
// writes the FP32 pre-activation and the BF16 ReLU.  The other products --
// the thin input and output layers (K or N of 8 and 4) and the backward
// pass -- run on mma.sync m16n8k16 (BF16 operands, FP32 accumulators), small,
// latency-bound products: a training batch of the 8 -> 256 -> 256 -> 4 network
// is five fused kernels (k_mlp_first, the hidden product, k_mlp_out,
// k_mlp_back2, k_mlp_back1), another shape's goes through one strided GEMM
// kernel.
#include "boids.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

namespace boidsgpu {
int set_last_error(int code, const char *msg);
}

namespace {

// A read-only BF16 matrix view: element (r, c) at p[r * rs + c * cs].
struct MatB {
    const __nv_bfloat16 *p;
    long long rs, cs;
    int rows, cols;
};

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi)
{
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ __nv_bfloat16 at(const MatB &m, int r, int c)
{
    return (r < m.rows && c < m.cols) ? m.p[r * m.rs + c * m.cs] : __float2bfloat16_rn(0.f);
}

// A training batch's kernels are launched with programmatic dependence: each
// is set up under the one before and waits here for its end (and its writes)
// before it touches anything; passes straight through without the attribute.
// 120 batches of 256 rows (30 epochs of 1024): 3.48 ms, 4.42 to 4.74 without.
__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int kWarpsM = 4;   // warps per CTA along M (16 rows each)
constexpr int kTileN = 32;   // columns per warp (4 MMA tiles of 8)

// C = A (M x K) * B (K x N) [+ bias] [* (mask > 0)], FP32 out (row-major,
// ldc) and optionally a BF16 copy of relu(C) or C (row-major, ldb16).
__global__ void __launch_bounds__(32 * kWarpsM)
k_mlp_gemm(MatB A, MatB B, float *__restrict__ C, int ldc, __nv_bfloat16 *__restrict__ C16, int ld16,
           const float *__restrict__ bias, const float *__restrict__ mask, int ldm, int relu16)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int r0 = (blockIdx.y * kWarpsM + warp) * 16;
    const int n0 = blockIdx.x * kTileN;
    const int M = A.rows, K = A.cols, N = B.cols;
    if (r0 >= M) return;
    float acc[4][4] = {};
    for (int kk = 0; kk < K; kk += 16) {
        const int ka = kk + 2 * t4;
        uint32_t a[4];
        a[0] = pack2(at(A, r0 + g, ka), at(A, r0 + g, ka + 1));
        a[1] = pack2(at(A, r0 + g + 8, ka), at(A, r0 + g + 8, ka + 1));
        a[2] = pack2(at(A, r0 + g, ka + 8), at(A, r0 + g, ka + 9));
        a[3] = pack2(at(A, r0 + g + 8, ka + 8), at(A, r0 + g + 8, ka + 9));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + 8 * j + g;
            const uint32_t b0 = pack2(at(B, ka, n), at(B, ka + 1, n));
            const uint32_t b1 = pack2(at(B, ka + 8, n), at(B, ka + 9, n));
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
                "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3])
                : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + g + (q >= 2 ? 8 : 0);
            const int c = n0 + 8 * j + 2 * t4 + (q & 1);
            if (r >= M || c >= N) continue;
            float v = acc[j][q];
            if (bias) v += bias[c];
            if (mask && !(mask[(long long)r * ldm + c] > 0.f)) v = 0.f;
            if (C) C[(long long)r * ldc + c] = v;
            if (C16) C16[(long long)r * ld16 + c] = __float2bfloat16_rn(relu16 ? fmaxf(v, 0.f) : v);
        }
    }
}

// ------------------------------------------------------------------ hidden layer on tcgen05

// C = A W + b for A rows x 256 (BF16, row-major), W 256 x 256 (BF16, fan-in
// rows), C to FP32 (pre) and BF16 ReLU (h); 128 rows per CTA.
//
// Shared memory holds both operands K-major in 8 x 16-byte core matrices
// (8 rows of 8 consecutive K elements, 128 bytes): element (r, k) at
// ((r / 8) * 32 + k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2, so core matrices
// adjacent along K are 128 bytes apart (the descriptor's leading byte offset)
// and 8-row groups 4096 bytes apart (its stride byte offset).  The weights
// arrive already in that layout, transposed (row n of the image holds
// column n of W), from k_mlp_tile_w.
constexpr int kTcM = 128, kTcN = 256, kTcK = 256;
constexpr int kTcThreads = 128;
constexpr uint32_t kTcABytes = kTcM * kTcK * 2;   // 64 KB
constexpr uint32_t kTcBBytes = kTcN * kTcK * 2;   // 128 KB
constexpr size_t kTcSmem = kTcABytes + kTcBBytes + 1024 + 64;
constexpr size_t kTcSplitSmem = kTcABytes + 64 * kTcK * 2 + 1024 + 64;  // 64 of the columns
constexpr uint32_t kTcSpinLimit = 1u << 22;      // bounded wait on the accumulator


__host__ __device__ constexpr uint32_t core_off(uint32_t r, uint32_t k)
{
    return ((r >> 3) * (kTcK / 8) + (k >> 3)) * 128 + (r & 7) * 16 + (k & 7) * 2;
}

// The weight image: W (K x N, row-major, fan-in rows) as N rows of K, in the
// core-matrix layout above, one 16-byte row chunk per thread.
__global__ void k_mlp_tile_w(const __nv_bfloat16 *__restrict__ w, __nv_bfloat16 *__restrict__ img)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;  // chunk: (n, k8)
    if (i >= (uint32_t)(kTcN * kTcK / 8)) return;
    const uint32_t n = i / (kTcK / 8), k0 = (i % (kTcK / 8)) * 8;
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = w[(size_t)(k0 + e) * kTcN + n];
    *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(img) + core_off(n, k0)) =
        *reinterpret_cast<const uint4 *>(v);
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    // start address, leading and stride byte offsets (all >> 4), the
    // descriptor version (0b001 at bit 46), no swizzle
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t src_bytes)
{
    // 16 bytes global -> shared without staging in registers; src_bytes 0
    // fills the destination with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// A CTA takes kN of the 256 columns of its 128-row tiles (kN = 256: one CTA
// per SM walks the tiles, the weight image is loaded once, and the next tile's
// activations are copied in (cp.async) while the current tile's accumulator is
// read out; kN = 64: a batch of few tiles is spread over four times as many
// CTAs, 9 against 18 us for the 256 rows of a training batch).
constexpr int kTcSplit = 64;
static_assert(kTcSplitSmem == kTcABytes + kTcSplit * kTcK * 2 + 1024 + 64, "kTcSplit columns of weights");
template <int kN>
__global__ void __launch_bounds__(kTcThreads, 1)
k_mlp_hidden_tc(const __nv_bfloat16 *__restrict__ a, int rows, const __nv_bfloat16 *__restrict__ wimg,
                const float *__restrict__ bias, float *__restrict__ pre, __nv_bfloat16 *__restrict__ h,
                uint32_t *err)
{
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    constexpr uint32_t kB = kN * kTcK * 2;  // its part of the weight image
    unsigned char *sa = tc_smem, *sb = tc_smem + kTcABytes;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(tc_smem + kTcABytes + kB);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tc_smem + kTcABytes + kB + 8);
    const int parts = kTcN / kN, tile0 = blockIdx.x / parts, tstep = gridDim.x / parts;
    const int n0 = (blockIdx.x % parts) * kN;
    wimg += (size_t)n0 * kTcK;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int ntiles = (rows + kTcM - 1) / kTcM;
    const uint32_t sa_s = (uint32_t)__cvta_generic_to_shared(sa), sb_s = (uint32_t)__cvta_generic_to_shared(sb);
    // a tile's activations into shared memory (rows past the end are zero)
    auto load_a = [&](int tile) {
        const int m0 = tile * kTcM;
        for (uint32_t i = t; i < (uint32_t)(kTcM * kTcK / 8); i += kTcThreads) {
            const uint32_t r = i / (kTcK / 8), k0 = (i % (kTcK / 8)) * 8;
            const bool in = m0 + (int)r < rows;
            cp_async16(sa_s + core_off(r, k0), a + (size_t)(in ? m0 + r : 0) * kTcK + k0, in ? 16u : 0u);
        }
    };
    const uint32_t mbar_a = (uint32_t)__cvta_generic_to_shared(mbar);
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // the accumulator: kN columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::
                         "r"((uint32_t)__cvta_generic_to_shared(tmem_slot)), "r"((uint32_t)kN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    chain_wait();
    for (uint32_t i = t; i < kB / 16; i += kTcThreads) cp_async16(sb_s + 16 * i, wimg + 8 * i, 16u);
    if (tile0 < ntiles) load_a(tile0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    // the shared-memory writes become visible to the tensor cores
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // kind::f16: FP32 D (bit 4), BF16 A and B (bits 7, 10), both K-major,
    // N / 8 at bit 17, M / 16 at bit 24
    const uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = tile0; tile < ntiles; tile += tstep) {
        if (t == 0) {
#pragma unroll 1
            for (int kk = 0; kk < kTcK / 16; ++kk) {
                const uint64_t ad = smem_desc(sa_s + kk * 256, 128, (kTcK / 8) * 128);
                const uint64_t bd = smem_desc(sb_s + kk * 256, 128, (kTcK / 8) * 128);
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(kk));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar_a)
                         : "memory");
        }
        // wait for the accumulator (bounded: a wait that gives up flags an error)
        uint32_t done = 0;
        for (uint32_t it = 0; it < kTcSpinLimit && !done; ++it)
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                         " selp.u32 %0, 1, 0, p;\n}\n"
                         : "=r"(done)
                         : "r"(mbar_a), "r"(phase)
                         : "memory");
        phase ^= 1u;
        done = __syncthreads_and(done);  // one decision for the whole CTA
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!done) {
            *reinterpret_cast<volatile uint32_t *>(err) = 1u;
            ok = false;
            break;
        }
        // the activations' buffer is free: the next tile's copy runs under the epilogue
        const int nxt = tile + tstep;
        if (nxt < ntiles) load_a(nxt);
        // epilogue: warp w reads tensor-memory lanes 32w.. (its rows), 32 columns at a time
        const int r = tile * kTcM + warp * 32 + lane;
        const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
        for (int c = 0; c < kN; c += 32) {
            uint32_t v[32];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(trow + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (r < rows) {
#pragma unroll
                for (int q = 0; q < 32; q += 8) {
                    float f[8];
                    __align__(16) __nv_bfloat16 hb[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        f[e] = __uint_as_float(v[q + e]) + __ldg(bias + n0 + c + q + e);
                        hb[e] = __float2bfloat16_rn(fmaxf(f[e], 0.f));
                    }
                    if (pre) {
                        float4 *po = reinterpret_cast<float4 *>(pre + (size_t)r * kTcN + n0 + c + q);
                        po[0] = make_float4(f[0], f[1], f[2], f[3]);
                        po[1] = make_float4(f[4], f[5], f[6], f[7]);
                    }
                    *reinterpret_cast<uint4 *>(h + (size_t)r * kTcN + n0 + c + q) = *reinterpret_cast<const uint4 *>(hb);
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();  // the accumulator is read and the next activations are in place
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    (void)ok;
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kN));
    }
}

// The whole forward pass for inference, fused: 8 -> 256 -> 256 -> 4 in one
// kernel that reads x and writes y.  Per 128-row tile the CTA computes the
// first layer into shared memory (each lane keeps its 8 columns of W1 in
// registers; the tile's x is copied in ahead with cp.async), the tensor
// cores run the hidden product into one of two accumulators in tensor
// memory, and the epilogue applies bias and ReLU and folds the 256 -> 4
// output layer in registers while the next tile's product runs in the other
// accumulator.  Sixteen warps: warps w, w + 4, w + 8 and w + 12 read the same
// accumulator lanes, 64 columns each, and their partial outputs meet in shared
// memory.  The rounding points are those of the unfused pass (BF16 x, h1, h2;
// FP32 sums).  Bound by the FP32 work around the product (the first layer's
// 8 FMA and the epilogue's 4 per activation) and its latencies.
constexpr int kTcIn = 8, kTcOut = 4;
constexpr int kTcFwdThreads = 512, kTcFwdParts = kTcFwdThreads / 128;  // warps w, w + 4, ...: a part of the columns each
constexpr uint32_t kTcXBytes = kTcM * kTcIn * 4;  // a tile's inputs, 4 KB
constexpr size_t kTcFwdSmem = kTcABytes + kTcBBytes + 1024 + 64 +
                              sizeof(float) * (kTcN * kTcOut + kTcN + kTcOut + kTcFwdParts * kTcM * kTcOut) + kTcXBytes;
static_assert(kTcFwdSmem <= 227 * 1024, "one CTA per SM");

__global__ void __launch_bounds__(kTcFwdThreads, 1)
k_mlp_forward_tc(const float *__restrict__ x, int rows, const __nv_bfloat16 *__restrict__ w1,
                 const float *__restrict__ b1, const __nv_bfloat16 *__restrict__ wimg, const float *__restrict__ b2,
                 const __nv_bfloat16 *__restrict__ w3, const float *__restrict__ b3, float *__restrict__ y, uint32_t *err)
{
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    unsigned char *sa = tc_smem, *sb = tc_smem + kTcABytes;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(tc_smem + kTcABytes + kTcBBytes);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tc_smem + kTcABytes + kTcBBytes + 8);
    float *sw3 = reinterpret_cast<float *>(tc_smem + kTcABytes + kTcBBytes + 64);  // W3 as float, [k][j]
    float *sb2 = sw3 + kTcN * kTcOut, *sb3 = sb2 + kTcN;
    float *ypart = sb3 + kTcOut;                        // [kTcFwdParts][kTcM][kTcOut]: the column parts' outputs
    float *sx = ypart + kTcFwdParts * kTcM * kTcOut;    // the current tile's inputs, [kTcM][kTcIn]
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int ntiles = (rows + kTcM - 1) / kTcM;
    const uint32_t sa_s = (uint32_t)__cvta_generic_to_shared(sa), sb_s = (uint32_t)__cvta_generic_to_shared(sb);
    const uint32_t sx_s = (uint32_t)__cvta_generic_to_shared(sx);
    auto load_x = [&](int tile) {  // one 16-byte chunk per thread
        static_assert(kTcXBytes / 16 <= kTcFwdThreads, "a tile's inputs are at most one chunk per thread");
        if (t >= (int)(kTcXBytes / 16)) return;
        const int m0 = tile * kTcM, r = t / 2;
        const bool in = m0 + r < rows;
        cp_async16(sx_s + 16 * t, x + (size_t)(in ? m0 + r : 0) * kTcIn + 4 * (t & 1), in ? 16u : 0u);
    };
    for (uint32_t i = t; i < kTcBBytes / 16; i += kTcFwdThreads) cp_async16(sb_s + 16 * i, wimg + 8 * i, 16u);
    if ((int)blockIdx.x < ntiles) load_x(blockIdx.x);
    for (int i = t; i < kTcN * kTcOut; i += kTcFwdThreads) sw3[i] = __bfloat162float(w3[i]);
    for (int i = t; i < kTcN; i += kTcFwdThreads) sb2[i] = b2[i];
    if (t < kTcOut) sb3[t] = b3[t];
    // this lane's 8 columns of the first layer (the same for every row it computes)
    const int k0 = lane * 8;
    float w1r[kTcIn][8], b1r[8];
#pragma unroll
    for (int i = 0; i < kTcIn; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) w1r[i][e] = __bfloat162float(w1[i * kTcN + k0 + e]);
#pragma unroll
    for (int e = 0; e < 8; ++e) b1r[e] = b1[k0 + e];
    // the first layer of a tile (its inputs in sx) into shared memory: warp w
    // takes rows w, w + 16, ..., lane its 8 columns; rows past the end are zero
    auto layer1 = [&](int tile) {
        const int m0 = tile * kTcM;
        for (int r = warp; r < kTcM; r += kTcFwdThreads / 32) {
            __align__(16) __nv_bfloat16 hb[8];
            if (m0 + r < rows) {
                float xb[kTcIn];
#pragma unroll
                for (int i = 0; i < kTcIn; ++i) xb[i] = __bfloat162float(__float2bfloat16_rn(sx[r * kTcIn + i]));
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float acc = 0.f;
#pragma unroll
                    for (int i = 0; i < kTcIn; ++i) acc = __fmaf_rn(xb[i], w1r[i][e], acc);
                    hb[e] = __float2bfloat16_rn(fmaxf(__fadd_rn(acc, b1r[e]), 0.f));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) hb[e] = __float2bfloat16_rn(0.f);
            }
            *reinterpret_cast<uint4 *>(sa + core_off(r, k0)) = *reinterpret_cast<const uint4 *>(hb);
        }
    };
    const uint32_t mbar_a = (uint32_t)__cvta_generic_to_shared(mbar);
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_a));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // two accumulators: 512 columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::
                         "r"((uint32_t)__cvta_generic_to_shared(tmem_slot)), "r"(2u * kTcN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the first tile's inputs and the tables are in place
    if ((int)blockIdx.x < ntiles) layer1(blockIdx.x);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const uint32_t idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTcN >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
    auto issue = [&](uint32_t acc_col) {  // one thread: the tile's product into the accumulator at acc_col
#pragma unroll 1
        for (int kk = 0; kk < kTcK / 16; ++kk) {
            const uint64_t ad = smem_desc(sa_s + kk * 256, 128, (kTcK / 8) * 128);
            const uint64_t bd = smem_desc(sb_s + kk * 256, 128, (kTcK / 8) * 128);
            asm volatile(
                "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem + acc_col),
                "l"(ad), "l"(bd), "r"(idesc), "r"(kk));
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar_a)
                     : "memory");
    };
    uint32_t phase = 0, buf = 0;
    if (t == 0 && (int)blockIdx.x < ntiles) issue(0);
    constexpr int kPart = kTcN / kTcFwdParts;  // columns of a warp
    const int quarter = warp & 3, part = warp >> 2;  // accumulator lanes 32 * quarter.., columns kPart * part..
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int nxt = tile + gridDim.x;
        if (nxt < ntiles) load_x(nxt);  // sx is free: this tile's first layer is done
        // wait for this tile's product (bounded: a wait that gives up flags an error)
        uint32_t done = 0;
        for (uint32_t it = 0; it < kTcSpinLimit && !done; ++it)
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                         " selp.u32 %0, 1, 0, p;\n}\n"
                         : "=r"(done)
                         : "r"(mbar_a), "r"(phase)
                         : "memory");
        phase ^= 1u;
        asm volatile("cp.async.wait_all;" ::: "memory");
        done = __syncthreads_and(done);  // one decision for the CTA; the next inputs are in place
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!done) {
            *reinterpret_cast<volatile uint32_t *>(err) = 1u;
            break;
        }
        // the next tile's first layer into the freed buffer, and its product
        // into the other accumulator, while this tile's is read out
        if (nxt < ntiles) {
            layer1(nxt);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            if (t == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                issue((buf ^ 1u) * kTcN);
            }
        }
        // epilogue: bias, ReLU, BF16 and the output layer over this warp's part of the columns
        const int rl = quarter * 32 + lane;  // row within the tile
        const uint32_t trow = tmem + buf * kTcN + ((uint32_t)(quarter * 32) << 16);
        float yo[kTcOut] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int c = part * kPart; c < (part + 1) * kPart; c += 32) {
            uint32_t v[32];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                  "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                  "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                : "r"(trow + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                const float hv = __bfloat162float(
                    __float2bfloat16_rn(fmaxf(__fadd_rn(__uint_as_float(v[e]), sb2[c + e]), 0.f)));
#pragma unroll
                for (int j = 0; j < kTcOut; ++j) yo[j] = __fmaf_rn(hv, sw3[(c + e) * kTcOut + j], yo[j]);
            }
        }
        *reinterpret_cast<float4 *>(ypart + (part * kTcM + rl) * kTcOut) = make_float4(yo[0], yo[1], yo[2], yo[3]);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();  // this accumulator is read before a later tile's product reuses it
        if (part == 0) {
            const int r = tile * kTcM + rl;
            float4 a = *reinterpret_cast<const float4 *>(ypart + rl * kTcOut);
#pragma unroll
            for (int q = 1; q < kTcFwdParts; ++q) {
                const float4 b = *reinterpret_cast<const float4 *>(ypart + (q * kTcM + rl) * kTcOut);
                a = make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
            }
            if (r < rows)
                *reinterpret_cast<float4 *>(y + (size_t)r * kTcOut) =
                    make_float4(__fadd_rn(a.x, sb3[0]), __fadd_rn(a.y, sb3[1]), __fadd_rn(a.z, sb3[2]),
                                __fadd_rn(a.w, sb3[3]));
        }
        buf ^= 1u;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kTcN));
    }
}

// Mean squared error over rows x cols and its gradient 2 (y - t) / (rows * cols).
__global__ void k_mlp_mse(const float *__restrict__ y, const float *__restrict__ t, int n, float scale,
                          float *__restrict__ dy, __nv_bfloat16 *__restrict__ dy16, double *loss)
{
    __shared__ double part[8];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double e2 = 0.0;
    if (i < n) {
        const float e = y[i] - t[i];
        e2 = (double)e * e;
        dy[i] = 2.f * e * scale;
        dy16[i] = __float2bfloat16_rn(2.f * e * scale);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = e2;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[w];
        atomicAdd(loss, s * scale);
    }
}

// db[c] = sum over rows of d[r][c].
__global__ void k_mlp_colsum(const float *__restrict__ d, int rows, int cols, float *__restrict__ db)
{
    const int c = blockIdx.x;
    float s = 0.f;
    for (int r = threadIdx.x; r < rows; r += blockDim.x) s += d[(long long)r * cols + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ float part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
        db[c] = t;
    }
}

// Adam on the FP32 master parameters; refreshes their BF16 copy.
__global__ void k_mlp_adam(float *__restrict__ p, const float *__restrict__ gr, float *__restrict__ m,
                           float *__restrict__ v, __nv_bfloat16 *__restrict__ p16, long long n, float lr, float b1,
                           float b2, float c1, float c2, float eps)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = gr[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float q = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = q;
    p16[i] = __float2bfloat16_rn(q);
}

__global__ void k_to_bf16(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

__global__ void k_gather_rows(const float *__restrict__ src, const int *__restrict__ idx, int rows, int cols,
                              float *__restrict__ dst)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)rows * cols) return;
    const long long r = i / cols, c = i - r * cols;
    dst[i] = src[(long long)idx[r] * cols + c];
}

// ------------------------------------------------------------------ a training batch in five kernels
//
// The 8 -> 256 -> 256 -> 4 network's forward and backward pass and its Adam
// step, for one batch: k_mlp_first (gather, first layer, weight image),
// k_mlp_hidden_tc, k_mlp_out (output layer, loss, gradient of the hidden
// layer's outputs), k_mlp_back2 (everything that needs those), k_mlp_back1
// (first layer's gradients, the update).  Every product is the same sequence
// of mma.m16n8k16 over ascending K as k_mlp_gemm's, and every column sum the
// same order as k_mlp_colsum's, so the results are the same bits.
//
// Bound by the chain of launches and of loads inside each (a batch is
// 0.1 GFLOP).  A batch of 256 rows took 17 launches and 174 us, most of it in
// k_mlp_gemm's 2-byte strided loads on few CTAs; the operands are now staged
// through shared memory with 16-byte copies and read with ldmatrix.
constexpr int kFH = 256, kFIn = 8, kFOut = 4, kFThreads = 256;

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool kTrans>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    if (kTrans)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

// rows x cols (cols a multiple of 8) of a row-major matrix of row length ld
// into shared memory with row length cols + 8; rows past `have` are zero.
__device__ __forceinline__ void stage_rows(__nv_bfloat16 *dst, const __nv_bfloat16 *src, int ld, int rows, int cols,
                                           int have)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int per = cols / 8;
    for (int i = threadIdx.x; i < rows * per; i += kFThreads) {
        const int r = i / per, c = (i - r * per) * 8;
        const bool in = r < have;
        cp_async16(d + 2 * (r * (cols + 8) + c), src + (size_t)(in ? r : 0) * ld + c, in ? 16u : 0u);
    }
}

struct AdamArgs {
    float *m, *v;
    float lr, b1, b2, c1, c2, eps;
};

// One parameter's update (null m: the gradient is stored instead).
__device__ __forceinline__ void adam_or_store(const AdamArgs &ad, float *p, __nv_bfloat16 *p16, float *grad,
                                              long long i, float gi)
{
    if (!ad.m) {
        grad[i] = gi;
        return;
    }
    const float mi = ad.b1 * ad.m[i] + (1.f - ad.b1) * gi;
    const float vi = ad.b2 * ad.v[i] + (1.f - ad.b2) * gi * gi;
    ad.m[i] = mi;
    ad.v[i] = vi;
    const float q = p[i] - ad.lr * (mi / ad.c1) / (sqrtf(vi / ad.c2) + ad.eps);
    p[i] = q;
    p16[i] = __float2bfloat16_rn(q);
}

// 16 rows a CTA: x[idx] rounded to BF16, and the first layer; further CTAs
// lay the hidden weights out for the tensor cores.
__global__ void __launch_bounds__(kFThreads)
k_mlp_first(const float *__restrict__ x, const int *__restrict__ idx, int rows, const __nv_bfloat16 *__restrict__ w1,
            const float *__restrict__ b1, const __nv_bfloat16 *__restrict__ w2, __nv_bfloat16 *__restrict__ img,
            __nv_bfloat16 *__restrict__ x16, float *__restrict__ pre1, __nv_bfloat16 *__restrict__ h1, int row_ctas)
{
    chain_wait();
    if ((int)blockIdx.x >= row_ctas) {  // as k_mlp_tile_w
        const uint32_t i = (blockIdx.x - row_ctas) * kFThreads + threadIdx.x;
        const uint32_t n = i % kTcN, k0 = i / kTcN * 8;
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = w2[(size_t)(k0 + e) * kTcN + n];
        *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(img) + core_off(n, k0)) =
            *reinterpret_cast<const uint4 *>(v);
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int r0 = blockIdx.x * 16;
    uint32_t a[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int r = r0 + g + 8 * q;
        if (r >= rows) continue;
        const float2 v = *reinterpret_cast<const float2 *>(x + (size_t)(idx ? idx[r] : r) * kFIn + 2 * t4);
        a[q] = pack2(__float2bfloat16_rn(v.x), __float2bfloat16_rn(v.y));
        if (warp == 0) *reinterpret_cast<uint32_t *>(x16 + (size_t)r * kFIn + 2 * t4) = a[q];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int nn = warp * 32 + 8 * j, n = nn + g;
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(d, a, pack2(w1[2 * t4 * kFH + n], w1[(2 * t4 + 1) * kFH + n]), 0u);
        const int c = nn + 2 * t4;
        const float2 bb = *reinterpret_cast<const float2 *>(b1 + c);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * q;
            if (r >= rows) continue;
            const float v0 = d[2 * q] + bb.x, v1 = d[2 * q + 1] + bb.y;
            *reinterpret_cast<float2 *>(pre1 + (size_t)r * kFH + c) = make_float2(v0, v1);
            *reinterpret_cast<uint32_t *>(h1 + (size_t)r * kFH + c) =
                pack2(__float2bfloat16_rn(fmaxf(v0, 0.f)), __float2bfloat16_rn(fmaxf(v1, 0.f)));
        }
    }
}

// 16 rows a CTA: y = h2 W3 + b3 (warp 0), the loss and dy, and
// d2 = (dy W3^T) * (pre2 > 0) (all warps, 32 columns each).
__global__ void __launch_bounds__(kFThreads)
k_mlp_out(const __nv_bfloat16 *__restrict__ h2, const float *__restrict__ pre2, const float *__restrict__ tgt,
          const int *__restrict__ idx, int rows, const __nv_bfloat16 *__restrict__ w3, const float *__restrict__ b3,
          float scale, float *__restrict__ dy, __nv_bfloat16 *__restrict__ dy16, float *__restrict__ d2,
          __nv_bfloat16 *__restrict__ d2_16, double *loss)
{
    __shared__ __align__(16) __nv_bfloat16 sh[16 * (kFH + 8)];
    __shared__ __align__(16) __nv_bfloat16 sw[kFH * kFOut];
    __shared__ __align__(4) __nv_bfloat16 sdy[16 * kFOut];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int r0 = blockIdx.x * 16;
    chain_wait();
    stage_rows(sh, h2 + (size_t)r0 * kFH, kFH, 16, kFH, rows - r0);
    if (threadIdx.x < kFH * kFOut / 8)
        cp_async16((uint32_t)__cvta_generic_to_shared(sw) + 16 * threadIdx.x, w3 + 8 * threadIdx.x, 16u);
    // this thread's pre-activations, in flight meanwhile
    float2 pm[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * q;
            pm[j][q] = r < rows ? *reinterpret_cast<const float2 *>(pre2 + (size_t)r * kFH + warp * 32 + 8 * j + 2 * t4)
                                : make_float2(0.f, 0.f);
        }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        const __nv_bfloat16 zero = __ushort_as_bfloat16(0);
#pragma unroll
        for (int kk = 0; kk < kFH; kk += 16) {
            uint32_t a[4];
            ldsm4<false>(a, sh + (lane & 15) * (kFH + 8) + kk + (lane >> 4) * 8);
            const int ka = kk + 2 * t4;
            const bool in = g < kFOut;
            mma16816(d, a, in ? pack2(sw[ka * kFOut + g], sw[(ka + 1) * kFOut + g]) : pack2(zero, zero),
                     in ? pack2(sw[(ka + 8) * kFOut + g], sw[(ka + 9) * kFOut + g]) : pack2(zero, zero));
        }
        double e2 = 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int rl = g + (q >= 2 ? 8 : 0), r = r0 + rl, c = 2 * t4 + (q & 1);
            if (c >= kFOut) continue;
            float gr = 0.f;
            if (r < rows) {
                const float e = (d[q] + b3[c]) - tgt[(size_t)(idx ? idx[r] : r) * kFOut + c];
                e2 += (double)e * e;
                gr = 2.f * e * scale;
                dy[(size_t)r * kFOut + c] = gr;
                dy16[(size_t)r * kFOut + c] = __float2bfloat16_rn(gr);
            }
            sdy[rl * kFOut + c] = __float2bfloat16_rn(gr);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e2 += __shfl_down_sync(0xffffffffu, e2, o);
        if (lane == 0) atomicAdd(loss, e2 * scale);
    }
    __syncthreads();
    uint32_t a[4] = {0u, 0u, 0u, 0u};
    if (t4 < 2) {
        a[0] = *reinterpret_cast<const uint32_t *>(sdy + g * kFOut + 2 * t4);
        a[1] = *reinterpret_cast<const uint32_t *>(sdy + (g + 8) * kFOut + 2 * t4);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int nn = warp * 32 + 8 * j, c = nn + 2 * t4;
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(d, a, t4 < 2 ? *reinterpret_cast<const uint32_t *>(sw + (nn + g) * kFOut + 2 * t4) : 0u, 0u);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * q;
            if (r >= rows) continue;
            const float v0 = pm[j][q].x > 0.f ? d[2 * q] : 0.f, v1 = pm[j][q].y > 0.f ? d[2 * q + 1] : 0.f;
            *reinterpret_cast<float2 *>(d2 + (size_t)r * kFH + c) = make_float2(v0, v1);
            *reinterpret_cast<uint32_t *>(d2_16 + (size_t)r * kFH + c) =
                pack2(__float2bfloat16_rn(v0), __float2bfloat16_rn(v1));
        }
    }
}

// Sums of columns c0 .. c0 + kC - 1 (kC 4 or 8) of d (row length cols), in
// k_mlp_colsum's order; thread j < kC returns column c0 + j's.
template <int kC>
__device__ __forceinline__ float colsums(const float *__restrict__ d, int rows, int cols, int c0, float *part)
{
    float s[kC] = {};
    for (int r = threadIdx.x; r < rows; r += kFThreads) {
#pragma unroll
        for (int j = 0; j < kC; j += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(d + (size_t)r * cols + c0 + j);
            s[j] += v.x;
            s[j + 1] += v.y;
            s[j + 2] += v.z;
            s[j + 3] += v.w;
        }
    }
#pragma unroll
    for (int j = 0; j < kC; ++j) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_down_sync(0xffffffffu, s[j], o);
        if ((threadIdx.x & 31) == 0) part[(threadIdx.x >> 5) * kC + j] = s[j];
    }
    __syncthreads();
    float t = 0.f;
    if (threadIdx.x < kC)
        for (int w = 0; w < kFThreads / 32; ++w) t += part[w * kC + threadIdx.x];
    return t;
}

// Everything that needs dy and d2, by ranges of CTAs:
//   32            dW2 = h1^T d2, 32 x 64 outputs each
//   8             dW3 = h2^T dy, 32 rows each
//   4 ceil(rows / 16)  d1 = (d2 W2^T) * (pre1 > 0), 16 x 64 outputs each
//   32, 1         db2, db3
constexpr int kBackK = 256;  // rows of a K pass
constexpr size_t kBackSmem = 2 * (size_t)(kBackK * (32 + 8) + kBackK * (64 + 8));
static_assert(kBackSmem >= 2 * (size_t)(16 + 64) * (kFH + 8), "d1's operands fit");

__global__ void __launch_bounds__(kFThreads)
k_mlp_back2(const __nv_bfloat16 *__restrict__ h1, const __nv_bfloat16 *__restrict__ h2,
            const float *__restrict__ pre1, const float *__restrict__ dy, const __nv_bfloat16 *__restrict__ dy16,
            const float *__restrict__ d2, const __nv_bfloat16 *__restrict__ d2_16, int rows,
            const __nv_bfloat16 *__restrict__ w2, float *__restrict__ gw2, float *__restrict__ gb2,
            float *__restrict__ gw3, float *__restrict__ gb3, float *__restrict__ d1,
            __nv_bfloat16 *__restrict__ d1_16)
{
    extern __shared__ __align__(16) unsigned char back_smem[];
    __shared__ float part[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3, mat = lane >> 3;
    int blk = blockIdx.x;
    chain_wait();
    if (blk < 32 + 8) {
        // A = h^T of 32 columns m0.., staged as K rows of h1 (dW2) or h2 (dW3)
        const bool w2part = blk < 32;
        const int m0 = w2part ? (blk >> 2) * 32 : (blk - 32) * 32, n0 = w2part ? (blk & 3) * 64 : 0;
        constexpr int la = 32 + 8, lb = 64 + 8;
        __nv_bfloat16 *sa = reinterpret_cast<__nv_bfloat16 *>(back_smem), *sb = sa + kBackK * la;
        const int mw = (warp & 1) * 16, nw = (warp >> 1) * 16;  // the warp's 16 x 16 outputs
        float d[2][4] = {};
        for (int k0 = 0; k0 < rows; k0 += kBackK) {
            const int have = min(kBackK, rows - k0), kr = (have + 15) & ~15;
            stage_rows(sa, (w2part ? h1 : h2) + (size_t)k0 * kFH + m0, kFH, kr, 32, have);
            if (w2part) stage_rows(sb, d2_16 + (size_t)k0 * kFH + n0, kFH, kr, 64, have);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (w2part) {
                for (int kk = 0; kk < kr; kk += 16) {
                    uint32_t a[4], b[4];
                    ldsm4<true>(a, sa + (kk + (lane & 7) + (mat >> 1) * 8) * la + mw + (mat & 1) * 8);
                    ldsm4<true>(b, sb + (kk + (lane & 7) + (mat & 1) * 8) * lb + nw + (mat >> 1) * 8);
                    mma16816(d[0], a, b[0], b[1]);
                    mma16816(d[1], a, b[2], b[3]);
                }
            } else if (warp < 2) {
                const __nv_bfloat16 zero = __ushort_as_bfloat16(0);
                auto el = [&](int k) { return g < kFOut && k < rows ? dy16[(size_t)k * kFOut + g] : zero; };
                for (int kk = 0; kk < kr; kk += 16) {
                    uint32_t a[4];
                    ldsm4<true>(a, sa + (kk + (lane & 7) + (mat >> 1) * 8) * la + mw + (mat & 1) * 8);
                    const int k = k0 + kk + 2 * t4;
                    mma16816(d[0], a, pack2(el(k), el(k + 1)), pack2(el(k + 8), el(k + 9)));
                }
            }
            __syncthreads();
        }
        if (w2part) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    *reinterpret_cast<float2 *>(gw2 + (size_t)(m0 + mw + g + 8 * q) * kFH + n0 + nw + 8 * j + 2 * t4) =
                        make_float2(d[j][2 * q], d[j][2 * q + 1]);
        } else if (warp < 2 && t4 < 2) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                gw3[(size_t)(m0 + mw + g + 8 * q) * kFOut + 2 * t4] = d[0][2 * q];
                gw3[(size_t)(m0 + mw + g + 8 * q) * kFOut + 2 * t4 + 1] = d[0][2 * q + 1];
            }
        }
        return;
    }
    blk -= 32 + 8;
    const int d1_ctas = 4 * ((rows + 15) / 16);
    if (blk < d1_ctas) {
        const int r0 = (blk >> 2) * 16, n0 = (blk & 3) * 64;
        constexpr int ld = kFH + 8;
        __nv_bfloat16 *sa = reinterpret_cast<__nv_bfloat16 *>(back_smem), *sb = sa + 16 * ld;
        stage_rows(sa, d2_16 + (size_t)r0 * kFH, kFH, 16, kFH, rows - r0);
        stage_rows(sb, w2 + (size_t)n0 * kFH, kFH, 64, kFH, 64);
        const int c = n0 + warp * 8 + 2 * t4;
        float2 pm[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * q;
            pm[q] = r < rows ? *reinterpret_cast<const float2 *>(pre1 + (size_t)r * kFH + c) : make_float2(0.f, 0.f);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kk = 0; kk < kFH; kk += 32) {
            uint32_t a0[4], a1[4], b[4];
            ldsm4<false>(a0, sa + (lane & 15) * ld + kk + (lane >> 4) * 8);
            ldsm4<false>(a1, sa + (lane & 15) * ld + kk + 16 + (lane >> 4) * 8);
            ldsm4<false>(b, sb + (warp * 8 + (lane & 7)) * ld + kk + mat * 8);
            mma16816(d, a0, b[0], b[1]);
            mma16816(d, a1, b[2], b[3]);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int r = r0 + g + 8 * q;
            if (r >= rows) continue;
            const float v0 = pm[q].x > 0.f ? d[2 * q] : 0.f, v1 = pm[q].y > 0.f ? d[2 * q + 1] : 0.f;
            *reinterpret_cast<float2 *>(d1 + (size_t)r * kFH + c) = make_float2(v0, v1);
            *reinterpret_cast<uint32_t *>(d1_16 + (size_t)r * kFH + c) =
                pack2(__float2bfloat16_rn(v0), __float2bfloat16_rn(v1));
        }
        return;
    }
    blk -= d1_ctas;
    if (blk < 32) {
        const float v = colsums<8>(d2, rows, kFH, 8 * blk, part);
        if (threadIdx.x < 8) gb2[8 * blk + threadIdx.x] = v;
    } else {
        const float v = colsums<4>(dy, rows, kFOut, 0, part);
        if (threadIdx.x < kFOut) gb3[threadIdx.x] = v;
    }
}

// The first layer's gradients and the update, by ranges of CTAs:
//   16        dW1 = x^T d1, two warps of 8 columns each
//   32        db1
//   the rest  Adam on the other parameters, 4 a thread (training only)
__global__ void __launch_bounds__(kFThreads)
k_mlp_back1(const __nv_bfloat16 *__restrict__ x16, const float *__restrict__ d1,
            const __nv_bfloat16 *__restrict__ d1_16, int rows, float *__restrict__ p, __nv_bfloat16 *__restrict__ p16,
            float *__restrict__ grad, long long np, AdamArgs ad)
{
    __shared__ __align__(16) __nv_bfloat16 sx[kBackK * kFIn], sd[kBackK * 16];
    __shared__ float part[64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    int blk = blockIdx.x;
    constexpr int kW1 = kFIn * kFH;
    chain_wait();
    if (blk < 16) {  // columns 16 blk .. 16 blk + 15, two warps
        const int n0 = 16 * blk;
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = 0; k0 < rows; k0 += kBackK) {
            const int have = min(kBackK, rows - k0), kr = (have + 15) & ~15;
            const uint32_t sxa = (uint32_t)__cvta_generic_to_shared(sx), sda = (uint32_t)__cvta_generic_to_shared(sd);
            for (int i = threadIdx.x; i < kr; i += kFThreads)
                cp_async16(sxa + 16 * i, x16 + (size_t)(i < have ? k0 + i : 0) * kFIn, i < have ? 16u : 0u);
            for (int i = threadIdx.x; i < 2 * kr; i += kFThreads)
                cp_async16(sda + 16 * i, d1_16 + (size_t)((i >> 1) < have ? k0 + (i >> 1) : 0) * kFH + n0 + 8 * (i & 1),
                           (i >> 1) < have ? 16u : 0u);
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            if (warp < 2) {
                const int n = 8 * warp + g;
                for (int kk = 0; kk < kr; kk += 16) {
                    const int k = kk + 2 * t4;
                    const uint32_t a[4] = {pack2(sx[k * kFIn + g], sx[(k + 1) * kFIn + g]), 0u,
                                           pack2(sx[(k + 8) * kFIn + g], sx[(k + 9) * kFIn + g]), 0u};
                    mma16816(d, a, pack2(sd[k * 16 + n], sd[(k + 1) * 16 + n]),
                             pack2(sd[(k + 8) * 16 + n], sd[(k + 9) * 16 + n]));
                }
            }
            __syncthreads();
        }
        if (warp < 2) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                adam_or_store(ad, p, p16, grad, (long long)g * kFH + n0 + 8 * warp + 2 * t4 + q, d[q]);
        }
        return;
    }
    blk -= 16;
    if (blk < 32) {
        const float v = colsums<8>(d1, rows, kFH, 8 * blk, part);
        if (threadIdx.x < 8) adam_or_store(ad, p, p16, grad, kW1 + 8 * blk + threadIdx.x, v);
        return;
    }
    const long long i = kW1 + kFH + 4 * ((long long)(blk - 32) * kFThreads + threadIdx.x);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (i + q < np) adam_or_store(ad, p, p16, grad, i + q, grad[i + q]);
}

unsigned nb(long long n, int t) { return (unsigned)((n + t - 1) / t); }

int fail(int code, const std::string &m) { return boidsgpu::set_last_error(code, m.c_str()); }

#define MCK(call)                                                                                   \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess) return fail(BOIDS_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

}  // namespace

// Parameter layout (FP32 master and BF16 copy): W1 [in x h], b1 [h],
// W2 [h x h], b2 [h], W3 [h x out], b3 [out]; W row-major (fan-in rows).
struct boids_mlp {
    int in = 0, h = 0, out = 0, device = 0;
    long long np = 0;
    long long off[6] = {};
    float *p = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
    __nv_bfloat16 *p16 = nullptr;
    long long step = 0;
    // activations for up to cap rows
    int cap = 0;
    float *x = nullptr, *t = nullptr, *pre1 = nullptr, *pre2 = nullptr, *y = nullptr, *dy = nullptr,
          *d2 = nullptr, *d1 = nullptr;
    __nv_bfloat16 *x16 = nullptr, *h1 = nullptr, *h2 = nullptr, *dy16 = nullptr, *d2_16 = nullptr, *d1_16 = nullptr;
    double *loss = nullptr;
    uint32_t *err = nullptr;  // pinned: set by a tile whose wait gave up
    cudaStream_t st = nullptr;
    __nv_bfloat16 *w2img = nullptr;  // the hidden weights in the tensor-core layout (hidden width 256)
    bool img_valid = false;           // it holds the present parameters' (p16)
    unsigned nsm = 1;                 // SMs: the tensor-core kernel's persistent grid
};

namespace {

void free_acts(boids_mlp *m)
{
    void *q[] = {m->x, m->t, m->pre1, m->pre2, m->y, m->dy, m->d2, m->d1, m->x16, m->h1, m->h2, m->dy16, m->d2_16,
                 m->d1_16};
    for (void *p : q)
        if (p) cudaFree(p);
    m->x = m->t = m->pre1 = m->pre2 = m->y = m->dy = m->d2 = m->d1 = nullptr;
    m->x16 = m->h1 = m->h2 = m->dy16 = m->d2_16 = m->d1_16 = nullptr;
    m->cap = 0;
}

int ensure_rows(boids_mlp *m, int rows)
{
    if (rows <= m->cap) return 0;
    free_acts(m);
    const long long r = rows;
    auto A = [&](auto **p, long long n) { return cudaMalloc((void **)p, sizeof(**p) * (size_t)(n ? n : 1)); };
    if (A(&m->x, r * m->in) || A(&m->t, r * m->out) || A(&m->pre1, r * m->h) || A(&m->pre2, r * m->h) ||
        A(&m->y, r * m->out) || A(&m->dy, r * m->out) || A(&m->d2, r * m->h) || A(&m->d1, r * m->h) ||
        A(&m->x16, r * m->in) || A(&m->h1, r * m->h) || A(&m->h2, r * m->h) || A(&m->dy16, r * m->out) ||
        A(&m->d2_16, r * m->h) || A(&m->d1_16, r * m->h)) {
        cudaGetLastError();
        free_acts(m);
        return fail(BOIDS_ENOMEM, "boids_mlp: cudaMalloc of activations failed");
    }
    m->cap = rows;
    return 0;
}

void gemm(boids_mlp *m, MatB A, MatB B, float *C, int ldc, __nv_bfloat16 *C16, int ld16, const float *bias,
          const float *mask, int ldm, int relu16)
{
    dim3 grid(nb(B.cols, kTileN), nb(A.rows, 16 * kWarpsM));
    k_mlp_gemm<<<grid, 32 * kWarpsM, 0, m->st>>>(A, B, C, ldc, C16, ld16, bias, mask, ldm, relu16);
}

MatB rowmajor(const __nv_bfloat16 *p, int rows, int cols) { return MatB{p, cols, 1, rows, cols}; }
MatB transposed(const __nv_bfloat16 *p, int rows, int cols)  // the transpose of a row-major rows x cols
{
    return MatB{p, 1, rows == 0 ? 0 : cols, cols, rows};
}

// Launches a kernel that calls chain_wait behind the stream's last one.
template <class... P, class... A>
void launch_chain(boids_mlp *m, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, A... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = m->st;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, P(args)...);  // (its error is the stream's last: callers look there)
}

// The hidden product of `rows` rows in m->h1: a few tiles are split by columns
// so that more SMs take part (up to a quarter of them have a tile).
void hidden_tc(boids_mlp *m, int rows, const float *b2, float *pre2)
{
    const unsigned tiles = nb(rows, kTcM), parts = kTcN / kTcSplit;
    if (tiles * parts <= m->nsm)
        launch_chain(m, k_mlp_hidden_tc<kTcSplit>, tiles * parts, kTcThreads, kTcSplitSmem, m->h1, rows, m->w2img, b2,
                     pre2, m->h2, m->err);
    else
        launch_chain(m, k_mlp_hidden_tc<kTcN>, tiles < m->nsm ? tiles : m->nsm, kTcThreads, kTcSmem, m->h1, rows,
                     m->w2img, b2, pre2, m->h2, m->err);
}

// One batch of the 8 -> 256 -> 256 -> 4 network in five kernels: rows idx[0..
// rows) (null: 0, 1, ...) of x and t.  ad.m null: the gradient into m->grad;
// else the Adam step.
bool batch_is_fused(const boids_mlp *m) { return m->w2img && m->in == kFIn && m->out == kFOut; }

void fused_batch(boids_mlp *m, const float *x, const float *t, const int *idx, int rows, const AdamArgs &ad)
{
    const __nv_bfloat16 *W1 = m->p16 + m->off[0], *W2 = m->p16 + m->off[2], *W3 = m->p16 + m->off[4];
    const float *b1 = m->p + m->off[1], *b2 = m->p + m->off[3], *b3 = m->p + m->off[5];
    const unsigned row_ctas = nb(rows, 16);
    launch_chain(m, k_mlp_first, row_ctas + kTcN * kTcK / 8 / kFThreads, kFThreads, 0, x, idx, rows, W1, b1, W2,
                 m->w2img, m->x16, m->pre1, m->h1, (int)row_ctas);
    hidden_tc(m, rows, b2, m->pre2);
    launch_chain(m, k_mlp_out, row_ctas, kFThreads, 0, m->h2, m->pre2, t, idx, rows, W3, b3,
                 1.f / (float)(rows * kFOut), m->dy, m->dy16, m->d2, m->d2_16, m->loss);
    launch_chain(m, k_mlp_back2, 32 + 8 + 4 * row_ctas + 32 + 1, kFThreads, kBackSmem, m->h1, m->h2, m->pre1, m->dy,
                 m->dy16, m->d2, m->d2_16, rows, W2, m->grad + m->off[2], m->grad + m->off[3], m->grad + m->off[4],
                 m->grad + m->off[5], m->d1, m->d1_16);
    const unsigned rest = ad.m ? nb(m->np - kFIn * kFH - kFH, 4 * kFThreads) : 0;
    launch_chain(m, k_mlp_back1, 16 + 32 + rest, kFThreads, 0, m->x16, m->d1, m->d1_16, rows, m->p, m->p16, m->grad,
                 m->np, ad);
}

// Forward pass of `rows` rows already in m->x16; output in m->y.  A hidden
// width of 256 puts the hidden-to-hidden product on the tensor cores.
void forward(boids_mlp *m, int rows, bool need_pre = true)
{
    const __nv_bfloat16 *W1 = m->p16 + m->off[0], *W2 = m->p16 + m->off[2], *W3 = m->p16 + m->off[4];
    const float *b1 = m->p + m->off[1], *b2 = m->p + m->off[3], *b3 = m->p + m->off[5];
    gemm(m, rowmajor(m->x16, rows, m->in), rowmajor(W1, m->in, m->h), m->pre1, m->h, m->h1, m->h, b1, nullptr, 0, 1);
    if (m->w2img) {
        k_mlp_tile_w<<<nb(kTcN * kTcK / 8, 256), 256, 0, m->st>>>(W2, m->w2img);
        m->img_valid = false;
        hidden_tc(m, rows, b2, need_pre ? m->pre2 : nullptr);
    } else {
        gemm(m, rowmajor(m->h1, rows, m->h), rowmajor(W2, m->h, m->h), m->pre2, m->h, m->h2, m->h, b2, nullptr, 0,
             1);
    }
    gemm(m, rowmajor(m->h2, rows, m->h), rowmajor(W3, m->h, m->out), m->y, m->out, nullptr, 0, b3, nullptr, 0, 0);
}

// Loss and gradient of `rows` rows (targets in m->t) into m->grad.
void backward(boids_mlp *m, int rows)
{
    const __nv_bfloat16 *W2 = m->p16 + m->off[2], *W3 = m->p16 + m->off[4];
    float *gW1 = m->grad + m->off[0], *gb1 = m->grad + m->off[1], *gW2 = m->grad + m->off[2],
          *gb2 = m->grad + m->off[3], *gW3 = m->grad + m->off[4], *gb3 = m->grad + m->off[5];
    const int n = rows * m->out;
    k_mlp_mse<<<nb(n, 256), 256, 0, m->st>>>(m->y, m->t, n, 1.f / (float)n, m->dy, m->dy16, m->loss);
    // layer 3: dW3 = h2^T dy, db3 = colsum(dy), d2 = (dy W3^T) * (pre2 > 0)
    gemm(m, transposed(m->h2, rows, m->h), rowmajor(m->dy16, rows, m->out), gW3, m->out, nullptr, 0, nullptr,
         nullptr, 0, 0);
    k_mlp_colsum<<<m->out, 256, 0, m->st>>>(m->dy, rows, m->out, gb3);
    gemm(m, rowmajor(m->dy16, rows, m->out), transposed(W3, m->h, m->out), m->d2, m->h, m->d2_16, m->h, nullptr,
         m->pre2, m->h, 0);
    // layer 2
    gemm(m, transposed(m->h1, rows, m->h), rowmajor(m->d2_16, rows, m->h), gW2, m->h, nullptr, 0, nullptr, nullptr,
         0, 0);
    k_mlp_colsum<<<m->h, 256, 0, m->st>>>(m->d2, rows, m->h, gb2);
    gemm(m, rowmajor(m->d2_16, rows, m->h), transposed(W2, m->h, m->h), m->d1, m->h, m->d1_16, m->h, nullptr,
         m->pre1, m->h, 0);
    // layer 1
    gemm(m, transposed(m->x16, rows, m->in), rowmajor(m->d1_16, rows, m->h), gW1, m->h, nullptr, 0, nullptr, nullptr,
         0, 0);
    k_mlp_colsum<<<m->h, 256, 0, m->st>>>(m->d1, rows, m->h, gb1);
}

// Waits for the call's work, and says whether a tensor-core tile's wait on its
// accumulator gave up (the word is cleared for the next call).  The word lies
// in pinned host memory, so that looking at it takes no copy (8 us of a call).
int finish_call(boids_mlp *m)
{
    MCK(cudaStreamSynchronize(m->st));
    if (!m->err || !*reinterpret_cast<volatile uint32_t *>(m->err)) return 0;
    *m->err = 0;
    return fail(BOIDS_ECUDA, "boids_mlp: a tensor-core tile's wait for its accumulator gave up");
}

int upload_rows(boids_mlp *m, const float *x, const float *t, int rows)
{
    MCK(cudaMemcpyAsync(m->x, x, sizeof(float) * (size_t)rows * m->in, cudaMemcpyHostToDevice, m->st));
    if (t) MCK(cudaMemcpyAsync(m->t, t, sizeof(float) * (size_t)rows * m->out, cudaMemcpyHostToDevice, m->st));
    k_to_bf16<<<nb((long long)rows * m->in, 256), 256, 0, m->st>>>(m->x, m->x16, (long long)rows * m->in);
    return 0;
}

// splitmix64-driven uniform in [-a, a]
float uni(uint64_t &s, float a)
{
    s += 0x9e3779b97f4a7c15ULL;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    z ^= z >> 31;
    return (float)(((double)(z >> 11) / 9007199254740992.0) * 2.0 - 1.0) * a;
}

}  // namespace

extern "C" {

int boids_mlp_create(int32_t n_in, int32_t n_hidden, int32_t n_out, uint64_t seed, int32_t device, boids_mlp **out)
{
    if (!out || n_in <= 0 || n_hidden <= 0 || n_out <= 0 || n_in > 4096 || n_hidden > 4096 || n_out > 4096)
        return fail(BOIDS_EINVAL, "boids_mlp_create: bad argument");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return fail(BOIDS_ECUDA, "boids_mlp_create: cudaSetDevice");
    boids_mlp *m = new boids_mlp();
    m->in = n_in;
    m->h = n_hidden;
    m->out = n_out;
    m->device = device;
    const long long sz[6] = {(long long)n_in * n_hidden, n_hidden, (long long)n_hidden * n_hidden, n_hidden,
                             (long long)n_hidden * n_out, n_out};
    for (int i = 0; i < 6; ++i) {
        m->off[i] = m->np;
        m->np += sz[i];
    }
    // He-uniform weights, zero biases
    std::vector<float> h(m->np, 0.f);
    uint64_t s = seed;
    const int fan[3] = {n_in, n_hidden, n_hidden};
    for (int l = 0; l < 3; ++l) {
        const float a = std::sqrt(6.f / (float)fan[l]);
        for (long long i = 0; i < sz[2 * l]; ++i) h[m->off[2 * l] + i] = uni(s, a);
    }
    bool ok = cudaMalloc(&m->p, 4 * m->np) == cudaSuccess && cudaMalloc(&m->grad, 4 * m->np) == cudaSuccess &&
              cudaMalloc(&m->m, 4 * m->np) == cudaSuccess && cudaMalloc(&m->v, 4 * m->np) == cudaSuccess &&
              cudaMalloc(&m->p16, 2 * m->np) == cudaSuccess && cudaMalloc(&m->loss, 8) == cudaSuccess &&
              cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && cudaMemcpy(m->p, h.data(), 4 * m->np, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemset(m->m, 0, 4 * m->np) == cudaSuccess && cudaMemset(m->v, 0, 4 * m->np) == cudaSuccess;
    if (ok) {
        k_to_bf16<<<nb(m->np, 256), 256, 0, m->st>>>(m->p, m->p16, m->np);
        ok = cudaStreamSynchronize(m->st) == cudaSuccess;
    }
    int nsm = 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && nsm > 0)
        m->nsm = (unsigned)nsm;
    if (ok && n_hidden == kTcN) {  // the hidden product on the tensor cores
        ok = cudaMalloc(&m->w2img, kTcBBytes) == cudaSuccess &&
             cudaHostAlloc(&m->err, sizeof *m->err, cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess &&
             cudaFuncSetAttribute(k_mlp_hidden_tc<kTcN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem) ==
                 cudaSuccess &&
             cudaFuncSetAttribute(k_mlp_hidden_tc<kTcSplit>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kTcSplitSmem) == cudaSuccess &&
             cudaFuncSetAttribute(k_mlp_back2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBackSmem) ==
                 cudaSuccess &&
             cudaFuncSetAttribute(k_mlp_forward_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kTcFwdSmem) == cudaSuccess;
    }
    if (m->err) *m->err = 0;
    if (!ok) {
        cudaGetLastError();
        boids_mlp_destroy(m);
        return fail(BOIDS_ENOMEM, "boids_mlp_create: device allocation failed");
    }
    *out = m;
    return BOIDS_OK;
}

void boids_mlp_destroy(boids_mlp *m)
{
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->st) cudaStreamSynchronize(m->st);
    free_acts(m);
    void *q[] = {m->p, m->grad, m->m, m->v, m->p16, m->loss, m->w2img};
    for (void *p : q)
        if (p) cudaFree(p);
    if (m->err) cudaFreeHost(m->err);
    if (m->st) cudaStreamDestroy(m->st);
    delete m;
}

int64_t boids_mlp_param_count(boids_mlp *m) { return m ? m->np : 0; }

int boids_mlp_get_params(boids_mlp *m, float *params)
{
    if (!m || !params) return fail(BOIDS_EINVAL, "boids_mlp_get_params: bad argument");
    cudaSetDevice(m->device);
    MCK(cudaMemcpyAsync(params, m->p, 4 * m->np, cudaMemcpyDeviceToHost, m->st));
    MCK(cudaStreamSynchronize(m->st));
    return BOIDS_OK;
}

int boids_mlp_set_params(boids_mlp *m, const float *params)
{
    if (!m || !params) return fail(BOIDS_EINVAL, "boids_mlp_set_params: bad argument");
    cudaSetDevice(m->device);
    MCK(cudaMemcpyAsync(m->p, params, 4 * m->np, cudaMemcpyHostToDevice, m->st));
    k_to_bf16<<<nb(m->np, 256), 256, 0, m->st>>>(m->p, m->p16, m->np);
    m->img_valid = false;
    MCK(cudaMemsetAsync(m->m, 0, 4 * m->np, m->st));
    MCK(cudaMemsetAsync(m->v, 0, 4 * m->np, m->st));
    m->step = 0;
    MCK(cudaStreamSynchronize(m->st));
    return BOIDS_OK;
}

int boids_mlp_forward(boids_mlp *m, const float *x, int32_t rows, float *y)
{
    if (!m || (!x && rows) || (!y && rows) || rows < 0) return fail(BOIDS_EINVAL, "boids_mlp_forward: bad argument");
    if (rows == 0) return BOIDS_OK;
    cudaSetDevice(m->device);
    if (int rc = ensure_rows(m, rows)) return rc;
    if (m->w2img && m->in == kTcIn && m->out == kTcOut) {
        // the fused pass: x in, y out, one kernel after the weight image
        MCK(cudaMemcpyAsync(m->x, x, sizeof(float) * (size_t)rows * m->in, cudaMemcpyHostToDevice, m->st));
        const __nv_bfloat16 *W1 = m->p16 + m->off[0], *W2 = m->p16 + m->off[2], *W3 = m->p16 + m->off[4];
        const float *b1 = m->p + m->off[1], *b2 = m->p + m->off[3], *b3 = m->p + m->off[5];
        if (!m->img_valid) {
            k_mlp_tile_w<<<nb(kTcN * kTcK / 8, 256), 256, 0, m->st>>>(W2, m->w2img);
            MCK(cudaGetLastError());
            m->img_valid = true;
        }
        const unsigned tiles = nb(rows, kTcM);
        k_mlp_forward_tc<<<tiles < m->nsm ? tiles : m->nsm, kTcFwdThreads, kTcFwdSmem, m->st>>>(
            m->x, rows, W1, b1, m->w2img, b2, W3, b3, m->y, m->err);
    } else {
        if (int rc = upload_rows(m, x, nullptr, rows)) return rc;
        forward(m, rows, false);  // inference: the backward pass's pre-activations are not needed
    }
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(y, m->y, sizeof(float) * (size_t)rows * m->out, cudaMemcpyDeviceToHost, m->st));
    return finish_call(m);
}

int boids_mlp_gradient(boids_mlp *m, const float *x, const float *t, int32_t rows, float *grad, double *loss)
{
    if (!m || !x || !t || !grad || rows <= 0) return fail(BOIDS_EINVAL, "boids_mlp_gradient: bad argument");
    cudaSetDevice(m->device);
    if (int rc = ensure_rows(m, rows)) return rc;
    MCK(cudaMemsetAsync(m->loss, 0, 8, m->st));
    if (batch_is_fused(m)) {
        MCK(cudaMemcpyAsync(m->x, x, sizeof(float) * (size_t)rows * m->in, cudaMemcpyHostToDevice, m->st));
        MCK(cudaMemcpyAsync(m->t, t, sizeof(float) * (size_t)rows * m->out, cudaMemcpyHostToDevice, m->st));
        fused_batch(m, m->x, m->t, nullptr, rows, AdamArgs{});
    } else {
        if (int rc = upload_rows(m, x, t, rows)) return rc;
        forward(m, rows);
        backward(m, rows);
    }
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(grad, m->grad, 4 * m->np, cudaMemcpyDeviceToHost, m->st));
    double l = 0;
    MCK(cudaMemcpyAsync(&l, m->loss, 8, cudaMemcpyDeviceToHost, m->st));
    const int rc = finish_call(m);
    if (loss) *loss = l;
    return rc;
}

int boids_mlp_train(boids_mlp *m, const float *x, const float *t, int32_t rows, int32_t epochs, int32_t batch,
                    float lr, uint64_t shuffle_seed, double *last_epoch_loss)
{
    if (!m || !x || !t || rows <= 0 || epochs < 0 || batch <= 0)
        return fail(BOIDS_EINVAL, "boids_mlp_train: bad argument");
    cudaSetDevice(m->device);
    if (batch > rows) batch = rows;
    m->img_valid = false;  // every batch lays its own out, and ends with other parameters
    if (int rc = ensure_rows(m, rows + batch)) return rc;
    // the whole set stays resident: rows [0, rows) of x/t
    float *X = m->x, *T = m->t;
    const bool fused = batch_is_fused(m);
    int *d_idx = nullptr;
    float *bx = nullptr, *bt = nullptr;  // a gathered batch (the fused one gathers for itself)
    // An epoch's order lies in one of two host arrays, and its copy may read the
    // array as late as the stream comes to it: `sent` says when it has, and the
    // array is rewritten after that.  With two, an epoch's order is drawn and
    // queued while the last one's is still waiting to be sent.
    std::vector<int> order[2] = {std::vector<int>(rows), std::vector<int>(rows)};
    cudaEvent_t sent[2] = {nullptr, nullptr};
    auto release = [&]() {
        for (cudaEvent_t ev : sent)
            if (ev) cudaEventDestroy(ev);
        cudaFree(d_idx);
        cudaFree(bx);
        cudaFree(bt);
    };
    if (cudaMalloc(&d_idx, sizeof(int) * rows) != cudaSuccess ||
        (!fused && (cudaMalloc(&bx, sizeof(float) * (size_t)batch * m->in) != cudaSuccess ||
                    cudaMalloc(&bt, sizeof(float) * (size_t)batch * m->out) != cudaSuccess))) {
        cudaGetLastError();
        release();
        return fail(BOIDS_ENOMEM, "boids_mlp_train: cudaMalloc failed");
    }
    for (int i = 0; i < rows; ++i) order[1][i] = i;
    uint64_t s = shuffle_seed;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    double epoch_loss = 0.0;
    int rc = 0;
    float *keep_x = m->x, *keep_t = m->t;
    if (cudaEventCreateWithFlags(&sent[0], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&sent[1], cudaEventDisableTiming) != cudaSuccess ||
        cudaMemcpyAsync(X, x, sizeof(float) * (size_t)rows * m->in, cudaMemcpyHostToDevice, m->st) != cudaSuccess ||
        cudaMemcpyAsync(T, t, sizeof(float) * (size_t)rows * m->out, cudaMemcpyHostToDevice, m->st) != cudaSuccess)
        rc = fail(BOIDS_ECUDA, "boids_mlp_train: copy failed");
    for (int ep = 0; ep < epochs && !rc; ++ep) {
        std::vector<int> &idx = order[ep & 1];
        if (ep >= 2 && cudaEventSynchronize(sent[ep & 1]) != cudaSuccess) {
            rc = fail(BOIDS_ECUDA, std::string("boids_mlp_train: ") + cudaGetErrorString(cudaGetLastError()));
            break;
        }
        idx = order[(ep + 1) & 1];  // the last epoch's order, shuffled on
        for (int i = rows - 1; i > 0; --i) {  // Fisher-Yates
            s += 0x9e3779b97f4a7c15ULL;
            uint64_t z = s;
            z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
            z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
            z ^= z >> 31;
            const int j = (int)(z % (uint64_t)(i + 1));
            std::swap(idx[i], idx[j]);
        }
        if (cudaMemcpyAsync(d_idx, idx.data(), sizeof(int) * rows, cudaMemcpyHostToDevice, m->st) != cudaSuccess ||
            cudaEventRecord(sent[ep & 1], m->st) != cudaSuccess ||
            cudaMemsetAsync(m->loss, 0, 8, m->st) != cudaSuccess) {
            rc = fail(BOIDS_ECUDA, "boids_mlp_train: copy failed");
            break;
        }
        int nbatch = 0;
        for (int b0 = 0; b0 < rows; b0 += batch, ++nbatch) {
            const int r = std::min(batch, rows - b0);
            ++m->step;
            const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
            if (fused) {
                fused_batch(m, X, T, d_idx + b0, r, AdamArgs{m->m, m->v, lr, b1, b2, c1, c2, eps});
                continue;
            }
            k_gather_rows<<<nb((long long)r * m->in, 256), 256, 0, m->st>>>(keep_x, d_idx + b0, r, m->in, bx);
            k_gather_rows<<<nb((long long)r * m->out, 256), 256, 0, m->st>>>(keep_t, d_idx + b0, r, m->out, bt);
            // the forward/backward buffers read x/t from m->x/m->t: point them at the batch
            m->x = bx;
            m->t = bt;
            k_to_bf16<<<nb((long long)r * m->in, 256), 256, 0, m->st>>>(bx, m->x16, (long long)r * m->in);
            forward(m, r);
            backward(m, r);
            m->x = keep_x;
            m->t = keep_t;
            k_mlp_adam<<<nb(m->np, 256), 256, 0, m->st>>>(m->p, m->grad, m->m, m->v, m->p16, m->np, lr, b1, b2, c1,
                                                         c2, eps);
        }
        if (ep + 1 < epochs) continue;  // the next epoch's indices follow on the stream
        double l = 0;
        if (cudaMemcpyAsync(&l, m->loss, 8, cudaMemcpyDeviceToHost, m->st) != cudaSuccess ||
            cudaStreamSynchronize(m->st) != cudaSuccess) {
            rc = fail(BOIDS_ECUDA, std::string("boids_mlp_train: ") + cudaGetErrorString(cudaGetLastError()));
            break;
        }
        epoch_loss = l / nbatch;
    }
    if (!rc && cudaGetLastError() != cudaSuccess) rc = fail(BOIDS_ECUDA, "boids_mlp_train: kernel launch failed");
    if (!rc) rc = finish_call(m);
    else cudaStreamSynchronize(m->st);  // no copy reads the caller's rows or the orders after the call
    release();
    if (last_epoch_loss) *last_epoch_loss = epoch_loss;
    return rc;
}

}  // extern "C"
