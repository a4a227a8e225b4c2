// sphmp_mlp.cu — the learned large-step corrector's network on the tensor cores:
// a per-particle MLP 48 -> 128 -> 128 -> 128 -> 4 with SiLU, bf16 weights and
// activations, FP32 accumulation in TMEM (tcgen05.mma kind::f16), its backward
// pass and Adam.
//
// * k_mlp_forward: all four layers of 128-particle tiles in one persistent
//   kernel, four tiles in flight per CTA. The weights stay in shared memory;
//   each layer is one chain of MMAs
//   into TMEM, and its epilogue (bias, SiLU, bf16) writes the next layer's
//   operand tile back into shared memory.
// * k_mlp_train: forward and backward pass of a batch in one persistent kernel, one
//   CTA per SM over 128-row tiles: the layer inputs stay in shared memory and the
//   pre-activations in registers from the forward half of a tile to its backward
//   half, the transposes are taken by the operand descriptors (MN-major), and the
//   weight and bias gradients accumulate in TMEM over the CTA's tiles;
//   k_sum_partials adds the CTAs' partial gradients in a fixed order.
// * k_gemm_tn: D = A B^T for K-major bf16 A [M][K] and B [N][K] (N <= 128),
//   M in tiles of 128, K split over gridDim.y into FP32 partials (the library's
//   GEMM entry point).
// * elementwise kernels: the loss, the sum of the partial gradients with the Adam
//   step, and the packing of the FP32 master parameters into the padded bf16
//   operand layouts.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "sphmp_mlp.h"
#include "sphmp_tc.cuh"

namespace sphmp {
namespace mlp {

using bf16 = __nv_bfloat16;

namespace {

__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float silu_grad(float z) {
    const float s = __fdividef(1.f, 1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ---------------------------------------------------------------------------
// Fused forward
// ---------------------------------------------------------------------------

constexpr int kGroups = 4;                     // tiles in flight per CTA, at most
constexpr int kFwdThreads = 1024;              // 32 warps, shared equally by the groups
constexpr int kTile = 128;
// dynamic shared memory of the forward kernel
constexpr int kOffW1 = 0;                                  // [128 rows][48] kc 48
constexpr int kOffW2 = kOffW1 + kHidden * kFeatures * 2;   // [128][128]
constexpr int kOffW3 = kOffW2 + kHidden * kHidden * 2;     // [128][128]
constexpr int kOffW4 = kOffW3 + kHidden * kHidden * 2;     // [16][128]
constexpr int kOffAct = kOffW4 + kOutPad * kHidden * 2;    // kGroups x [128][128] operand tiles
constexpr int kActBytes = kTile * kHidden * 2;
constexpr int kOffBias = kOffAct + kGroups * kActBytes;    // 3 * 128 + 16 floats
constexpr int kOffNorm = kOffBias + (3 * kHidden + kOutPad) * 4;  // shift[48], scale[48]
constexpr int kFwdSmem = kOffNorm + 2 * kFeatures * 4;
// TMEM: group g uses columns [128 g, 128 g + 128) for layers 1-3 and the first
// 16 of them again for layer 4 (after layer 3's epilogue has read them). With one
// CTA per SM the allocation always takes every column.
constexpr uint32_t kGroupTmemCols = 128;
constexpr uint32_t kFwdTmemCols = kGroups * kGroupTmemCols;
static_assert(kFwdTmemCols <= 512, "TMEM holds 512 columns");
static_assert(kFwdSmem > 116 * 1024, "one CTA per SM: the TMEM allocation takes every column");
static_assert(kFwdSmem <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void cp_async16(uint8_t* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A read-only 16-byte load that stays where it is written (an ordinary one sinks down
// to its use, past the waits that it should overlap).
__device__ __forceinline__ float4 load_early(const float4* p) {
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// The first kc columns of weights [rows][stride] as a K-major tile (16-byte copies in
// flight together; the caller commits and waits).
__device__ __forceinline__ void stage_weights(uint8_t* dst, const bf16* src, int rows, int kc, int stride, int tid,
                                              int nthreads) {
    for (int q = tid; q < rows * (kc / 8); q += nthreads) {
        const int r = q / (kc / 8), k = (q % (kc / 8)) * 8;
        cp_async16(dst + tc::kmajor_offset(r, k, kc), src + (size_t)r * stride + k);
    }
}

// one MMA chain: D[tmem_col ...] = act (K = kc) x W^T (N rows)
__device__ __forceinline__ void issue_layer(uint32_t tmem, uint32_t act, uint32_t w, int kc, int n, uint64_t* bar) {
    const uint32_t idesc = tc::idesc_bf16_f32(kTile, n);
    for (int ks = 0; ks < kc / 16; ks++)
        tc::mma_bf16(tmem, tc::kmajor_desc(act, kc, ks), tc::kmajor_desc(w, kc, ks), idesc, ks > 0 ? 1u : 0u);
    tc::mma_commit(bar);
}

// Every thread of the CTA waits; the CTA agrees on the outcome (a barrier).
__device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t& parity) {
    const bool ok = tc::mbar_wait(bar, parity, tc::kWaitLimitNs);
    parity ^= 1u;
    const bool all = __syncthreads_and(ok) != 0;
    tc::fence_after_sync();
    return all;
}

// shared-memory writes of this thread done: order them before the next MMA
__device__ __forceinline__ void handoff_to_mma() {
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
}

// The same for the T threads of one tile group (named barrier 1 + g).
template <int T>
__device__ __forceinline__ void group_sync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(T) : "memory");
}
template <int T>
__device__ __forceinline__ bool group_all(int g, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(1 + g), "n"(T)
        : "memory");
    return r != 0;
}
template <int T>
__device__ __forceinline__ bool group_wait(uint64_t* bar, uint32_t& parity, int g) {
    const bool ok = tc::mbar_wait(bar, parity, tc::kWaitLimitNs);
    parity ^= 1u;
    const bool all = group_all<T>(g, ok);
    tc::fence_after_sync();
    return all;
}
template <int T>
__device__ __forceinline__ void group_handoff(int g) {
    tc::fence_async_smem();
    tc::fence_before_sync();
    group_sync<T>(g);
}

// SiLU of 16 columns (c0 on) of a hidden layer's accumulator row, the bf16
// activations into the operand tile (row r, K = 128); z (FP16) into zs if wanted.
// SiLU is z/2 (1 + tanh(z/2)) with the hardware tanh (tanh.approx.f32, relative
// error about 2^-11, below the bf16 rounding of the result): one special-function
// operation per element instead of two (exp and reciprocal). hb = bias / 2: z/2 is
// then one multiply-add (exactly half of the rounded z).
template <bool SAVE>
__device__ __forceinline__ void silu16(const uint32_t (&v)[16], int c0, const float* hb, uint8_t* act, int r,
                                       uint32_t* zs) {
    const float2 half = make_float2(0.5f, 0.5f);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int c = c0 + 8 * q;
        const float4 b[2] = {*reinterpret_cast<const float4*>(hb + c), *reinterpret_cast<const float4*>(hb + c + 4)};
        uint32_t hw[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 bb = i & 1 ? make_float2(b[i >> 1].z, b[i >> 1].w) : make_float2(b[i >> 1].x, b[i >> 1].y);
            const float2 a = make_float2(__uint_as_float(v[8 * q + 2 * i]), __uint_as_float(v[8 * q + 2 * i + 1]));
            const float2 hz = __ffma2_rn(a, half, bb);
            const float2 h = __ffma2_rn(hz, make_float2(tanh_approx(hz.x), tanh_approx(hz.y)), hz);
            hw[i] = pack2(h.x, h.y);
            if (SAVE) {
                const float2 z = __fadd2_rn(hz, hz);
                const __half2 zz = __floats2half2_rn(z.x, z.y);
                zs[4 * q + i] = *reinterpret_cast<const uint32_t*>(&zz);
            }
        }
        *reinterpret_cast<uint4*>(act + tc::kmajor_offset(r, c, kHidden)) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    }
}

// NC columns from c0 on, the accumulator's next 16 loading while the last 16 are
// processed.
template <int NC>
__device__ __forceinline__ void hidden_epilogue(uint32_t tmem, int warp, int c0, const float* hb, uint8_t* act, int r) {
    uint32_t va[16], vb[16];
    tc::tmem_issue16(tc::tmem_lane_addr(tmem, warp, c0), va);
#pragma unroll
    for (int c = 0; c < NC; c += 32) {
        tc::tmem_wait16(va);
        if (c + 16 < NC) tc::tmem_issue16(tc::tmem_lane_addr(tmem, warp, c0 + c + 16), vb);
        silu16<false>(va, c0 + c, hb, act, r, nullptr);
        if (c + 16 < NC) {
            tc::tmem_wait16(vb);
            if (c + 32 < NC) tc::tmem_issue16(tc::tmem_lane_addr(tmem, warp, c0 + c + 32), va);
            silu16<false>(vb, c0 + c + 16, hb, act, r, nullptr);
        }
    }
}

// The input tile of rows [row0, row0 + 128) by T threads: normalised features,
// bf16 (K = 48). Four lanes a row, so that a warp's load touches eight contiguous
// pieces of 64 bytes.
template <int T>
struct InputTile {
    static constexpr int kRows = T / 4, kPasses = kTile / kRows;
    static_assert(kRows * kPasses == kTile, "whole passes");
    float4 f[kPasses][3];
    __device__ __forceinline__ void load(const float* __restrict__ x, int row0, int n, int gt) {
#pragma unroll
        for (int p = 0; p < kPasses; p++) {
            const int grow = row0 + (gt >> 2) + p * kRows;
            const float4* src = reinterpret_cast<const float4*>(x + (size_t)(grow < n ? grow : 0) * kFeatures) + (gt & 3);
#pragma unroll
            for (int m = 0; m < 3; m++) f[p][m] = load_early(src + 4 * m);
        }
    }
    __device__ __forceinline__ void store(int row0, int n, const float* fshift, const float* fscale, uint8_t* act,
                                          int gt) const {
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const int c = 4 * ((gt & 3) + 4 * m);
            const float4 sh = *reinterpret_cast<const float4*>(fshift + c);
            const float4 sc = *reinterpret_cast<const float4*>(fscale + c);
#pragma unroll
            for (int p = 0; p < kPasses; p++) {
                const int r = (gt >> 2) + p * kRows;
                const float4 a = f[p][m];
                uint2 q;
                q.x = pack2((a.x - sh.x) * sc.x, (a.y - sh.y) * sc.y);
                q.y = pack2((a.z - sh.z) * sc.z, (a.w - sh.w) * sc.w);
                if (row0 + r >= n) q = make_uint2(0u, 0u);
                *reinterpret_cast<uint2*>(act + tc::kmajor_offset(r, c, kFeatures)) = q;
            }
        }
    }
};

// Biases (halved for the hidden layers) and normalisation into shared memory.
__device__ __forceinline__ void stage_constants(const Packed& W, float* bias, float* norm, int tid, int nthreads) {
    for (int i = tid; i < 3 * kHidden + kOutPad; i += nthreads) bias[i] = (i < 3 * kHidden ? 0.5f : 1.f) * W.bias[i];
    for (int i = tid; i < kFeatures; i += nthreads) {
        norm[i] = W.fshift[i];
        norm[kFeatures + i] = W.fscale[i];
    }
}

// kGroups independent tile pipelines per CTA (8 warps each), so that one group's
// epilogue runs while the others' MMAs and loads are in flight; the weights in
// shared memory are shared. The warps of a group split each epilogue by lane
// quadrant and by columns. Few tiles are spread over the CTAs first.
// Bound: one tanh per hidden activation, 16 a clock and SM (76 us per million rows,
// 55 % of the time), beside the chain of a tile (its load, four MMAs and three
// epilogues). A million rows: 139 us; 204 us with 4 warps a group, a thread reading
// whole rows of features and no load of the accumulators beside the arithmetic.
// Up to 128 rows: 11 us and 14 us (32 or 16 warps a tile instead of 8 change nothing).
__global__ void __launch_bounds__(kFwdThreads, 1) k_mlp_forward(const float* __restrict__ x, int n,
                                                                 const Packed W, float* __restrict__ y,
                                                                 uint32_t* err) {
    constexpr int T = kFwdThreads / kGroups;  // threads of a group
    constexpr int NC = kHidden / (T / 128);   // epilogue columns of a warp
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bars[kGroups];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int g = tid / T, gt = tid % T;
    const int r = gt & 127, c0 = (gt >> 7) * NC;  // this thread's row and first column
    uint8_t* act = smem + kOffAct + g * kActBytes;
    float* bias = reinterpret_cast<float*>(smem + kOffBias);
    float* norm = reinterpret_cast<float*>(smem + kOffNorm);

    stage_weights(smem + kOffW1, W.w1, kHidden, kFeatures, kInPad, tid, kFwdThreads);
    stage_weights(smem + kOffW2, W.w2, kHidden, kHidden, kHidden, tid, kFwdThreads);
    stage_weights(smem + kOffW3, W.w3, kHidden, kHidden, kHidden, tid, kFwdThreads);
    stage_weights(smem + kOffW4, W.w4, kOutPad, kHidden, kHidden, tid, kFwdThreads);
    cp_async_commit();
    stage_constants(W, bias, norm, tid, kFwdThreads);
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, kFwdTmemCols);
        tc::tmem_relinquish();
    }
    if (tid == 0)
        for (int k = 0; k < kGroups; k++) tc::mbar_init(&bars[k], 1);
    cp_async_wait<0>();
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base + (uint32_t)g * kGroupTmemCols;
    const uint32_t a_act = tc::smem_addr(act);
    uint64_t* bar = &bars[g];
    uint32_t parity = 0;
    bool ok = true;
    const int ntiles = (n + kTile - 1) / kTile;
    for (int t = g * gridDim.x + blockIdx.x; t < ntiles && ok; t += kGroups * gridDim.x) {
        const int row0 = t * kTile;
        {
            InputTile<T> in;
            in.load(x, row0, n, gt);
            in.store(row0, n, norm, norm + kFeatures, act, gt);
        }
        group_handoff<T>(g);
        // layer 1
        if (gt == 0) {
            tc::fence_after_sync();
            issue_layer(tmem, a_act, tc::smem_addr(smem + kOffW1), kFeatures, kHidden, bar);
        }
        if (!(ok = group_wait<T>(bar, parity, g))) break;
        hidden_epilogue<NC>(tmem, warp, c0, bias, act, r);
        group_handoff<T>(g);
        // layer 2
        if (gt == 0) {
            tc::fence_after_sync();
            issue_layer(tmem, a_act, tc::smem_addr(smem + kOffW2), kHidden, kHidden, bar);
        }
        if (!(ok = group_wait<T>(bar, parity, g))) break;
        hidden_epilogue<NC>(tmem, warp, c0, bias + kHidden, act, r);
        group_handoff<T>(g);
        // layer 3
        if (gt == 0) {
            tc::fence_after_sync();
            issue_layer(tmem, a_act, tc::smem_addr(smem + kOffW3), kHidden, kHidden, bar);
        }
        if (!(ok = group_wait<T>(bar, parity, g))) break;
        hidden_epilogue<NC>(tmem, warp, c0, bias + 2 * kHidden, act, r);
        group_handoff<T>(g);
        // layer 4 (N = 16: outputs 0..3 and zero padding)
        if (gt == 0) {
            tc::fence_after_sync();
            issue_layer(tmem, a_act, tc::smem_addr(smem + kOffW4), kHidden, kOutPad, bar);
        }
        if (!(ok = group_wait<T>(bar, parity, g))) break;
        if (gt < kTile) {
            float v[16];
            tc::tmem_ld16(tc::tmem_lane_addr(tmem, warp, 0), v);
            const float* b4 = bias + 3 * kHidden;
            if (row0 + gt < n)
                reinterpret_cast<float4*>(y)[row0 + gt] = make_float4(v[0] + b4[0], v[1] + b4[1], v[2] + b4[2], v[3] + b4[3]);
        }
        // the accumulator reads above come before the next tile's first MMA (its handoff)
    }
    if (!ok) {
        if (gt == 0) atomicOr(err, kErrMmaTimeout);
        tc::mbar_wait(bar, parity ^ 1u, tc::kWaitLimitNs);  // the chain still in flight, bounded
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem_base, kFwdTmemCols);
}

// ---------------------------------------------------------------------------
// GEMM D = A B^T (K-major bf16 operands), split-K partials
// ---------------------------------------------------------------------------

constexpr int kGemmThreads = 128;
constexpr int kKc = 64;
// two stages of A tile + B tile (N <= 128): 64 KB, so at most 3 CTAs share an
// SM, 384 of its 512 TMEM columns at 128 each
constexpr int kStageBytes = kTile * kKc * 2 + 128 * kKc * 2;
constexpr int kGemmSmem = 2 * kStageBytes;

__global__ void __launch_bounds__(kGemmThreads) k_gemm_tn(const bf16* __restrict__ A, int lda,
                                                          const bf16* __restrict__ B, int ldb, float* __restrict__ D,
                                                          int M, int N, int K, int kper, uint32_t* err) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base;
    // two stages of (A tile, B tile): chunk c + 1 loads while chunk c's MMAs run
    auto stage_a = [&](int c) { return smem + (c & 1) * kStageBytes; };
    auto stage_b = [&](int c) { return smem + (c & 1) * kStageBytes + kTile * kKc * 2; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kTile;
    const int kb = blockIdx.y * kper, ke = min(K, kb + kper);
    const uint32_t ncols = N <= 32 ? 32u : N <= 64 ? 64u : 128u;
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, ncols);
        tc::tmem_relinquish();
    }
    if (tid == 0) tc::mbar_init(&bar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = tc::idesc_bf16_f32(kTile, N);
    auto load_chunk = [&](int k0, uint8_t* a_s, uint8_t* b_s) {
        for (int q = tid; q < kTile * (kKc / 8); q += kGemmThreads) {
            const int r = q >> 3, k = (q & 7) * 8;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (m0 + r < M && k0 + k < ke) v = *reinterpret_cast<const uint4*>(A + (size_t)(m0 + r) * lda + k0 + k);
            *reinterpret_cast<uint4*>(a_s + tc::kmajor_offset(r, k, kKc)) = v;
        }
        for (int q = tid; q < N * (kKc / 8); q += kGemmThreads) {
            const int r = q >> 3, k = (q & 7) * 8;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (k0 + k < ke) v = *reinterpret_cast<const uint4*>(B + (size_t)r * ldb + k0 + k);
            *reinterpret_cast<uint4*>(b_s + tc::kmajor_offset(r, k, kKc)) = v;
        }
    };
    uint32_t parity = 0;
    bool ok = true;
    const int nchunks = ke > kb ? (ke - kb + kKc - 1) / kKc : 0;
    if (nchunks > 0) load_chunk(kb, stage_a(0), stage_b(0));
    int chunks = 0;
    for (int c = 0; c < nchunks; c++) {
        handoff_to_mma();  // chunk c in shared memory for the tensor core
        if (tid == 0) {
            tc::fence_after_sync();
            const uint32_t a = tc::smem_addr(stage_a(c)), b = tc::smem_addr(stage_b(c));
            for (int ks = 0; ks < kKc / 16; ks++)
                tc::mma_bf16(tmem, tc::kmajor_desc(a, kKc, ks), tc::kmajor_desc(b, kKc, ks), idesc,
                             (c > 0 || ks > 0) ? 1u : 0u);
            tc::mma_commit(&bar);
        }
        // the other stage was last read by chunk c - 1's MMAs, complete since the last wait
        if (c + 1 < nchunks) load_chunk(kb + (c + 1) * kKc, stage_a(c + 1), stage_b(c + 1));
        if (!(ok = wait_all(&bar, parity))) break;
        chunks++;
    }
    const int r = warp * 32 + lane;
    float* drow = D + ((size_t)blockIdx.y * M + (m0 + r)) * N;
    if (ok) {
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tc::tmem_lane_addr(tmem, warp, c0), v);
            if (m0 + r < M) {
                // four 16-byte stores per 16 columns (N is a multiple of 16, the partials 16-byte aligned)
                float4* d4 = reinterpret_cast<float4*>(drow + c0);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    d4[q] = chunks ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    } else {
        if (tid == 0) atomicOr(err, kErrMmaTimeout);
        tc::mbar_wait(&bar, parity ^ 1u, tc::kWaitLimitNs);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem, ncols);
}

// ---------------------------------------------------------------------------
// Fused training pass: one persistent CTA per SM, 128-row tiles in turn
// ---------------------------------------------------------------------------
//
// For each tile (rows r of the batch), the forward pass
//   Z1 = H0 W1^T + b1,  H1 = SiLU(Z1),  Z2, H2, Z3, H3 likewise,  Y = H3 W4^T + b4
// and with dY = 2 (Y - T) / batch, the gradient of the mean squared output error,
//   dW4^T += H3^T dY          dH3 = dY W4
//   dZ3 = dH3 * SiLU'(Z3)     dW3 += dZ3^T H2   db3 += sum_r dZ3   dH2 = dZ3 W3   (Z kept in FP16)
//   dZ2 = dH2 * SiLU'(Z2)     dW2 += dZ2^T H1   db2 += sum_r dZ2   dH1 = dZ2 W2
//   dZ1 = dH1 * SiLU'(Z1)     dW1 += dZ1^T H0   db1 += sum_r dZ1
// Nothing of a tile but its rows of x and T comes from memory and nothing goes
// there: the layer inputs H stay in shared memory, Z in registers (each thread's
// row and 32 columns of three layers: 48 registers), and the weight and bias
// gradients accumulate in TMEM over all tiles of the CTA (the bias sums as MMAs
// against a tile of ones); Z or dH of the current layer lives in the first 128
// columns. Every operand is in shared memory once, without swizzling, and its
// transpose is the same tile read MN-major. The batch is a multiple of 128 rows
// (no tails). Warp w handles rows 32 (w % 4) .. + 31 (its TMEM lane quadrant) and
// columns 32 (w / 4) .. + 31 of every epilogue.
// Bound: the chain of a tile, seven GEMMs each with an epilogue after it (one special-
// function operation an element forward, two backward, 16 a clock and SM). In the
// backward half dH is issued and committed first and the weight gradients' MMAs
// run beside the epilogue, which writes dZ elsewhere than they read: dZ3 into a tile of
// its own, dZ2 over H3, dZ1 over dZ3 (MMAs complete in order, so the commit that an
// epilogue waits for covers everything before it).
// 65,536 rows (a step with the sum of the partials and Adam): 60 us; as two
// kernels that passed Z and H through memory 80 us, with transposed copies of
// H and dZ as well 145 us. 8,192 rows: 26, 37 and 87 us.
constexpr int kTrnThreads = 512;  // 16 warps: four per TMEM lane quadrant, one per column quarter
constexpr int kTHid = kTile * kHidden * 2;                    // bytes of a [128][128] tile
constexpr int kTOffW1 = 0;                                    // [128][48]   kc 48
constexpr int kTOffW2 = kTOffW1 + kHidden * kFeatures * 2;    // [128][128]  kc 128
constexpr int kTOffW3 = kTOffW2 + kHidden * kHidden * 2;      // [128][128]
constexpr int kTOffW4 = kTOffW3 + kHidden * kHidden * 2;      // [16][128]
constexpr int kTOffOnes = kTOffW4 + kOutPad * kHidden * 2;    // [16][16]    kc 16, all 1 (for every step of K)
constexpr int kTOffDy = kTOffOnes + kOutPad * 16 * 2;         // [128][16]   kc 16
constexpr int kTOffBias = kTOffDy + kTile * kOutPad * 2;
constexpr int kTOffNorm = kTOffBias + (3 * kHidden + kOutPad) * 4;
constexpr int kTOffH0 = kTOffNorm + 2 * kFeatures * 4;        // [128][48]   kc 48
constexpr int kTOffH1 = kTOffH0 + kTile * kFeatures * 2;      // [128][128]  kc 128
constexpr int kTOffH2 = kTOffH1 + kTHid;
constexpr int kTOffH3 = kTOffH2 + kTHid;                      // later dZ2
constexpr int kTOffDz = kTOffH3 + kTHid;                      // dZ3, later dZ1
constexpr int kTrnSmem = kTOffDz + kTHid;
static_assert(kTrnSmem + 256 <= 227 * 1024, "shared memory of one CTA (with the static part)");
static_assert(kTrnSmem > 116 * 1024, "one CTA per SM: the TMEM allocation takes every column");
static_assert(kTrnSmem - kTOffH1 >= kHidden * (kHidden + 4) * 4, "the partials' staging tile fits the operand tiles");
static_assert(kTOffBias % 16 == 0 && kTOffNorm % 16 == 0 && kTOffH0 % 16 == 0, "16-byte tiles");
// TMEM columns
constexpr uint32_t kTcD = 0, kTcW3 = 128, kTcW2 = 256, kTcW1 = 384, kTcW4 = 448, kTcB3 = 464, kTcB2 = 480,
                   kTcB1 = 496, kTrnTmemCols = 512;

// MMA chain D (+)= A B^T over K = 16 * ksteps; a and b give the descriptors of step ks.
template <class A, class B>
__device__ __forceinline__ void mma_chain(uint32_t d, A&& a, B&& b, int ksteps, uint32_t idesc, bool accumulate) {
    for (int ks = 0; ks < ksteps; ks++) tc::mma_bf16(d, a(ks), b(ks), idesc, (accumulate || ks > 0) ? 1u : 0u);
}

// This CTA's partial gradients, in the flat parameter layout: row r of the
// accumulators is TMEM lane r; the four warps of a lane quadrant share the
// columns. The weight blocks go through a shared-memory tile (rows padded by 4
// floats) so that the global stores are contiguous; called by every thread
// once the operand buffers are free (tile: at least 128 x 132 floats).
__device__ __forceinline__ void store_partials(uint32_t tmem, int warp, int lane, int tid, bool have,
                                                   const float* db4, float* tile, float* __restrict__ out) {
    const int r = (warp & 3) * 32 + lane;
    const int quarter = warp >> 2;
    auto block = [&](uint32_t col, int ncols, float* dst) {  // dst [128][ncols] = D[.][col .. col + ncols)
        const int ts = ncols + 4;
        for (int c0 = 16 * quarter; c0 < ncols; c0 += 64) {
            float v[16];
            if (have) tc::tmem_ld16(tc::tmem_lane_addr(tmem + col, warp, c0), v);
#pragma unroll
            for (int q = 0; q < 4; q++)
                *reinterpret_cast<float4*>(tile + r * ts + c0 + 4 * q) =
                    have ? make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3])
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        const int q4 = ncols / 4;
        for (int q = tid; q < kHidden * q4; q += kTrnThreads) {
            const int rr = q / q4, cc = (q % q4) * 4;
            *reinterpret_cast<float4*>(dst + (size_t)rr * ncols + cc) = *reinterpret_cast<const float4*>(tile + rr * ts + cc);
        }
        __syncthreads();
    };
    block(kTcW3, kHidden, out + kOffParamW3);
    block(kTcW2, kHidden, out + kOffParamW2);
    block(kTcW1, kFeatures, out + kOffParamW1);
    // W4 (D[h][o] = dW4[o][h]) and the biases: one value per row and column, contiguous across lanes
    const uint32_t col = quarter == 0 ? kTcW4 : quarter == 1 ? kTcB3 : quarter == 2 ? kTcB2 : kTcB1;
    float v[16];
    if (have) tc::tmem_ld16(tc::tmem_lane_addr(tmem + col, warp, 0), v);
    if (quarter == 0) {
#pragma unroll
        for (int o = 0; o < kOutputs; o++) out[kOffParamW4 + o * kHidden + r] = have ? v[o] : 0.f;
        if (r < kOutputs) out[kOffParamB4 + r] = db4[r];
    } else {
        out[(quarter == 1 ? kOffParamB3 : quarter == 2 ? kOffParamB2 : kOffParamB1) + r] = have ? v[0] : 0.f;
    }
}

__global__ void __launch_bounds__(kTrnThreads, 1) k_mlp_train(const float* __restrict__ x, const float* __restrict__ t,
                                                              int batch, const Packed W, float* __restrict__ part,
                                                              float* __restrict__ loss_part, uint32_t* err) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ float db4s[4][kOutputs];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = tid & 127, quarter = warp >> 2, c0 = 32 * quarter;
    const int ntiles = batch / kTile;
    float* bias = reinterpret_cast<float*>(smem + kTOffBias);
    float* norm = reinterpret_cast<float*>(smem + kTOffNorm);

    stage_weights(smem + kTOffW1, W.w1, kHidden, kFeatures, kInPad, tid, kTrnThreads);
    cp_async_commit();
    stage_weights(smem + kTOffW2, W.w2, kHidden, kHidden, kHidden, tid, kTrnThreads);
    stage_weights(smem + kTOffW3, W.w3, kHidden, kHidden, kHidden, tid, kTrnThreads);
    stage_weights(smem + kTOffW4, W.w4, kOutPad, kHidden, kHidden, tid, kTrnThreads);
    cp_async_commit();
    InputTile<kTrnThreads> in;
    in.load(x, blockIdx.x * kTile, batch, tid);
    stage_constants(W, bias, norm, tid, kTrnThreads);
    if (tid < 32)  // bf16 ones
        *reinterpret_cast<uint4*>(smem + kTOffOnes + 16 * tid) = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, kTrnTmemCols);
        tc::tmem_relinquish();
    }
    if (tid == 0) tc::mbar_init(&bar, 1);
    cp_async_wait<1>();  // W1; the others before layer 2
    handoff_to_mma();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    auto at = [&](int off) { return tc::smem_addr(smem + off); };
    constexpr int kSteps = kTile / 16;
    // operands: a tile of kc columns by rows, transposed, and the ones
    auto rows = [](uint32_t a, int kc) { return [a, kc](int ks) { return tc::kmajor_desc(a, kc, ks); }; };
    auto cols = [](uint32_t a, int kc) { return [a, kc](int ks) { return tc::mnmajor_desc(a, kc, ks); }; };
    auto ones = [&](int) { return tc::kmajor_desc(at(kTOffOnes), 16, 0); };
    float db4[kOutputs] = {0.f, 0.f, 0.f, 0.f};
    uint32_t parity = 0;
    bool ok = true, any = false;
    uint32_t z1[16], z2[16], z3[16];  // this thread's row and columns, FP16 pairs
    uint32_t v[2][16];
    auto load_d = [&]() {
        tc::tmem_issue16(tc::tmem_lane_addr(tmem + kTcD, warp, c0), v[0]);
        tc::tmem_issue16(tc::tmem_lane_addr(tmem + kTcD, warp, c0 + 16), v[1]);
        tc::tmem_wait16(v[0]);
        tc::tmem_wait16(v[1]);
    };
    // H = SiLU(Z) into the tile at off
    auto forward_epilogue = [&](const float* hb, int off, uint32_t(&z)[16]) {
        load_d();
        silu16<true>(v[0], c0, hb, smem + off, r, z);
        silu16<true>(v[1], c0 + 16, hb, smem + off, r, z + 8);
    };
    // dZ = dH * SiLU'(Z) into the tile at off
    auto backward_epilogue = [&](const uint32_t(&z)[16], int off) {
        load_d();
#pragma unroll
        for (int c = 0; c < 4; c++) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float2 zz = __half22float2(*reinterpret_cast<const __half2*>(&z[4 * c + k]));
                w[k] = pack2(__uint_as_float(v[c >> 1][8 * (c & 1) + 2 * k]) * silu_grad(zz.x),
                             __uint_as_float(v[c >> 1][8 * (c & 1) + 2 * k + 1]) * silu_grad(zz.y));
            }
            *reinterpret_cast<uint4*>(smem + off + tc::kmajor_offset(r, c0 + 8 * c, kHidden)) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
    };
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int row0 = tile * kTile;
        float4 target = make_float4(0.f, 0.f, 0.f, 0.f);
        if (quarter == 0) target = load_early(reinterpret_cast<const float4*>(t) + row0 + r);
        in.store(row0, batch, norm, norm + kFeatures, smem + kTOffH0, tid);
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            issue_layer(tmem + kTcD, at(kTOffH0), at(kTOffW1), kFeatures, kHidden, &bar);
        }
        if (!(ok = wait_all(&bar, parity))) break;
        forward_epilogue(bias, kTOffH1, z1);
        cp_async_wait<0>();
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            issue_layer(tmem + kTcD, at(kTOffH1), at(kTOffW2), kHidden, kHidden, &bar);
        }
        if (!(ok = wait_all(&bar, parity))) break;
        forward_epilogue(bias + kHidden, kTOffH2, z2);
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            issue_layer(tmem + kTcD, at(kTOffH2), at(kTOffW3), kHidden, kHidden, &bar);
        }
        if (!(ok = wait_all(&bar, parity))) break;
        forward_epilogue(bias + 2 * kHidden, kTOffH3, z3);
        handoff_to_mma();
        if (tid == 0) {  // N = 16: outputs 0..3 and zero padding
            tc::fence_after_sync();
            issue_layer(tmem + kTcD, at(kTOffH3), at(kTOffW4), kHidden, kOutPad, &bar);
        }
        if (!(ok = wait_all(&bar, parity))) break;
        if (quarter == 0) {  // dY [rows][16] (bf16, zero padded), the warp's sum of squared errors
            float o[16];
            tc::tmem_ld16(tc::tmem_lane_addr(tmem + kTcD, warp, 0), o);
            const float* b4 = bias + 3 * kHidden;
            const float d[4] = {(o[0] + b4[0]) - target.x, (o[1] + b4[1]) - target.y, (o[2] + b4[2]) - target.z,
                                (o[3] + b4[3]) - target.w};
            const float s = 2.f / (float)batch;
            const uint32_t q[2] = {pack2(s * d[0], s * d[1]), pack2(s * d[2], s * d[3])};
            *reinterpret_cast<uint4*>(smem + kTOffDy + tc::kmajor_offset(r, 0, kOutPad)) = make_uint4(q[0], q[1], 0u, 0u);
            *reinterpret_cast<uint4*>(smem + kTOffDy + tc::kmajor_offset(r, 8, kOutPad)) = make_uint4(0u, 0u, 0u, 0u);
            float se = 0.f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                se += d[k] * d[k];
                db4[k] += __bfloat162float(reinterpret_cast<const bf16*>(q)[k]);
            }
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) se += __shfl_xor_sync(0xffffffffu, se, k);
            if (lane == 0) loss_part[(row0 + r) >> 5] = se;
        }
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            mma_chain(tmem + kTcD, rows(at(kTOffDy), kOutPad), cols(at(kTOffW4), kHidden), 1,
                      tc::idesc_bf16_f32(kTile, kHidden, false, true), false);  // dH3 = dY W4
            tc::mma_commit(&bar);
            mma_chain(tmem + kTcW4, cols(at(kTOffH3), kHidden), cols(at(kTOffDy), kOutPad), kSteps,
                      tc::idesc_bf16_f32(kTile, kOutPad, true, true), any);  // dW4^T += H3^T dY
        }
        if (!(ok = wait_all(&bar, parity))) break;
        backward_epilogue(z3, kTOffDz);
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            mma_chain(tmem + kTcD, rows(at(kTOffDz), kHidden), cols(at(kTOffW3), kHidden), kSteps,
                      tc::idesc_bf16_f32(kTile, kHidden, false, true), false);  // dH2 = dZ3 W3
            tc::mma_commit(&bar);
            mma_chain(tmem + kTcW3, cols(at(kTOffDz), kHidden), cols(at(kTOffH2), kHidden), kSteps,
                      tc::idesc_bf16_f32(kTile, kHidden, true, true), any);  // dW3 += dZ3^T H2
            mma_chain(tmem + kTcB3, cols(at(kTOffDz), kHidden), ones, kSteps,
                      tc::idesc_bf16_f32(kTile, kOutPad, true, false), any);  // db3 (every column)
        }
        if (!(ok = wait_all(&bar, parity))) break;
        backward_epilogue(z2, kTOffH3);
        if (tile + (int)gridDim.x < ntiles) in.load(x, row0 + (int)gridDim.x * kTile, batch, tid);
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            mma_chain(tmem + kTcD, rows(at(kTOffH3), kHidden), cols(at(kTOffW2), kHidden), kSteps,
                      tc::idesc_bf16_f32(kTile, kHidden, false, true), false);  // dH1 = dZ2 W2
            tc::mma_commit(&bar);
            mma_chain(tmem + kTcW2, cols(at(kTOffH3), kHidden), cols(at(kTOffH1), kHidden), kSteps,
                      tc::idesc_bf16_f32(kTile, kHidden, true, true), any);  // dW2 += dZ2^T H1
            mma_chain(tmem + kTcB2, cols(at(kTOffH3), kHidden), ones, kSteps,
                      tc::idesc_bf16_f32(kTile, kOutPad, true, false), any);  // db2
        }
        if (!(ok = wait_all(&bar, parity))) break;
        backward_epilogue(z1, kTOffDz);
        handoff_to_mma();
        if (tid == 0) {
            tc::fence_after_sync();
            mma_chain(tmem + kTcW1, cols(at(kTOffDz), kHidden), cols(at(kTOffH0), kFeatures), kSteps,
                      tc::idesc_bf16_f32(kTile, kFeatures, true, true), any);  // dW1 += dZ1^T H0
            mma_chain(tmem + kTcB1, cols(at(kTOffDz), kHidden), ones, kSteps,
                      tc::idesc_bf16_f32(kTile, kOutPad, true, false), any);  // db1
            tc::mma_commit(&bar);
        }
        if (!(ok = wait_all(&bar, parity))) break;  // the tile's operands are free
        any = true;
    }
    cp_async_wait<0>();
    if (!ok) {
        if (tid == 0) atomicOr(err, kErrMmaTimeout);
        tc::mbar_wait(&bar, parity ^ 1u, tc::kWaitLimitNs);  // the chain still in flight, bounded
    }
    // db4: the sum over this CTA's rows (held by warps 0-3), in a fixed order
#pragma unroll
    for (int o = 0; o < kOutputs; o++) {
        float s = db4[o];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0 && quarter == 0) db4s[warp][o] = s;
    }
    __syncthreads();
    float db4t[kOutputs];
#pragma unroll
    for (int o = 0; o < kOutputs; o++) db4t[o] = (db4s[0][o] + db4s[1][o]) + (db4s[2][o] + db4s[3][o]);
    store_partials(tmem, warp, lane, tid, ok && any, db4t, reinterpret_cast<float*>(smem + kTOffH1),
                   part + (size_t)blockIdx.x * kParams);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem_base, kTrnTmemCols);
}

// Parameter p (flat layout) into its bf16 operand positions, as k_pack writes them.
__device__ __forceinline__ void pack_param(const PackedMut& W, int p, float val) {
    const bf16 b = __float2bfloat16_rn(val);
    if (p < kOffParamB1) {  // W1 [128][48] -> w1 [128][64]
        W.w1[(p / kFeatures) * kInPad + p % kFeatures] = b;
    } else if (p < kOffParamW2) {
        W.bias[p - kOffParamB1] = val;
    } else if (p < kOffParamB2) {
        W.w2[p - kOffParamW2] = b;
    } else if (p < kOffParamW3) {
        W.bias[kHidden + p - kOffParamB2] = val;
    } else if (p < kOffParamB3) {
        W.w3[p - kOffParamW3] = b;
    } else if (p < kOffParamW4) {
        W.bias[2 * kHidden + p - kOffParamB3] = val;
    } else if (p < kOffParamB4) {  // W4 [4][128] -> w4 [16][128]
        W.w4[p - kOffParamW4] = b;
    } else {
        W.bias[3 * kHidden + p - kOffParamB4] = val;
    }
}

// grads[p] = the sum over the CTAs' partials: 128 parameters per block, eight
// threads per four parameters summing every eighth CTA's partial (a warp reads 512
// contiguous bytes of one partial), the eight sums added in a fixed order; with an
// Adam step (adam.lr > 0) the parameter is updated in the same pass. Bound by the
// latency of reading the partials from L2 (152 of 159 KB: 24 MB), so every
// thread keeps eight 16-byte loads in flight. (With 4-byte loads, four threads per
// parameter: 10.8 us instead of 7.1.)
constexpr int kSumParams = 128, kSumSlices = 8;
static_assert(kParams % 4 == 0, "16-byte loads of the partials");
__global__ void __launch_bounds__(kSumSlices* kSumParams / 4) k_sum_partials(const float* __restrict__ part, int nparts,
                                                                             float* __restrict__ grads,
                                                                             const AdamStep adam) {
    __shared__ float4 sh[kSumSlices][kSumParams / 4];
    const int j = threadIdx.x / (kSumParams / 4), q = threadIdx.x % (kSumParams / 4);
    const int p4 = blockIdx.x * (kSumParams / 4) + q;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p4 < kParams / 4) {
        const float4* src = reinterpret_cast<const float4*>(part) + p4;
#pragma unroll 8
        for (int k = j; k < nparts; k += kSumSlices) {
            const float4 v = __ldg(src + (size_t)k * (kParams / 4));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
    sh[j][q] = s;
    __syncthreads();
    const int p = blockIdx.x * kSumParams + threadIdx.x;
    if (threadIdx.x >= kSumParams || p >= kParams) return;
    float g = 0.f;
#pragma unroll
    for (int k = 0; k < kSumSlices; k++) g += reinterpret_cast<const float*>(sh[k])[threadIdx.x];
    grads[p] = g;
    if (adam.lr > 0.f) {
        const float mi = adam.b1 * adam.m[p] + (1.f - adam.b1) * g;
        const float vi = adam.b2 * adam.v[p] + (1.f - adam.b2) * g * g;
        adam.m[p] = mi;
        adam.v[p] = vi;
        const float np = adam.p[p] - adam.lr * (mi / adam.c1) / (sqrtf(vi / adam.c2) + adam.eps);
        adam.p[p] = np;
        pack_param(adam.w, p, np);
    }
}

// ---------------------------------------------------------------------------
// Backward and optimiser helpers
// ---------------------------------------------------------------------------

// loss = sum of the partials / batch (one block, fixed order)
__global__ void k_loss_sum(const float* __restrict__ part, int nparts, int batch, float* __restrict__ loss) {
    __shared__ float red[256];
    float s = 0.f;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) s += part[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / (float)batch;
}


// FP32 master parameters -> padded bf16 operands + biases
__global__ void k_pack(const float* __restrict__ p, PackedMut W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const float* w1 = p + kOffParamW1;
    const float* w2 = p + kOffParamW2;
    const float* w3 = p + kOffParamW3;
    const float* w4 = p + kOffParamW4;
    if (i < kHidden * kInPad) {  // w1 [128][64]
        const int o = i / kInPad, k = i % kInPad;
        W.w1[i] = __float2bfloat16_rn(k < kFeatures ? w1[o * kFeatures + k] : 0.f);
    }
    if (i < kHidden * kHidden) {
        W.w2[i] = __float2bfloat16_rn(w2[i]);
        W.w3[i] = __float2bfloat16_rn(w3[i]);
    }
    if (i < kOutPad * kHidden) {  // w4 [16][128]
        const int o = i / kHidden, k = i % kHidden;
        W.w4[i] = __float2bfloat16_rn(o < kOutputs ? w4[o * kHidden + k] : 0.f);
    }
    if (i < 3 * kHidden + kOutPad) {
        float b;
        if (i < kHidden) b = p[kOffParamB1 + i];
        else if (i < 2 * kHidden) b = p[kOffParamB2 + i - kHidden];
        else if (i < 3 * kHidden) b = p[kOffParamB3 + i - 2 * kHidden];
        else b = (i - 3 * kHidden) < kOutputs ? p[kOffParamB4 + i - 3 * kHidden] : 0.f;
        W.bias[i] = b;
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

cudaError_t launch_forward(const float* x, int n, const Packed& W, float* y, uint32_t* err, int num_sms,
                           cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int tiles = (n + kTile - 1) / kTile;
    // per call (a host-side attribute of the current device): threads and devices stay independent
    cudaError_t e = cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
    if (e != cudaSuccess) return e;
    const int grid = tiles < num_sms ? tiles : num_sms;
    k_mlp_forward<<<grid, kFwdThreads, kFwdSmem, s>>>(x, n, W, y, err);
    return cudaGetLastError();
}

cudaError_t launch_gemm_tn(const bf16* A, int lda, const bf16* B, int ldb, float* D, int M, int N, int K,
                           int splits, uint32_t* err, cudaStream_t s) {
    if (M <= 0 || N <= 0 || N > 128 || (N % 16) != 0 || K < 0 || (K % 8) != 0 || splits < 1 || (lda % 8) != 0 ||
        (ldb % 8) != 0)
        return cudaErrorInvalidValue;
    int kper = (K + splits - 1) / splits;
    kper = (kper + kKc - 1) / kKc * kKc;
    if (kper == 0) kper = kKc;
    cudaError_t e = cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
    if (e != cudaSuccess) return e;
    dim3 grid((M + kTile - 1) / kTile, splits);
    k_gemm_tn<<<grid, kGemmThreads, kGemmSmem, s>>>(A, lda, B, ldb, D, M, N, K, kper, err);
    return cudaGetLastError();
}

cudaError_t launch_train(const float* x, const float* t, int batch, const Packed& W, float* part, float* loss_part,
                         float* grads, const AdamStep& adam, float* loss, uint32_t* err, int num_sms, cudaStream_t s) {
    if (batch <= 0 || batch % kTile != 0) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrnSmem);
    if (e != cudaSuccess) return e;
    const int tiles = batch / kTile;
    const int grid = tiles < num_sms ? tiles : num_sms;
    k_mlp_train<<<grid, kTrnThreads, kTrnSmem, s>>>(x, t, batch, W, part, loss_part, err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (loss) k_loss_sum<<<1, 256, 0, s>>>(loss_part, batch / 32, batch, loss);
    k_sum_partials<<<(kParams + kSumParams - 1) / kSumParams, kSumSlices * kSumParams / 4, 0, s>>>(part, grid, grads, adam);
    return cudaGetLastError();
}

AdamStep adam_step(float* p, float* m, float* v, float lr, float b1, float b2, float eps, int step,
                   const PackedMut& w) {
    return AdamStep{p, m, v, lr, b1, b2, eps, 1.f - powf(b1, (float)step), 1.f - powf(b2, (float)step), w};
}

cudaError_t launch_pack(const float* p, const PackedMut& W, cudaStream_t s) {
    k_pack<<<(kHidden * kHidden + 255) / 256, 256, 0, s>>>(p, W);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace sphmp
