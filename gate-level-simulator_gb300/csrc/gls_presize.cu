// Learned presize: per-gate features, MLP inference on the tensor cores
// (tcgen05, BF16 operands, FP32 accumulation in tensor memory) with an FP32
// CUDA-core twin, and FP32 training kernels (GEMM, Huber loss, Adam).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cstdint>
#include "gls_presize.h"

namespace gls {

// ------------------------------------------------------------- features
// Expected output changes (est) and probability of a 1 (pone) of a gate output
// of M input nets, from their lengths and 1-probabilities and its truth table
// over their values; unrolled, so that nothing is looked up in memory.
template <int M>
__device__ __forceinline__ void sensitized(const uint4 &t, const float *len, const float *p1, float &est, float &pone)
{
    uint32_t F[1 << M];
#pragma unroll
    for (uint32_t b = 0; b < (1u << M); ++b)
        F[b] = (((b & 4u) ? t.w : t.x) >> (((b & 1u) ? 6u : 0u) + ((b & 2u) ? 24u : 0u))) & 3u;
#pragma unroll
    for (uint32_t b = 0; b < (1u << M); ++b) {
        float w = 1.f;
#pragma unroll
        for (int j = 0; j < M; ++j) w *= ((b >> j) & 1u) ? p1[j] : 1.f - p1[j];
        if (F[b] == kV1) pone += w;
#pragma unroll
        for (int j = 0; j < M; ++j) {
            if ((b >> j) & 1u) continue;
            if (F[b | (1u << j)] != F[b]) {
                float wo = 1.f;   // probability of the other inputs' values
#pragma unroll
                for (int i = 0; i < M; ++i)
                    if (i != j) wo *= ((b >> i) & 1u) ? p1[i] : 1.f - p1[i];
                est += wo * len[j];
            }
        }
    }
}

// Row of a gate output: its static features (cell, pins, delays, fan-out,
// truth-table sensitivity) with the input-net entries filled from the
// lengths of its input nets' change lists.
__device__ __forceinline__ void gate_features(const PresizeArgs &a, uint32_t r, float x[kIn])
{
    if (a.rows) {
#pragma unroll
        for (int k = 0; k < kIn; ++k) x[k] = a.rows[(uint64_t)r * kIn + k];
        return;
    }
    const uint32_t d = a.lo + r;
    const float4 *fs = reinterpret_cast<const float4 *>(a.feat_static + (uint64_t)d * kIn);
#pragma unroll
    for (int q = 0; q < kIn / 4; ++q) {
        const float4 v = __ldg(fs + q);
        x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
    }
    const DrvMeta &md = a.meta[d];
    float sum = 0.f, mx = 0.f, mn = 0.f, len[kMaxSlots], p1[kMaxSlots];
#pragma unroll
    for (int j = 0; j < kMaxSlots; ++j) {
        float l = 0.f, q = 0.5f;
        if (j < md.m) {
            const uint32_t net = md.net[j];
            const uint32_t n_ev = a.net_len[net];
            l = n_ev == 0xFFFFFFFFu ? 0.f : (float)n_ev;
            sum += l;
            mx = fmaxf(mx, l);
            mn = j == 0 ? l : fminf(mn, l);
            // share of the window the net spends at 1 (of its time at 0 or 1)
            const unsigned long long t0 = a.saif[3ull * net], t1 = a.saif[3ull * net + 1];
            if (t0 != ~0ull && t0 + t1 > 0) q = (float)((double)t1 / (double)(t0 + t1));
        }
        len[j] = l;
        p1[j] = q;
        if (j < 3) x[15 + j] = log1pf(l) * (1.f / 12.f);
    }
    x[18] = log1pf(sum) * (1.f / 12.f);
    x[19] = log1pf(mx) * (1.f / 12.f);
    x[20] = log1pf(mn) * (1.f / 12.f);
    // expected output changes with independent inputs: every input change
    // passes when the other inputs sensitize the output to it (the Boolean
    // difference of the truth table, weighted by their 1-probabilities)
    const uint8_t *lut = a.lut + md.lut_off;
    const int m = md.m;
    float est = 0.f, pone = 0.f, pmean = 0.f;
    const uint4 t = __ldg(a.slut + d);   // of up to three input nets
    if (m == 1) sensitized<1>(t, len, p1, est, pone);
    else if (m == 2) sensitized<2>(t, len, p1, est, pone);
    else if (m == 3) sensitized<3>(t, len, p1, est, pone);
    else
    for (uint32_t b = 0; b < (1u << m); ++b) {
        uint32_t idx = 0;
        for (int p = 0; p < md.n_pins; ++p)
            idx |= (((b >> ((md.pin_slot >> (3 * p)) & 7u)) & 1u) ? 3u : 0u) << (2 * p);
        const uint32_t F = __ldg(lut + idx);
        float w = 1.f;
        for (int j = 0; j < m; ++j) w *= ((b >> j) & 1u) ? p1[j] : 1.f - p1[j];
        if (F == kV1) pone += w;
        for (int j = 0; j < m; ++j) {
            if ((b >> j) & 1u) continue;
            uint32_t idx2 = 0;
            const uint32_t b2 = b | (1u << j);
            for (int p = 0; p < md.n_pins; ++p)
                idx2 |= (((b2 >> ((md.pin_slot >> (3 * p)) & 7u)) & 1u) ? 3u : 0u) << (2 * p);
            if (__ldg(lut + idx2) != F) {
                float wo = 1.f;   // probability of the other inputs' values
                for (int i = 0; i < m; ++i)
                    if (i != j) wo *= ((b >> i) & 1u) ? p1[i] : 1.f - p1[i];
                est += wo * len[j];
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kMaxSlots; ++j)
        if (j < m) pmean += p1[j];
    x[21] = log1pf(est) * (1.f / 12.f);
    x[22] = pone;
    x[23] = m ? pmean / m : 0.f;
}

__device__ __forceinline__ uint32_t reserve_of(const PresizeArgs &a, float y)
{
    const float len = expm1f(fminf(fmaxf(y, 0.f), 30.f)) * (1.f + a.margin);
    const float r = ceilf(len) + (float)a.slack;
    return r >= 4.0e9f ? 0xFFFFFFF0u : (uint32_t)r;
}

// the window's own buffers when the rows are gate outputs of a batch of windows
__device__ __forceinline__ PresizeArgs for_window(const PresizeArgs &a)
{
    PresizeArgs b = a;
    if (a.wv) {
        const WinDev &w = a.wv[blockIdx.y];
        b.net_len = w.net_len;
        b.saif = w.saif;
        b.pred = w.pred;
        b.err = w.err;
    }
    return b;
}

__global__ void __launch_bounds__(256) k_features(PresizeArgs a, float *out)
{
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n) return;
    float x[kIn];
    gate_features(a, r, x);
#pragma unroll
    for (int k = 0; k < kIn; ++k) out[(uint64_t)r * kIn + k] = x[k];
}

// ------------------------------------------------ FP32 CUDA-core inference
// One thread per row; the FP32 weights sit in shared memory.
__global__ void __launch_bounds__(128) k_presize_f32(PresizeArgs a0)
{
    const PresizeArgs a = for_window(a0);
    extern __shared__ float sp[];
    for (uint32_t k = threadIdx.x; k < (uint32_t)kParams; k += blockDim.x) sp[k] = a.params[k];
    __syncthreads();
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n) return;
    float x[kIn], h1[kHid];
    gate_features(a, r, x);
#pragma unroll 4
    for (int u = 0; u < kHid; ++u) {
        float z = sp[kOffB1 + u];
#pragma unroll
        for (int k = 0; k < kIn; ++k) z = fmaf(sp[kOffW1 + u * kIn + k], x[k], z);
        h1[u] = fmaxf(z, 0.f);
    }
    float y = sp[kOffB3];
    for (int u = 0; u < kHid; ++u) {
        float z = sp[kOffB2 + u];
#pragma unroll
        for (int v = 0; v < kHid; ++v) z = fmaf(sp[kOffW2 + u * kHid + v], h1[v], z);
        y = fmaf(sp[kOffW3 + u], fmaxf(z, 0.f), y);
    }
    if (a.y) a.y[r] = y;
    if (a.pred) a.pred[r] = reserve_of(a, y);
}

// -------------------------------------------------- tcgen05 inference
// One CTA of 128 threads per 128 rows: thread t builds row t's features and
// owns row t of both accumulators.  Layer 1 (128 x 32 by 32 x 128) and
// layer 2 (128 x 128 by 128 x 128) are tcgen05.mma kind::f16 with BF16
// operands in shared memory and the FP32 accumulator in tensor memory
// (128 lanes x 128 columns); the 128 -> 1 output layer runs on the CUDA
// cores from the tcgen05.ld of layer 2.
constexpr uint32_t kSmA1 = 0, kSmB1 = 8192, kSmB2 = kSmB1 + kImgW2, kSmA2 = kSmB1 + kImgBytes,
                   kSmBar = kSmA2 + kHid * kHid * 2, kSmTotal = kSmBar + 64;
static_assert(kSmB2 == 16384 && kSmA2 == 49152, "tensor-core kernel shared-memory map");
// instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A
// and B (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kHid >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kWaitSpins = 1u << 20;

// shared-memory matrix descriptor: start address, leading (K-direction) and
// stride (8-row-group) byte offsets, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem), "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// bounded wait on an mbarrier phase: false after kWaitSpins polls
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t it = 0; it < kWaitSpins; ++it) {
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

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__global__ void __launch_bounds__(128, 1) k_presize_tc(PresizeArgs a0)
{
    const PresizeArgs a = for_window(a0);
    extern __shared__ __align__(1024) uint8_t sm[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t bar = sbase + kSmBar, tslot = sbase + kSmBar + 8;
    // weights: the prepared BF16 image goes to B1 | B2 unchanged
    {
        uint4 *dst = reinterpret_cast<uint4 *>(sm + kSmB1);
        for (uint32_t k = tid; k < kImgBytes / 16; k += 128) dst[k] = __ldg(a.img + k);
    }
    if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tslot), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // launched while the level before still runs, whose lists the features are
    // made of.  The level's gate outputs wait for the end of this kernel: their
    // blocks stay on an SM for the whole level, and next to this kernel's
    // shared memory they have little L1 (75.8 instead of 67.7 ms on the 2 M
    // cell design; launched one after the other 69.7).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // A1: this thread's feature row in BF16, 16 bytes per 8 features
    const uint32_t r = blockIdx.x * 128 + tid;
    {
        float x[kIn];
        if (r < a.n) gate_features(a, r, x);
        else {
#pragma unroll
            for (int k = 0; k < kIn; ++k) x[k] = 0.f;
        }
#pragma unroll
        for (int k8 = 0; k8 < kIn / 8; ++k8) {
            uint4 q;
            q.x = pack_bf16(x[8 * k8 + 0], x[8 * k8 + 1]);
            q.y = pack_bf16(x[8 * k8 + 2], x[8 * k8 + 3]);
            q.z = pack_bf16(x[8 * k8 + 4], x[8 * k8 + 5]);
            q.w = pack_bf16(x[8 * k8 + 6], x[8 * k8 + 7]);
            *reinterpret_cast<uint4 *>(sm + kSmA1 + canon_off(tid, 8 * k8, kIn)) = q;
        }
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(sm + kSmBar + 8);
    const uint32_t trow = tmem + ((warp * 32u) << 16);   // this warp's 32 lanes
    // layer 1: K = 32 in two K-steps of 16
    if (tid == 0) {
#pragma unroll
        for (uint32_t ks = 0; ks < kIn / 16; ++ks)
            mma_bf16(tmem, smem_desc(sbase + kSmA1 + ks * 256, 128, (kIn / 8) * 128),
                     smem_desc(sbase + kSmB1 + ks * 256, 128, (kIn / 8) * 128), ks);
        mma_commit(bar);
    }
    bool ok = __syncthreads_and(mbar_wait(bar, 0));
    fence_after();
    if (ok) {
        // hidden layer 1 = ReLU(acc + b1) -> A2 in BF16
#pragma unroll 1
        for (uint32_t c = 0; c < kHid / 32; ++c) {
            float v[32];
            tmem_ld32(trow + c * 32, v);
#pragma unroll
            for (int j8 = 0; j8 < 4; ++j8) {
                float h[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int col = c * 32 + j8 * 8 + j;
                    h[j] = fmaxf(v[j8 * 8 + j] + __ldg(a.params + kOffB1 + col), 0.f);
                }
                uint4 q;
                q.x = pack_bf16(h[0], h[1]);
                q.y = pack_bf16(h[2], h[3]);
                q.z = pack_bf16(h[4], h[5]);
                q.w = pack_bf16(h[6], h[7]);
                *reinterpret_cast<uint4 *>(sm + kSmA2 + canon_off(tid, c * 32 + j8 * 8, kHid)) = q;
            }
        }
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    // layer 2: K = 128 in eight K-steps, accumulator columns reused
    if (ok && tid == 0) {
#pragma unroll
        for (uint32_t ks = 0; ks < kHid / 16; ++ks)
            mma_bf16(tmem, smem_desc(sbase + kSmA2 + ks * 256, 128, (kHid / 8) * 128),
                     smem_desc(sbase + kSmB2 + ks * 256, 128, (kHid / 8) * 128), ks);
        mma_commit(bar);
    }
    if (ok) ok = __syncthreads_and(mbar_wait(bar, 1));
    fence_after();
    if (ok) {
        float y = __ldg(a.params + kOffB3);
#pragma unroll 1
        for (uint32_t c = 0; c < kHid / 32; ++c) {
            float v[32];
            tmem_ld32(trow + c * 32, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const int col = c * 32 + j;
                y = fmaf(__ldg(a.params + kOffW3 + col), fmaxf(v[j] + __ldg(a.params + kOffB2 + col), 0.f), y);
            }
        }
        if (r < a.n) {
            if (a.y) a.y[r] = y;
            if (a.pred) a.pred[r] = reserve_of(a, y);
        }
    } else if (tid == 0) {
        atomicOr(a.err, 1u);
    }
    fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

void launch_features(const PresizeArgs &a, float *out, cudaStream_t st)
{
    if (!a.n) return;
    k_features<<<(a.n + 255) / 256, 256, 0, st>>>(a, out);
}

// the dynamic shared-memory limits of both inference kernels (the current
// device; called before any launch and outside stream capture)
void prepare_presize_kernels()
{
    cudaFuncSetAttribute(k_presize_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmTotal);
    cudaFuncSetAttribute(k_presize_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kParams * 4));
}

void launch_presize(const PresizeArgs &a, bool tensor_cores, cudaStream_t st)
{
    if (!a.n) return;
    const dim3 grid((a.n + 127) / 128, a.wv ? a.nwin : 1);
    if (tensor_cores) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = grid;
        lc.blockDim = dim3(128);
        lc.dynamicSmemBytes = kSmTotal;
        lc.stream = st;
        lc.attrs = &at;
        lc.numAttrs = 1;
        cudaLaunchKernelEx(&lc, k_presize_tc, a);
    } else k_presize_f32<<<grid, 128, kParams * 4, st>>>(a);
}

// ------------------------------------------------------------- training
// k_mlp_grad: loss and gradient over a minibatch in one launch.  A block takes
// 64 rows at a time and keeps the weights and the rows' activations in shared
// memory: both forward layers, the loss, and the backward products; its parts
// of the weight gradients stay in registers over all its rows and reach one of
// eight copies of the gradient (cleared before) by one round of atomics; the
// copies are summed in 64 bits (k_sum_copies).  Block b adds to copy b % 8:
// FP32 atomics of many blocks on one copy round more (8,192 rows, a call, and
// the largest error against 64 bits relative to the largest entry: one copy 88
// us, 3.7e-7; 64-bit atomics 116 us, 4.8e-8; eight copies 77 us, 5.8e-8; the
// separate launches before 429 us, 2.5e-7).
//
// What bounds it: latency at two warps a scheduler.  8,192 rows take 52 us of a
// call of 78 (launches, read-back), 14 at the peak FP32 rate of their 114 kFLOP
// each; the FMA pipe is busy 23 % of the cycles, issue 38 % of those with work,
// and of 5.3 cycles between a warp's instructions 1.7 wait for memory and .6
// for the queue of the atomics at the end.  254 registers a thread (the parts
// of the gradient) leave no room for more warps.  Fifteen launches over
// activations in HBM, with 4 x 4 outputs a thread, took 430 us a call.  Eight
// warps of eight rows each: a warp's lanes
// share the row operand (broadcast reads), 4 columns a lane make 32 FMAs for
// every three 16-byte reads; row strides of 4 more floats than a multiple of
// 32 keep the 16-byte reads down a column free of bank conflicts.
constexpr int kRows = 64;
constexpr int kCopies = 8, kCopy = kParams + 1;   // a copy: the gradient and the loss sum
constexpr int kLdX = kIn + 4, kLdH = kHid + 4;
struct GradSmem {
    float w1[kHid * kLdX], w2[kHid * kLdH];
    float x[kRows * kLdX];
    float h[kRows * kLdH];   // hidden layer 1, then its gradient
    float d[kRows * kLdH];   // gradient at hidden layer 2
};

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void fma4(float &acc, const float4 &a, const float4 &b)
{
    acc = fmaf(a.x, b.x, acc);
    acc = fmaf(a.y, b.y, acc);
    acc = fmaf(a.z, b.z, acc);
    acc = fmaf(a.w, b.w, acc);
}

// rows first .. first + nb - 1 of the data, or (mul != 0) rows (mul * (first + i) + add) mod n
__global__ void __launch_bounds__(256, 1) k_mlp_grad(int nb, uint64_t first, uint64_t mul, uint64_t add, uint64_t n,
                                                     const float *__restrict__ X, const float *__restrict__ T,
                                                     const float *__restrict__ P, float huber, float scale,
                                                     float *__restrict__ G)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    GradSmem &sm = *reinterpret_cast<GradSmem *>(s_raw);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, r0 = ty * 8;
    G += (blockIdx.x % kCopies) * kCopy;
    for (int q = tid; q < kHid * kIn; q += 256) sm.w1[(q / kIn) * kLdX + q % kIn] = P[kOffW1 + q];
    for (int q = tid; q < kHid * kHid; q += 256) sm.w2[(q / kHid) * kLdH + q % kHid] = P[kOffW2 + q];
    float b1[4], b2[4], w3[4];   // columns tx + 32 c
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        b1[c] = P[kOffB1 + tx + 32 * c];
        b2[c] = P[kOffB2 + tx + 32 * c];
        w3[c] = P[kOffW3 + tx + 32 * c];
    }
    const float b3 = P[kOffB3];
    // this thread's part of the gradient: w2 rows u0 .. u0 + 7, columns k0 and
    // 64 + k0 (4 each); w1 rows j0, columns x0 (4 each)
    const int u0 = (tid >> 4) * 8, k0 = (tid & 15) * 4, j0 = (tid >> 3) * 4, x0 = (tid & 7) * 4;
    float gw2[8][8] = {}, gw1[4][4] = {}, gw3[4] = {}, gb2[4] = {}, gb1[4] = {}, gb3 = 0.f, ls = 0.f;
    const int tiles = (nb + kRows - 1) / kRows;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();   // the weights are there; the tile before is done with x and h
        const int base = tile * kRows;
        for (int q = tid; q < kRows * kIn; q += 256) {
            const int i = q / kIn, k = q % kIn;
            float v = 0.f;
            if (base + i < nb) {
                const uint64_t at = first + base + i;
                const uint64_t row = mul ? (uint64_t)(((unsigned __int128)mul * at + add) % n) : at;
                v = X[row * kIn + k];
            }
            sm.x[i * kLdX + k] = v;
        }
        float t = 0.f;   // lanes 0 .. 7: the target of row r0 + lane
        if (tx < 8 && base + r0 + tx < nb) {
            const uint64_t at = first + base + r0 + tx;
            t = T[mul ? (uint64_t)(((unsigned __int128)mul * at + add) % n) : at];
        }
        __syncthreads();
        // forward, layer 1: rows r0 .. r0 + 7, columns tx + 32 c
        float acc[8][4] = {};
#pragma unroll
        for (int k = 0; k < kIn; k += 4) {
            float4 bv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) bv[c] = ld4(&sm.w1[(tx + 32 * c) * kLdX + k]);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 av = ld4(&sm.x[(r0 + r) * kLdX + k]);
#pragma unroll
                for (int c = 0; c < 4; ++c) fma4(acc[r][c], av, bv[c]);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                sm.h[(r0 + r) * kLdH + tx + 32 * c] = fmaxf(acc[r][c] + b1[c], 0.f);
                acc[r][c] = 0.f;
            }
        __syncwarp();   // a warp reads its own rows only
        // layer 2
#pragma unroll 2
        for (int k = 0; k < kHid; k += 4) {
            float4 bv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) bv[c] = ld4(&sm.w2[(tx + 32 * c) * kLdH + k]);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 av = ld4(&sm.h[(r0 + r) * kLdH + k]);
#pragma unroll
                for (int c = 0; c < 4; ++c) fma4(acc[r][c], av, bv[c]);
            }
        }
        // output, loss and the gradient at layer 2
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            float y = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                acc[r][c] += b2[c];
                y = fmaf(fmaxf(acc[r][c], 0.f), w3[c], y);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            const float res = y + b3 - __shfl_sync(0xffffffffu, t, r), ab = fabsf(res);
            const bool in = ab <= huber, valid = base + r0 + r < nb;
            const float dy = valid ? scale * (in ? res : copysignf(huber, res)) : 0.f;
            if (valid && tx == 0) {
                ls += in ? 0.5f * res * res : huber * (ab - 0.5f * huber);
                gb3 += dy;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float z = acc[r][c], dz = z > 0.f ? dy * w3[c] : 0.f;
                gw3[c] = fmaf(fmaxf(z, 0.f), dy, gw3[c]);
                gb2[c] += dz;
                sm.d[(r0 + r) * kLdH + tx + 32 * c] = dz;
                acc[r][c] = 0.f;
            }
        }
        __syncthreads();
        // gradient at layer 1: rows r0 .. r0 + 7, columns 4 tx + c
#pragma unroll 2
        for (int u = 0; u < kHid; u += 4) {
            float4 bv[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) bv[q] = ld4(&sm.w2[(u + q) * kLdH + 4 * tx]);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 av = ld4(&sm.d[(r0 + r) * kLdH + u]);
                const float a4[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    acc[r][0] = fmaf(a4[q], bv[q].x, acc[r][0]);
                    acc[r][1] = fmaf(a4[q], bv[q].y, acc[r][1]);
                    acc[r][2] = fmaf(a4[q], bv[q].z, acc[r][2]);
                    acc[r][3] = fmaf(a4[q], bv[q].w, acc[r][3]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float4 h = ld4(&sm.h[(r0 + r) * kLdH + 4 * tx]);
            acc[r][0] = h.x > 0.f ? acc[r][0] : 0.f;
            acc[r][1] = h.y > 0.f ? acc[r][1] : 0.f;
            acc[r][2] = h.z > 0.f ? acc[r][2] : 0.f;
            acc[r][3] = h.w > 0.f ? acc[r][3] : 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) gb1[c] += acc[r][c];
        }
        // weight gradient of layer 2
#pragma unroll 2
        for (int i = 0; i < kRows; ++i) {
            const float4 da = ld4(&sm.d[i * kLdH + u0]), db = ld4(&sm.d[i * kLdH + u0 + 4]);
            const float4 ha = ld4(&sm.h[i * kLdH + k0]), hb = ld4(&sm.h[i * kLdH + 64 + k0]);
            const float dv[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
            const float hv[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int p = 0; p < 8; ++p)
#pragma unroll
                for (int q = 0; q < 8; ++q) gw2[p][q] = fmaf(dv[p], hv[q], gw2[p][q]);
        }
        __syncthreads();   // hidden layer 1 is read
#pragma unroll
        for (int r = 0; r < 8; ++r)
            *reinterpret_cast<float4 *>(&sm.h[(r0 + r) * kLdH + 4 * tx]) =
                make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        __syncthreads();
        // weight gradient of layer 1
#pragma unroll 4
        for (int i = 0; i < kRows; ++i) {
            const float4 d = ld4(&sm.h[i * kLdH + j0]), v = ld4(&sm.x[i * kLdX + x0]);
            const float dv[4] = {d.x, d.y, d.z, d.w}, xv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) gw1[p][q] = fmaf(dv[p], xv[q], gw1[p][q]);
        }
    }
#pragma unroll
    for (int p = 0; p < 8; ++p)
#pragma unroll
        for (int q = 0; q < 8; ++q)
            atomicAdd(G + kOffW2 + (u0 + p) * kHid + (q < 4 ? k0 + q : 60 + k0 + q), gw2[p][q]);
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) atomicAdd(G + kOffW1 + (j0 + p) * kIn + x0 + q, gw1[p][q]);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        atomicAdd(G + kOffW3 + tx + 32 * c, gw3[c]);
        atomicAdd(G + kOffB2 + tx + 32 * c, gb2[c]);
        atomicAdd(G + kOffB1 + 4 * tx + c, gb1[c]);
    }
    if (tx == 0) {
        atomicAdd(G + kOffB3, gb3);
        atomicAdd(G + kParams, ls);
    }
}

__device__ __forceinline__ float sum_copies(const float *__restrict__ g, int k)
{
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < kCopies; ++c) s += g[c * kCopy + k];
    return (float)s;
}

__global__ void __launch_bounds__(256) k_sum_copies(const float *__restrict__ g, float *__restrict__ out)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kCopy) out[k] = sum_copies(g, k);
}

// loss: the epoch's loss sum, which the minibatch's is added to
__global__ void __launch_bounds__(256) k_adam(int P, float *__restrict__ p, const float *__restrict__ g,
                                              float *__restrict__ m, float *__restrict__ v, float lr, float c1,
                                              float c2, double *loss)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == P) *loss += (double)sum_copies(g, P);
    if (k >= P) return;
    const float gk = sum_copies(g, k);
    const float mk = 0.9f * m[k] + 0.1f * gk, vk = 0.999f * v[k] + 0.001f * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk * c1) / (sqrtf(vk * c2) + 1e-8f);
}

}  // namespace gls

// =============================================================== host side
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "gls_ctx.h"

using namespace gls;

namespace {

// round-to-nearest-even float -> bfloat16 bits
uint16_t to_bf16(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7FFFFFFFu) > 0x7F800000u) return 0x7FC0;
    return (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}

// the BF16 weight image the tensor-core kernel copies to shared memory
std::vector<uint8_t> weight_image(const float *params)
{
    std::vector<uint8_t> img(kImgBytes, 0);
    for (uint32_t n = 0; n < (uint32_t)kHid; ++n) {
        for (uint32_t k = 0; k < (uint32_t)kIn; ++k) {
            const uint16_t b = to_bf16(params[kOffW1 + n * kIn + k]);
            std::memcpy(&img[kImgW1 + canon_off(n, k, kIn)], &b, 2);
        }
        for (uint32_t k = 0; k < (uint32_t)kHid; ++k) {
            const uint16_t b = to_bf16(params[kOffW2 + n * kHid + k]);
            std::memcpy(&img[kImgW2 + canon_off(n, k, kHid)], &b, 2);
        }
    }
    return img;
}

int setf(std::string *err, int code, const char *msg, cudaError_t e = cudaSuccess)
{
    if (err) *err = e == cudaSuccess ? std::string(msg) : std::string(msg) + ": " + cudaGetErrorString(e);
    return code;
}

}  // namespace

// ------------------------------------------------------------- trainer
struct gls_trainer {
    int device = 0;
    cudaStream_t st = nullptr;
    std::string err;
    uint64_t n = 0, seed = 0, adam_t = 0;
    int sm_count = 1;
    DevBuf X, T, P, G, Mo, Vo;
    PinBuf host;
    DevBuf sum;   // an epoch's loss sum; a gradient's entries and loss
};

namespace {

// Loss sum and gradient over nb rows (see k_mlp_grad) into the copies of G
void tr_step_grad(gls_trainer *tr, int nb, uint64_t first, uint64_t mul, uint64_t add, float huber)
{
    cudaMemsetAsync(tr->G.p, 0, (size_t)kCopies * kCopy * 4, tr->st);
    const int tiles = (nb + kRows - 1) / kRows;
    k_mlp_grad<<<std::min(tiles, tr->sm_count), 256, sizeof(GradSmem), tr->st>>>(
        nb, first, mul, add, tr->n, tr->X.as<float>(), tr->T.as<float>(), tr->P.as<float>(), huber, 1.f / nb,
        tr->G.as<float>());
}

uint64_t splitmix(uint64_t &s)
{
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

uint64_t gcd64(uint64_t a, uint64_t b)
{
    while (b) {
        const uint64_t t = a % b;
        a = b;
        b = t;
    }
    return a;
}

}  // namespace

extern "C" int gls_trainer_create(int device, uint64_t seed, gls_trainer **out)
{
    if (!out) return GLS_EINVAL;
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return GLS_ECUDA;
    gls_trainer *tr = new gls_trainer;
    tr->device = device;
    tr->seed = seed;
    cudaError_t e = cudaStreamCreateWithFlags(&tr->st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = tr->P.ensure(kParams * 4);
    if (e == cudaSuccess) e = tr->G.ensure(kCopies * kCopy * 4);
    if (e == cudaSuccess) e = tr->sum.ensure(kCopy * 4 + 16);
    if (e == cudaSuccess) e = tr->Mo.ensure(kParams * 4);
    if (e == cudaSuccess) e = tr->Vo.ensure(kParams * 4);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&tr->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem));
    if (e != cudaSuccess) {
        delete tr;
        return GLS_ECUDA;
    }
    // He-uniform initialization from the seed
    std::vector<float> p(kParams, 0.f);
    uint64_t s = seed;
    auto uni = [&](float lim) { return (float)(((splitmix(s) >> 11) * 0x1.0p-53) * 2.0 - 1.0) * lim; };
    for (int k = 0; k < kHid * kIn; ++k) p[kOffW1 + k] = uni(std::sqrt(6.f / kIn));
    for (int k = 0; k < kHid * kHid; ++k) p[kOffW2 + k] = uni(std::sqrt(6.f / kHid));
    for (int k = 0; k < kHid; ++k) p[kOffW3 + k] = uni(std::sqrt(6.f / kHid)) * 0.1f;
    cudaMemcpy(tr->P.p, p.data(), kParams * 4, cudaMemcpyHostToDevice);
    cudaMemset(tr->Mo.p, 0, kParams * 4);
    cudaMemset(tr->Vo.p, 0, kParams * 4);
    *out = tr;
    return GLS_OK;
}

extern "C" int gls_trainer_destroy(gls_trainer *tr)
{
    if (!tr) return GLS_OK;
    cudaSetDevice(tr->device);
    DevBuf *all[] = {&tr->X, &tr->T, &tr->P, &tr->G, &tr->Mo, &tr->Vo, &tr->sum};
    for (DevBuf *b : all) b->release();
    tr->host.release();
    if (tr->st) cudaStreamDestroy(tr->st);
    delete tr;
    return GLS_OK;
}

extern "C" const char *gls_trainer_error(const gls_trainer *tr) { return tr ? tr->err.c_str() : "null trainer"; }

extern "C" int gls_trainer_set_data(gls_trainer *tr, const float *feat, const float *target, uint64_t n)
{
    if (!tr || !feat || !target || !n) return GLS_EINVAL;
    cudaSetDevice(tr->device);
    cudaError_t e = tr->X.ensure(n * kIn * 4);
    if (e == cudaSuccess) e = tr->T.ensure(n * 4);
    if (e != cudaSuccess) return setf(&tr->err, GLS_ENOMEM, "training data", e);
    e = cudaMemcpy(tr->X.p, feat, n * kIn * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(tr->T.p, target, n * 4, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return setf(&tr->err, GLS_ECUDA, "upload training data", e);
    tr->n = n;
    // start the output bias at the mean target
    double mean = 0.0;
    for (uint64_t i = 0; i < n; ++i) mean += target[i];
    const float b3 = (float)(mean / (double)n);
    cudaMemcpy(tr->P.as<float>() + kOffB3, &b3, 4, cudaMemcpyHostToDevice);
    return GLS_OK;
}

extern "C" int gls_trainer_fit(gls_trainer *tr, const gls_train_opts *o, float *loss)
{
    if (!tr || !o || !o->batch || !tr->n) return GLS_EINVAL;
    cudaSetDevice(tr->device);
    const uint32_t nb_max = (uint32_t)std::min<uint64_t>(o->batch, tr->n);
    uint64_t s = o->seed ^ 0x5DEECE66Dull;
    for (uint32_t ep = 0; ep < o->epochs; ++ep) {
        // a fresh pseudo-random permutation of the rows every epoch
        uint64_t mul = splitmix(s) % tr->n;
        if (mul == 0) mul = 1;
        while (gcd64(mul, tr->n) != 1) mul = mul + 1 < tr->n ? mul + 1 : 1;
        const uint64_t add = splitmix(s) % tr->n;
        cudaMemsetAsync(tr->sum.p, 0, 8, tr->st);
        for (uint64_t b0 = 0; b0 < tr->n; b0 += nb_max) {
            const int nb = (int)std::min<uint64_t>(nb_max, tr->n - b0);
            tr_step_grad(tr, nb, b0, mul, add, o->huber);
            ++tr->adam_t;
            const float c1 = 1.f / (1.f - std::pow(0.9f, (float)tr->adam_t));
            const float c2 = 1.f / (1.f - std::pow(0.999f, (float)tr->adam_t));
            k_adam<<<kParams / 256 + 1, 256, 0, tr->st>>>(kParams, tr->P.as<float>(), tr->G.as<float>(),
                                                          tr->Mo.as<float>(), tr->Vo.as<float>(), o->lr, c1, c2,
                                                          tr->sum.as<double>());
        }
        double ls = 0.0;
        cudaMemcpyAsync(&ls, tr->sum.p, 8, cudaMemcpyDeviceToHost, tr->st);
        const cudaError_t e = cudaStreamSynchronize(tr->st);
        if (e != cudaSuccess) return setf(&tr->err, GLS_ECUDA, "training step", e);
        if (loss) loss[ep] = (float)(ls / (double)tr->n);
    }
    return GLS_OK;
}

extern "C" int gls_trainer_grad(gls_trainer *tr, uint64_t first, uint64_t n, float huber, float *grad, float *loss)
{
    if (!tr || !grad || !n || first + n > tr->n || n > 0x7FFFFFFFull) return GLS_EINVAL;
    cudaSetDevice(tr->device);
    tr_step_grad(tr, (int)n, first, 0, 0, huber);
    k_sum_copies<<<kCopy / 256 + 1, 256, 0, tr->st>>>(tr->G.as<float>(), tr->sum.as<float>());
    // the gradient and the loss sum behind it in one copy, through page-locked
    // memory kept with the trainer
    cudaError_t e = cudaSuccess;
    if (!tr->host.ensure(kCopy * 4)) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(tr->host.p, tr->sum.p, kCopy * 4, cudaMemcpyDeviceToHost, tr->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(tr->st);
    if (e != cudaSuccess) return setf(&tr->err, GLS_ECUDA, "gradient", e);
    std::memcpy(grad, tr->host.p, kParams * 4);
    const float ls = tr->host.as<float>()[kParams];
    if (loss) *loss = ls / (float)n;
    return GLS_OK;
}

extern "C" int gls_trainer_get_params(gls_trainer *tr, float *params)
{
    if (!tr || !params) return GLS_EINVAL;
    cudaSetDevice(tr->device);
    return cudaMemcpy(params, tr->P.p, kParams * 4, cudaMemcpyDeviceToHost) == cudaSuccess ? GLS_OK : GLS_ECUDA;
}

extern "C" int gls_trainer_set_params(gls_trainer *tr, const float *params)
{
    if (!tr || !params) return GLS_EINVAL;
    cudaSetDevice(tr->device);
    if (cudaMemcpy(tr->P.p, params, kParams * 4, cudaMemcpyHostToDevice) != cudaSuccess) return GLS_ECUDA;
    cudaMemset(tr->Mo.p, 0, kParams * 4);
    cudaMemset(tr->Vo.p, 0, kParams * 4);
    tr->adam_t = 0;
    return GLS_OK;
}

// ------------------------------------------------- context-side presize
extern "C" int gls_set_presize_model(gls_ctx *ctx, const gls_presize_model *m)
{
    if (!ctx || !m) return GLS_EINVAL;
    if (!(m->margin >= 0.f) || m->margin > 100.f) return ctx_fail(ctx, GLS_EINVAL, "presize margin out of range");
    for (int k = 0; k < kParams; ++k)
        if (!std::isfinite(m->params[k])) return ctx_fail(ctx, GLS_EINVAL, "presize parameter %d is not finite", k);
    cudaSetDevice(ctx->opts.device);
    const std::vector<uint8_t> img = weight_image(m->params);
    cudaError_t e = ctx->mlp_params.ensure(kParams * 4);
    if (e == cudaSuccess) e = ctx->mlp_img.ensure(kImgBytes);
    if (e == cudaSuccess) e = ctx->aux.ensure(64);
    if (e == cudaSuccess) e = cudaMemcpy(ctx->mlp_params.p, m->params, kParams * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(ctx->mlp_img.p, img.data(), kImgBytes, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ECUDA, "upload presize model: %s", cudaGetErrorString(e));
    ctx->margin = m->margin;
    ctx->slack = m->slack;
    ctx->have_model = true;
    ctx_drop_graphs(ctx);
    prepare_presize_kernels();
    return GLS_OK;
}

void ctx_presize_args(const gls_ctx *ctx, PresizeArgs *a)
{
    std::memset(a, 0, sizeof *a);
    a->feat_static = ctx->feat_static.as<float>();
    a->meta = ctx->meta.as<DrvMeta>();
    a->lut = ctx->lut.as<uint8_t>();
    a->slut = ctx->slut.as<uint4>();
    a->params = ctx->mlp_params.as<float>();
    a->img = ctx->mlp_img.as<uint4>();
    a->margin = ctx->margin;
    a->slack = ctx->slack;
}

extern "C" int gls_presize_samples(gls_ctx *ctx, uint32_t window, float *feat, uint32_t *count, uint64_t cap,
                                   uint64_t *n)
{
    if (!ctx || !n) return GLS_EINVAL;
    if (!ctx->loaded) return ctx_fail(ctx, GLS_ESTATE, "presize_samples before load_netlist");
    if (window >= ctx->windows.size() || !ctx->windows[window]->done)
        return ctx_fail(ctx, GLS_ESTATE, "presize_samples: window %u has not run", window);
    *n = ctx->n_drv;
    if (!feat || !count) return GLS_OK;
    if (cap < ctx->n_drv) return ctx_fail(ctx, GLS_EINVAL, "presize_samples: room for %llu rows, %u needed",
                                          (unsigned long long)cap, ctx->n_drv);
    cudaSetDevice(ctx->opts.device);
    Window *w = ctx->windows[window];
    PresizeArgs a;
    ctx_presize_args(ctx, &a);
    a.net_len = w->net_len.as<uint32_t>();
    a.saif = w->saif.as<unsigned long long>();
    a.lo = 0;
    a.n = ctx->n_drv;
    DevBuf out;
    cudaError_t e = out.ensure((size_t)ctx->n_drv * kIn * 4);
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ENOMEM, "presize_samples: %s", cudaGetErrorString(e));
    launch_features(a, out.as<float>(), ctx->stream);
    e = cudaMemcpyAsync(feat, out.p, (size_t)ctx->n_drv * kIn * 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    out.release();
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ECUDA, "presize_samples: %s", cudaGetErrorString(e));
    // output lengths in driver order
    std::vector<uint32_t> len(ctx->n_nets);
    e = cudaMemcpy(len.data(), w->net_len.p, (size_t)ctx->n_nets * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ECUDA, "presize_samples: %s", cudaGetErrorString(e));
    std::vector<DrvMeta> meta(ctx->n_drv);
    e = cudaMemcpy(meta.data(), ctx->meta.p, (size_t)ctx->n_drv * sizeof(DrvMeta), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ECUDA, "presize_samples: %s", cudaGetErrorString(e));
    for (uint32_t d = 0; d < ctx->n_drv; ++d) count[d] = len[meta[d].out_net];
    return GLS_OK;
}

extern "C" int gls_presize_predict(gls_ctx *ctx, const gls_presize_model *m, const float *feat, uint64_t n, float *y,
                                   int tensor_cores)
{
    if (!ctx || !m || !feat || !y || !n || n > 0x7FFFFFFFull) return GLS_EINVAL;
    cudaSetDevice(ctx->opts.device);
    const std::vector<uint8_t> img = weight_image(m->params);
    DevBuf prm, im, rows, out, er;
    cudaError_t e = prm.ensure(kParams * 4);
    if (e == cudaSuccess) e = im.ensure(kImgBytes);
    if (e == cudaSuccess) e = rows.ensure(n * kIn * 4);
    if (e == cudaSuccess) e = out.ensure(n * 4);
    if (e == cudaSuccess) e = er.ensure(16);
    if (e == cudaSuccess) e = cudaMemcpy(prm.p, m->params, kParams * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(im.p, img.data(), kImgBytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(rows.p, feat, n * kIn * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(er.p, 0, 16);
    prepare_presize_kernels();
    uint32_t flag = 0;
    if (e == cudaSuccess) {
        PresizeArgs a;
        std::memset(&a, 0, sizeof a);
        a.rows = rows.as<float>();
        a.n = (uint32_t)n;
        a.params = prm.as<float>();
        a.img = im.as<uint4>();
        a.y = out.as<float>();
        a.err = er.as<uint32_t>();
        launch_presize(a, tensor_cores != 0, ctx->stream);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(y, out.p, n * 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, er.p, 4, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    prm.release(); im.release(); rows.release(); out.release(); er.release();
    if (e != cudaSuccess) return ctx_fail(ctx, GLS_ECUDA, "presize_predict: %s", cudaGetErrorString(e));
    if (flag) return ctx_fail(ctx, GLS_ECUDA, "presize_predict: tensor-core kernel timed out waiting for its MMA");
    return GLS_OK;
}
