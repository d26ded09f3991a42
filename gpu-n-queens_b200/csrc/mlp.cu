// Learned cost model: an MLP 112 -> 128 -> 128 -> 1 (GELU) that predicts log2 of the number
// of search nodes below a state.  Trained on the GPU by the kernels in this file (FP16
// operands, FP32 accumulation on the tensor cores; FP32 master weights, Adam), on node
// counts the batched search kernel records per item; inference (predict_kernel) runs on
// tcgen05 with the accumulator in tensor memory.  Used only to order and split the batched
// form's queue (schedule.cu); counts never depend on it.
//
// Training step on a batch of B rows (X: B x 112 fp16):
//   Z1 = X W1           H1 = gelu(Z1 + b1)      (fp16 copy of H1 feeds the next GEMM)
//   Z2 = H1 W2          H2 = gelu(Z2 + b2)
//   y  = H2 w3 + b3     loss = mean (y - t)^2
//   dy = 2 (y - t)      dZ2 = dy w3^T * gelu'(Z2 + b2)      dH1 = dZ2 W2^T
//   dZ1 = dH1 * gelu'(Z1 + b1)
//   dW2 = H1^T dZ2 / B  dW1 = X^T dZ1 / B  dw3 = H2^T dy / B  (bias grads: column sums / B)
// One kernel runs the whole step for 128 rows at a time, with every intermediate in shared or
// tensor memory (train_kernel); a second one adds up the blocks' gradients and applies Adam.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "epoch_order.h"
#include "mlp.cuh"
#include "nqb_internal.h"

namespace nqb {
namespace mlp {
namespace {

// ---- tcgen05 building blocks -----------------------------------------------------------
// Operand tiles are 128 rows x K fp16 in the 128-byte-swizzled K-major layout: 16-byte
// chunk j (8 K-elements) of row r sits at (j / 8) x 16 KB + r x 128 + ((j % 8) ^ (r % 8)) x 16
// from a 1024-byte-aligned base.  One thread issues the MMAs; the accumulator lives in
// tensor memory and each warp reads its 32 lanes back with tcgen05.ld.
constexpr int kTileRows = 128;
constexpr uint32_t kOpBytes = kTileRows * 128 * 2;  // one 128 x 128 fp16 operand tile: 32 KB
constexpr uint32_t kAtomBytes = kTileRows * 128;    // 64 K-elements (128 B) of all 128 rows: 16 KB
constexpr uint32_t kTmemCols = 128;
constexpr uint32_t kSpinLimit = 1u << 22;  // waits: far above the ~1 us a product takes
// instruction descriptor, kind::f16: D fp32 (bits 4-5 = 1), A and B fp16 and K-major,
// N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr uint32_t kIdesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ uint32_t sw128_chunk(uint32_t r, uint32_t j) {
    return (j >> 3) * kAtomBytes + r * 128u + (((j & 7u) ^ (r & 7u)) << 4);
}

// Shared-memory matrix descriptor of a 128-byte-swizzled K-major tile starting at `addr`
// (1024-byte aligned atom, or an offset of 32 bytes times the K step inside it).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu)  // start address, 16-byte units
           | ((uint64_t)1u << 16)             // leading byte offset (not used with swizzling)
           | ((uint64_t)(1024u >> 4) << 32)   // stride byte offset: 8 rows x 128 B
           | ((uint64_t)1u << 46)             // descriptor version of sm_100
           | ((uint64_t)2u << 61);            // 128-byte swizzle
}

// Byte offset of K step k (16 elements) inside an operand tile.
__device__ __forceinline__ uint32_t kstep_offset(int k) { return (uint32_t)(k >> 2) * kAtomBytes + (uint32_t)(k & 3) * 32u; }

// The same tile read the other way round (MN-major): its rows are the K index and its columns,
// contiguous in memory, the M or N index.  64 columns are one 128-byte row of an atom; the
// next 64 are kAtomBytes on (leading offset), the next 8 rows 1024 bytes (stride offset).  A K
// step of 16 rows is 2048 bytes.
__device__ __forceinline__ uint64_t sw128_desc_mn(uint32_t addr) {
    return sw128_desc(addr) - ((uint64_t)1u << 16) + ((uint64_t)(kAtomBytes >> 4) << 16);
}
constexpr uint32_t kKstepRows = 16u * 128u;
constexpr uint32_t kMnA = 1u << 15, kMnB = 1u << 16;  // instruction descriptor: A, B MN-major

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accumulate,
                                         uint32_t idesc = kIdesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(accumulate), "r"(idesc), "r"(0u));
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Bounded wait for a phase of the completion barrier.  By default mbarrier.try_wait, which
// may suspend the thread until the phase completes (no issue slots burnt while the tensor
// cores work); with probe_only, `limit` non-blocking mbarrier.test_wait probes, an exact
// count whatever the hardware's suspend time (a caller-chosen bound).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = kSpinLimit,
                                          bool probe_only = false) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t done;
        if (probe_only)
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        else
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// ---- features and fp16 weights ------------------------------------------------------------
__global__ void features_kernel(const uint4* __restrict__ st, uint64_t n_rows, __half* __restrict__ X) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_rows * kIn) return;
    X[e] = __float2half(feature(st[e / kIn], (int)(e % kIn)));
}

__global__ void to_half_kernel(const float* __restrict__ p, __half* __restrict__ w1h, __half* __restrict__ w2h) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kW1Size) w1h[i] = __float2half(p[kW1 + i]);
    if (i < kH * kH) w2h[i] = __float2half(p[kW2 + i]);
}

__device__ __forceinline__ void store_chunk(uint32_t tile, uint32_t r, uint32_t j, uint4 q) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(tile + sw128_chunk(r, j)), "r"(q.x), "r"(q.y),
                 "r"(q.z), "r"(q.w)
                 : "memory");
}

// Features 8 j .. 8 j + 7 of a state as four fp16 pairs.
__device__ __forceinline__ void feature_chunk(const uint4 s, uint32_t j, uint32_t q[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) q[e] = pack_half2(feature(s, (int)j * 8 + 2 * e), feature(s, (int)j * 8 + 2 * e + 1));
}

// ---- fused inference (tcgen05) ----------------------------------------------------------------
// A block of 16 warps runs 128-row tiles: features -> layer 1 -> GELU -> layer 2 -> GELU -> head.
// Both layers are M=128, N=128 products (K = 112 and 128) issued as K=16 tcgen05.mma by one
// thread, with FP16 operands in shared memory and the FP32 accumulator in tensor memory.
// Threads share the work as in train_kernel: row 32 quad + lane, hidden columns (and feature
// columns) 32 group .. 32 group + 31; the head's four partial sums of a row meet in shared
// memory.  H1 replaces the features in the row tile.  Every wait on the MMA completion barrier
// is bounded; on a timeout the block sets the error word and leaves, freeing its tensor memory
// on the way out.
//
// What bounds it: instruction issue (71% of the slots; ALU pipe 43%, FMA 36%, XU 34%) for the
// features and the tanh of 256 activations of each row; two blocks an SM take turns at the waits of a
// tile's chain.  300,000 rows: 119 us (190 us with 4 warps a block, each thread a whole row).
constexpr uint32_t kPredictThreads = 512;
constexpr uint32_t kPredictFloats = 3 * kH + 4 + 4 * kTileRows;  // b1 b2 w3 b3 | y partials
constexpr size_t kPredictSmem = 1024 /* alignment slack */ + 3 * kOpBytes + kPredictFloats * sizeof(float) + 16;

__global__ void __launch_bounds__(kPredictThreads, 2)
    predict_kernel(const uint4* __restrict__ st, uint32_t count, const __half* __restrict__ w1h,
                   const __half* __restrict__ w2h, const float* __restrict__ params, float* __restrict__ out,
                   uint32_t wait_limit, unsigned* __restrict__ err) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
    const uint32_t w1s = base, w2s = base + kOpBytes, xs = base + 2 * kOpBytes;
    float* const vec = reinterpret_cast<float*>(smem_raw + (base - raw) + 3 * kOpBytes);  // b1 | b2 | w3 | b3
    float* const ysum = vec + 3 * kH + 4;
    const uint32_t bar = base + 3 * kOpBytes + kPredictFloats * sizeof(float);
    const uint32_t tmem_slot = bar + 8;
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31, quad = warp & 3, group = warp >> 2;
    const uint32_t r = quad * 32 + lane, c0 = group * 32;

    for (uint32_t j = group * 4; j < group * 4 + 4; ++j) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        store_chunk(w1s, r, j, r < (uint32_t)kIn ? reinterpret_cast<const uint4*>(w1h + (size_t)r * kH)[j] : zero);
        store_chunk(w2s, r, j, reinterpret_cast<const uint4*>(w2h + (size_t)r * kH)[j]);
    }
    if (t < (uint32_t)kH) {
        vec[t] = params[kB1 + t];
        vec[kH + t] = params[kB2 + t];
        vec[2 * kH + t] = params[kW3 + t];
    }
    if (t == 0) {
        vec[3 * kH] = params[kB3];
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem = 0;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    const uint32_t mine = tmem + ((quad * 32u) << 16) + c0;
    uint32_t phase = 0;
    bool failed = false, undrained = false;

    for (uint32_t tile = blockIdx.x; (uint64_t)tile * kTileRows < count && !failed; tile += gridDim.x) {
        const uint64_t i = (uint64_t)tile * kTileRows + r;
        const uint4 s = i < count ? st[i] : make_uint4(0, 0, 0, 0);
#pragma unroll 1
        for (uint32_t e = 0; e < 4; ++e) {  // 32 of the row's features (zero for rows past the end)
            const uint32_t j = group * 4 + e;
            uint32_t q[4] = {0u, 0u, 0u, 0u};
            if (i < count) feature_chunk(s, j, q);
            store_chunk(xs, r, j, make_uint4(q[0], q[1], q[2], q[3]));
        }
        float sum = 0.0f;
        for (int layer = 0; layer < 2 && !failed; ++layer) {
            proxy_fence();  // make the operand tile visible to the tensor cores
            tc_fence_before();
            __syncthreads();
            if (t == 0) {
                tc_fence_after();
                const uint32_t wt = layer == 0 ? w1s : w2s;
                const int steps = layer == 0 ? kIn / 16 : kH / 16;
                for (int k = 0; k < steps; ++k)
                    umma_f16(tmem, sw128_desc(xs + kstep_offset(k)), sw128_desc_mn(wt + k * kKstepRows), k > 0 ? 1u : 0u,
                             kIdesc | kMnB);
                umma_commit(bar);
            }
            const bool ok = wait_limit ? mbar_wait(bar, phase, wait_limit, true) : mbar_wait(bar, phase);
            if (__syncthreads_or(!ok)) {  // timed out: drain the MMAs in flight (bounded), then leave
                undrained = !__syncthreads_and(mbar_wait(bar, phase));
                failed = true;
                break;
            }
            phase ^= 1u;
            tc_fence_after();
            const float* bias = vec + layer * kH + c0;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                float v[16];
                tmem_ld16(mine + h * 16, v);
                uint32_t q[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    q[e] = pack_half2(gelu(v[2 * e] + bias[h * 16 + 2 * e]),
                                      gelu(v[2 * e + 1] + bias[h * 16 + 2 * e + 1]));
                if (layer == 0) {  // H1 becomes the A operand of layer 2
                    store_chunk(xs, r, group * 4 + h * 2, make_uint4(q[0], q[1], q[2], q[3]));
                    store_chunk(xs, r, group * 4 + h * 2 + 1, make_uint4(q[4], q[5], q[6], q[7]));
                } else {  // head: H2 rounded to fp16 as in the training forward pass
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&q[e]));
                        const float* w3 = vec + 2 * kH + c0 + h * 16 + 2 * e;
                        sum += f.x * w3[0] + f.y * w3[1];
                    }
                }
            }
            tc_fence_before();
        }
        if (!failed) {
            ysum[group * kTileRows + r] = sum;
            __syncthreads();  // also: the operand tile and the accumulator are free for the next tile
            if (group == 0 && i < count)
                out[i] = ysum[r] + ysum[kTileRows + r] + ysum[2 * kTileRows + r] + ysum[3 * kTileRows + r] + vec[3 * kH];
        }
    }
    // bit 0: a completion wait timed out; bit 1: the drain timed out too, so products may still
    // have been in flight when the tensor memory was freed
    if (failed && t == 0) atomicOr(err, undrained ? 3u : 1u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// ---- one training step (tcgen05) ------------------------------------------------------------
// A block of 16 warps takes 128 rows of the batch through the whole step.  Thread (quad, lane,
// group): row 32 quad + lane of the tile (tensor-memory lane 32 quad + lane, which a warp may
// read only in its quad), hidden columns 32 group .. 32 group + 31.  Both weight matrices and
// the row tiles X, H1, dZ2 and H2 (then dZ1) lie in shared memory as 128 x 128 fp16 tiles,
// rows contiguous; a product reads a tile along its rows or its columns as it needs (K-major
// or MN-major), so nothing is transposed.  The accumulators have 128 tensor-memory columns
// each: Z1; Z2, then dH1; dW2 and dW1, which go on over the block's tiles.  gelu' of both
// layers stays in registers between the passes, so each activation's tanh is computed once.
// A block writes its share of every gradient to a slot of its own (GradParts) and the
// optimizer kernel adds the slots up in a fixed order: no atomics, and two runs on the same
// inputs give the same weights.
//
// What bounds it: the latency of one tile's chain of products, loads and barriers, 29 us a step at the
// default batch of 4096; its 32 blocks leave 116 SMs idle and issue in 28% of their own slots.  As 5
// GEMMs, 10 elementwise or reducing kernels and 2 gathers through global memory the step took 230 us
// on the device (two thirds of it in the GEMMs, 20-50 us each); two epochs over 65,536 samples, whole
// call: 6.75 ms before, 1.51 ms now.
constexpr uint32_t kTrainThreads = 512;
constexpr uint32_t kTrainTmem = 512;
constexpr uint32_t kTrainFloats = 3 * kH + 4 + 4 * kTileRows + kTileRows;  // b1 b2 w3 b3 | y partials | dy
constexpr size_t kTrainSmem = 1024 /* alignment slack */ + 6 * kOpBytes + kTrainFloats * sizeof(float) + 16;

// Gradients of the blocks, one slot a block; tail: {gradient of b3, squared error}.
struct GradParts {
    float *w1, *b1, *w2, *b2, *w3, *tail;
};

__device__ __forceinline__ float half_at(uint32_t tile, uint32_t r, uint32_t c) {
    unsigned short h;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(tile + sw128_chunk(r, c >> 3) + (c & 7u) * 2u));
    return __half2float(__ushort_as_half(h));
}

// gelu and its derivative at x (one tanh).
__device__ __forceinline__ void gelu_both(float x, float* h, float* g) {
    const float th = tanhf(kGeluC * (x + kGeluA * x * x * x));
    *h = 0.5f * x * (1.0f + th);
    *g = 0.5f * (1.0f + th) + 0.5f * x * (1.0f - th * th) * kGeluC * (1.0f + 3.0f * kGeluA * x * x);
}

__global__ void __launch_bounds__(kTrainThreads, 1)
    train_kernel(const __half* __restrict__ X, const float* __restrict__ target, const uint32_t* __restrict__ perm,
                 uint32_t rows, const __half* __restrict__ w1h, const __half* __restrict__ w2h,
                 const float* __restrict__ params, float inv, GradParts out, unsigned* __restrict__ err) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t w1s = base, w2s = base + kOpBytes, xs = base + 2 * kOpBytes, h1s = base + 3 * kOpBytes,
                   dz2s = base + 4 * kOpBytes, ts = base + 5 * kOpBytes;  // ts: H2, then dZ1
    float* const b1v = reinterpret_cast<float*>(smem_raw + (base - raw) + 6 * kOpBytes);
    float *const b2v = b1v + kH, *const w3v = b1v + 2 * kH, *const ysum = b1v + 3 * kH + 4, *const dyv = ysum + 4 * kTileRows;
    const uint32_t bar = base + 6 * kOpBytes + kTrainFloats * sizeof(float), tmem_slot = bar + 8;
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31, quad = warp & 3, group = warp >> 2;
    const uint32_t r = quad * 32 + lane, c0 = group * 32;
    const uint32_t col = t & 127u;  // column sums: this thread's column, over rows c0 .. c0 + 31

    for (uint32_t j = group * 4; j < group * 4 + 4; ++j) {
        const uint4 zero = make_uint4(0, 0, 0, 0);
        store_chunk(w1s, r, j, r < (uint32_t)kIn ? reinterpret_cast<const uint4*>(w1h + (size_t)r * kH)[j] : zero);
        store_chunk(w2s, r, j, reinterpret_cast<const uint4*>(w2h + (size_t)r * kH)[j]);
    }
    if (t < (uint32_t)kH) {
        b1v[t] = params[kB1 + t];
        b2v[t] = params[kB2 + t];
        w3v[t] = params[kW3 + t];
    }
    if (t == 0) {
        b1v[3 * kH] = params[kB3];
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot),
                     "r"(kTrainTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem = 0;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    const uint32_t z1t = tmem, z2t = tmem + 128, dw2t = tmem + 256, dw1t = tmem + 384;
    const uint32_t my_lanes = (quad * 32u) << 16;
    uint32_t phase = 0;
    bool failed = false, undrained = false;
    // Issues products from one thread and waits (bounded) for them; all threads call it.
    auto run = [&](auto issue) {
        proxy_fence();  // make the operand tiles visible to the tensor cores
        tc_fence_before();
        __syncthreads();
        if (t == 0) {
            tc_fence_after();
            issue();
            umma_commit(bar);
        }
        const bool ok = mbar_wait(bar, phase);
        if (__syncthreads_or(!ok)) {  // timed out: drain the products in flight (bounded), then leave
            undrained = !__syncthreads_and(mbar_wait(bar, phase));
            failed = true;
            return false;
        }
        phase ^= 1u;
        tc_fence_after();
        return true;
    };

    float s_w3 = 0.0f, s_b2 = 0.0f, s_b1 = 0.0f, s_b3 = 0.0f, s_loss = 0.0f;
    for (uint32_t tile = blockIdx.x; (uint64_t)tile * kTileRows < rows; tile += gridDim.x) {
        const uint32_t i = tile * kTileRows + r;
        const bool valid = i < rows;
        const uint32_t src = valid ? (perm ? perm[i] : i) : 0u;
        const uint4* const xrow = reinterpret_cast<const uint4*>(X + (size_t)src * kIn);
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            const uint32_t j = group * 4 + e;
            store_chunk(xs, r, j, valid && j < (uint32_t)kIn / 8 ? xrow[j] : make_uint4(0, 0, 0, 0));
        }
        const float goal = valid ? target[src] : 0.0f;
        const uint32_t more = tile != blockIdx.x;  // the weight gradients go on from the tile before
        if (!run([&] {
                for (uint32_t k = 0; k < kIn / 16; ++k)
                    umma_f16(z1t, sw128_desc(xs + kstep_offset(k)), sw128_desc_mn(w1s + k * kKstepRows), k > 0,
                             kIdesc | kMnB);
            }))
            break;
        float g1[32], g2[32];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            float v[16];
            tmem_ld16(z1t + my_lanes + c0 + h * 16, v);
            uint32_t q[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float a, b;
                gelu_both(v[2 * e] + b1v[c0 + h * 16 + 2 * e], &a, &g1[h * 16 + 2 * e]);
                gelu_both(v[2 * e + 1] + b1v[c0 + h * 16 + 2 * e + 1], &b, &g1[h * 16 + 2 * e + 1]);
                q[e] = pack_half2(a, b);
            }
            store_chunk(h1s, r, group * 4 + h * 2, make_uint4(q[0], q[1], q[2], q[3]));
            store_chunk(h1s, r, group * 4 + h * 2 + 1, make_uint4(q[4], q[5], q[6], q[7]));
        }
        if (!run([&] {
                for (uint32_t k = 0; k < 8; ++k)
                    umma_f16(z2t, sw128_desc(h1s + kstep_offset(k)), sw128_desc_mn(w2s + k * kKstepRows), k > 0,
                             kIdesc | kMnB);
            }))
            break;
        float y = 0.0f;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            float v[16];
            tmem_ld16(z2t + my_lanes + c0 + h * 16, v);
            uint32_t q[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const uint32_t c = c0 + h * 16 + 2 * e;
                float a, b;
                gelu_both(v[2 * e] + b2v[c], &a, &g2[h * 16 + 2 * e]);
                gelu_both(v[2 * e + 1] + b2v[c + 1], &b, &g2[h * 16 + 2 * e + 1]);
                q[e] = pack_half2(a, b);
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&q[e]));  // H2 is fp16
                y += f.x * w3v[c] + f.y * w3v[c + 1];
            }
            store_chunk(ts, r, group * 4 + h * 2, make_uint4(q[0], q[1], q[2], q[3]));
            store_chunk(ts, r, group * 4 + h * 2 + 1, make_uint4(q[4], q[5], q[6], q[7]));
        }
        ysum[group * kTileRows + r] = y;
        __syncthreads();
        y = ysum[r] + ysum[kTileRows + r] + ysum[2 * kTileRows + r] + ysum[3 * kTileRows + r] + b1v[3 * kH];
        const float d = valid ? y - goal : 0.0f, dy = 2.0f * d;
        if (group == 0) {
            dyv[r] = dy;
            s_b3 += dy;
            s_loss += d * d;
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t c = e * 8 + 2 * k;
                q[k] = pack_half2(dy * w3v[c0 + c] * g2[c], dy * w3v[c0 + c + 1] * g2[c + 1]);
            }
            store_chunk(dz2s, r, group * 4 + e, make_uint4(q[0], q[1], q[2], q[3]));
        }
        __syncthreads();
#pragma unroll 8
        for (uint32_t k = c0; k < c0 + 32; ++k) {
            s_w3 += half_at(ts, k, col) * dyv[k];
            s_b2 += half_at(dz2s, k, col);
        }
        if (!run([&] {
                for (uint32_t k = 0; k < 8; ++k)
                    umma_f16(dw2t, sw128_desc_mn(h1s + k * kKstepRows), sw128_desc_mn(dz2s + k * kKstepRows),
                             more | (k > 0), kIdesc | kMnA | kMnB);
                for (uint32_t k = 0; k < 8; ++k)
                    umma_f16(z2t, sw128_desc(dz2s + kstep_offset(k)), sw128_desc(w2s + kstep_offset(k)), k > 0);
            }))
            break;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            float v[16];
            tmem_ld16(z2t + my_lanes + c0 + h * 16, v);  // dH1
            uint32_t q[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                q[e] = pack_half2(v[2 * e] * g1[h * 16 + 2 * e], v[2 * e + 1] * g1[h * 16 + 2 * e + 1]);
            store_chunk(ts, r, group * 4 + h * 2, make_uint4(q[0], q[1], q[2], q[3]));
            store_chunk(ts, r, group * 4 + h * 2 + 1, make_uint4(q[4], q[5], q[6], q[7]));
        }
        if (!run([&] {
                for (uint32_t k = 0; k < 8; ++k)
                    umma_f16(dw1t, sw128_desc_mn(xs + k * kKstepRows), sw128_desc_mn(ts + k * kKstepRows),
                             more | (k > 0), kIdesc | kMnA | kMnB);
            }))
            break;
#pragma unroll 8
        for (uint32_t k = c0; k < c0 + 32; ++k) s_b1 += half_at(ts, k, col);
        __syncthreads();  // the row tiles are free for the next 128 rows
    }
    if (!failed) {
        const uint32_t slot = blockIdx.x;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            float v[16];
            tmem_ld16(dw2t + my_lanes + c0 + h * 16, v);
            float4* p = reinterpret_cast<float4*>(out.w2 + (size_t)slot * kH * kH + (size_t)r * kH + c0 + h * 16);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                p[e] = make_float4(inv * v[4 * e], inv * v[4 * e + 1], inv * v[4 * e + 2], inv * v[4 * e + 3]);
            tmem_ld16(dw1t + my_lanes + c0 + h * 16, v);
            p = reinterpret_cast<float4*>(out.w1 + (size_t)slot * kW1Size + (size_t)r * kH + c0 + h * 16);
            if (r < (uint32_t)kIn)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    p[e] = make_float4(inv * v[4 * e], inv * v[4 * e + 1], inv * v[4 * e + 2], inv * v[4 * e + 3]);
        }
        // column sums: the four row groups of each column, then b3 and the loss over the rows
        float* const part = reinterpret_cast<float*>(smem_raw + (base - raw) + 2 * kOpBytes);  // X is free
        part[t] = s_w3;
        part[kTrainThreads + t] = s_b2;
        part[2 * kTrainThreads + t] = s_b1;
        part[3 * kTrainThreads + t] = s_b3;
        part[4 * kTrainThreads + t] = s_loss;
        __syncthreads();
        if (t < (uint32_t)kH) {
            auto sum4 = [&](uint32_t k) {
                const float* p = part + k * kTrainThreads + t;
                return (p[0] + p[kH]) + (p[2 * kH] + p[3 * kH]);
            };
            out.w3[slot * kH + t] = inv * sum4(0);
            out.b2[slot * kH + t] = inv * sum4(1);
            out.b1[slot * kH + t] = inv * sum4(2);
        }
        if (warp < 2) {  // only the threads of group 0 (t < 128) have summed these
            const float* p = part + (3 + warp) * kTrainThreads + lane;
            float v = (p[0] + p[32]) + (p[64] + p[96]);
#pragma unroll
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
            if (lane == 0) out.tail[slot * 2 + warp] = warp == 0 ? inv * v : v;
        }
    }
    // bit 0: a completion wait timed out; bit 1: the drain timed out too, so products may still
    // have been in flight when the tensor memory was freed
    if (failed && t == 0) atomicOr(err, undrained ? 3u : 1u);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTrainTmem) : "memory");
    }
}

// Gradient of parameter i: the sum over the blocks' slots, in slot order.
__device__ __forceinline__ float grad_of(const GradParts& g, int i, int slots) {
    const float* p;
    size_t stride = kH;
    if (i < kB1) p = g.w1 + i, stride = kW1Size;
    else if (i < kW2) p = g.b1 + (i - kB1);
    else if (i < kB2) p = g.w2 + (i - kW2), stride = kH * kH;
    else if (i < kW3) p = g.b2 + (i - kB2);
    else if (i < kB3) p = g.w3 + (i - kW3);
    else p = g.tail, stride = 2;
    float s = 0.0f;
#pragma unroll 8
    for (int b = 0; b < slots; ++b) s += p[b * stride];
    return s;
}

__device__ __forceinline__ void add_loss(const GradParts& g, int slots, float* loss) {
    float s = 0.0f;
    for (int b = 0; b < slots; ++b) s += g.tail[2 * b + 1];
    *loss += s;
}

__global__ void grad_kernel(GradParts g, int slots, float* __restrict__ out, float* __restrict__ loss,
                            const unsigned* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (*err || i >= kParams) return;
    out[i] = grad_of(g, i, slots);
    if (i == 0) add_loss(g, slots, loss);
}

// Adam (Kingma & Ba 2015) on the flat fp32 parameters; refreshes the fp16 copies of W1, W2.
__global__ void adam_kernel(float* __restrict__ p, GradParts g, int slots, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2,
                            __half* __restrict__ w1h, __half* __restrict__ w2h, float* __restrict__ loss,
                            const unsigned* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (*err || i >= kParams) return;
    const float gi = grad_of(g, i, slots);
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = w;
    if (i < kW1Size) w1h[i] = __float2half(w);
    else if (i >= kW2 && i < kB2) w2h[i - kW2] = __float2half(w);
    if (i == 0) add_loss(g, slots, loss);
}

// Device buffers of the training steps of one call, for batches of up to `rows` rows.
struct Work {
    GradParts parts{};
    float* loss = nullptr;
    unsigned* err = nullptr;  // set by a step whose tensor-core completion wait timed out
    int max_slots = 0;
    cudaStream_t stream;  // the buffers are allocated and freed in its order
    std::vector<void*> owned;

    explicit Work(cudaStream_t s) : stream(s) {}
    Work(const Work&) = delete;
    Work& operator=(const Work&) = delete;

    int init(uint32_t rows, int device) {
        int sms = 0, s = cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        max_slots = (int)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)rows + kTileRows - 1) / kTileRows, sms));
        owned.reserve(8);  // may throw, but before anything is allocated; push_back then does not
        auto get = [&](auto** p, size_t count) {
            void* v = nullptr;
            const int st = dev_alloc_bytes(&v, count * sizeof(**p), stream);
            if (st == NQB_OK) {
                owned.push_back(v);
                *p = static_cast<std::remove_pointer_t<decltype(p)>>(v);
            }
            return st;
        };
        const size_t n = max_slots;
        if (!s) s = get(&parts.w1, n * kW1Size);
        if (!s) s = get(&parts.b1, n * kH);
        if (!s) s = get(&parts.w2, n * kH * kH);
        if (!s) s = get(&parts.b2, n * kH);
        if (!s) s = get(&parts.w3, n * kH);
        if (!s) s = get(&parts.tail, n * 2);
        if (!s) s = get(&loss, 1);
        if (!s) s = get(&err, 1);
        if (!s) s = cuda_status(cudaMemsetAsync(err, 0, sizeof(unsigned), stream));
        if (!s)
            s = cuda_status(cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)kTrainSmem));
        return s;
    }
    // NQB_E_STALL if a step so far timed out (synchronises the stream).
    int check(cudaStream_t s) const {
        unsigned h = 0;
        int st = cuda_status(cudaMemcpyAsync(&h, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        if (!st) st = cuda_status(cudaStreamSynchronize(s));
        return st ? st : (h & 2u) ? NQB_E_DEVICE : (h ? NQB_E_STALL : NQB_OK);
    }
    ~Work() {
        for (void* p : owned) dev_free(p, stream);
    }
};

unsigned blocks_for(uint64_t n, unsigned per = 256) { return (unsigned)((n + per - 1) / per); }

}  // namespace
}  // namespace mlp
}  // namespace nqb

// ---- the model object ---------------------------------------------------------------------
struct nqb_model {
    int device = 0;
    float* params = nullptr;  // fp32 master weights (kParams)
    float* grad = nullptr;
    float* m = nullptr;  // Adam moments
    float* v = nullptr;
    __half* w1h = nullptr;  // fp16 copies fed to the tensor cores
    __half* w2h = nullptr;
    long adam_step = 0;
};

namespace nqb {
namespace mlp {
namespace {

// Forward and backward over `rows` rows (of X and target, through perm when given): the blocks'
// shares of the mean gradient and of the summed squared error into w.parts.  Returns the
// number of slots through *slots.
int pass(const nqb_model* m, Work& w, const __half* X, const float* target, const uint32_t* perm, uint32_t rows,
         int* slots, cudaStream_t s) {
    const uint64_t tiles = ((uint64_t)rows + kTileRows - 1) / kTileRows;
    *slots = (int)std::min<uint64_t>(tiles, (uint64_t)w.max_slots);
    train_kernel<<<*slots, kTrainThreads, kTrainSmem, s>>>(X, target, perm, rows, m->w1h, m->w2h, m->params,
                                                           1.0f / (float)rows, w.parts, w.err);
    return cuda_status(cudaGetLastError());
}

// Seeded uniform initialisation: W ~ U(-sqrt(6/(fan_in+fan_out)), +) (Glorot), biases 0,
// b3 = the mean target so the first steps start near the data.
void init_params(std::vector<float>& p, uint64_t seed) {
    p.assign(kParams, 0.0f);
    uint64_t st = seed ? seed : 0x9E3779B97F4A7C15ull;
    auto next = [&]() {
        uint64_t z = (st += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](int off, int n, int fin, int fout) {
        const double a = std::sqrt(6.0 / (fin + fout));
        for (int i = 0; i < n; ++i) p[off + i] = (float)((2.0 * next() - 1.0) * a);
    };
    fill(kW1, kIn * kH, 100, kH);  // 100 live inputs of the 112
    fill(kW2, kH * kH, kH, kH);
    fill(kW3, kH, kH, 1);
}

}  // namespace
}  // namespace mlp
}  // namespace nqb

using namespace nqb;
using namespace nqb::mlp;

namespace {

struct CallScope {  // current device for the call, restored afterwards; one stream
    int prev = 0;
    cudaStream_t s = nullptr;
    int status = NQB_OK;
    explicit CallScope(int dev) {
        cudaGetDevice(&prev);
        if ((status = cuda_status(cudaSetDevice(dev)))) return;
        status = stream_take(&s);
    }
    ~CallScope() {
        if (s) stream_give(s);
        cudaSetDevice(prev);
    }
};

// Device buffer of one call, stream-ordered.
template <class T>
struct DevBuf {
    T* p = nullptr;
    cudaStream_t s;
    explicit DevBuf(cudaStream_t st) : s(st) {}
    int alloc(size_t n) { return dev_alloc(&p, (n ? n : 1) * sizeof(T), s); }
    ~DevBuf() { dev_free(p, s); }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
};

int refresh_half(nqb_model* m, cudaStream_t s) {
    to_half_kernel<<<blocks_for(kH * kH), 256, 0, s>>>(m->params, m->w1h, m->w2h);
    return cuda_status(cudaGetLastError());
}

}  // namespace

extern "C" {

int nqb_model_create(int device, uint64_t seed, nqb_model** out) try {
    if (!out) return NQB_E_INVALID;
    *out = nullptr;
    int st = nqb_device_check(device);
    if (st) return st;
    CallScope cs(device);
    if (cs.status) return cs.status;
    std::vector<float> p;  // before the model object: nothing to release if this throws
    init_params(p, seed);
    nqb_model* m = new nqb_model();
    m->device = device;
    st = cuda_malloc(&m->params, kParams * sizeof(float));
    if (!st) st = cuda_malloc(&m->grad, kParams * sizeof(float));
    if (!st) st = cuda_malloc(&m->m, kParams * sizeof(float));
    if (!st) st = cuda_malloc(&m->v, kParams * sizeof(float));
    if (!st) st = cuda_malloc(&m->w1h, kW1Size * sizeof(__half));
    if (!st) st = cuda_malloc(&m->w2h, kH * kH * sizeof(__half));
    if (!st) st = cuda_status(cudaMemcpyAsync(m->params, p.data(), kParams * sizeof(float), cudaMemcpyHostToDevice, cs.s));
    if (!st) st = cuda_status(cudaMemsetAsync(m->m, 0, kParams * sizeof(float), cs.s));
    if (!st) st = cuda_status(cudaMemsetAsync(m->v, 0, kParams * sizeof(float), cs.s));
    if (!st) st = refresh_half(m, cs.s);
    if (!st) st = cuda_status(cudaStreamSynchronize(cs.s));
    if (st) {
        nqb_model_destroy(m);
        return st;
    }
    *out = m;
    return NQB_OK;
} NQB_ABI_CATCH

void nqb_model_destroy(nqb_model* m) {
    if (!m) return;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(m->device);
    cudaFree(m->params);
    cudaFree(m->grad);
    cudaFree(m->m);
    cudaFree(m->v);
    cudaFree(m->w1h);
    cudaFree(m->w2h);
    cudaSetDevice(prev);
    delete m;
}

int nqb_model_get_params(const nqb_model* m, float* out) {
    if (!m || !out) return NQB_E_INVALID;
    CallScope cs(m->device);
    if (cs.status) return cs.status;
    int st = cuda_status(cudaMemcpyAsync(out, m->params, kParams * sizeof(float), cudaMemcpyDeviceToHost, cs.s));
    if (!st) st = cuda_status(cudaStreamSynchronize(cs.s));
    return st;
}

int nqb_model_set_params(nqb_model* m, const float* in) {
    if (!m || !in) return NQB_E_INVALID;
    CallScope cs(m->device);
    if (cs.status) return cs.status;
    int st = cuda_status(cudaMemcpyAsync(m->params, in, kParams * sizeof(float), cudaMemcpyHostToDevice, cs.s));
    if (!st) st = cuda_status(cudaMemsetAsync(m->m, 0, kParams * sizeof(float), cs.s));
    if (!st) st = cuda_status(cudaMemsetAsync(m->v, 0, kParams * sizeof(float), cs.s));
    if (!st) st = refresh_half(m, cs.s);
    if (!st) st = cuda_status(cudaStreamSynchronize(cs.s));
    m->adam_step = 0;
    return st;
}

int nqb_model_features(const nqb_state* states, uint64_t count, float* out) try {
    if (count && (!states || !out)) return NQB_E_INVALID;
    for (uint64_t i = 0; i < count; ++i) {
        uint4 st;
        std::memcpy(&st, &states[i], sizeof(st));
        for (int j = 0; j < kIn; ++j) out[i * kIn + j] = feature(st, j);
    }
    return NQB_OK;
} NQB_ABI_CATCH

int nqb_model_predict(const nqb_model* m, const nqb_state* states, uint64_t count, float* out) try {
    return nqb_model_predict_ex(m, states, count, out, 0);
} NQB_ABI_CATCH

int nqb_model_predict_ex(const nqb_model* m, const nqb_state* states, uint64_t count, float* out,
                         uint32_t wait_limit) try {
    if (!m || (count && (!states || !out))) return NQB_E_INVALID;
    if (count == 0) return NQB_OK;
    if (count > 0xFFFFFFFFull) return NQB_E_RANGE;
    CallScope cs(m->device);
    if (cs.status) return cs.status;
    DevBuf<nqb_state> d_st(cs.s);
    DevBuf<float> d_out(cs.s);
    int st = d_st.alloc(count);
    if (!st) st = d_out.alloc(count);
    if (!st) st = cuda_status(cudaMemcpyAsync(d_st.p, states, count * sizeof(nqb_state), cudaMemcpyHostToDevice, cs.s));
    if (!st) st = nqb::model_predict_device(m, d_st.p, (uint32_t)count, d_out.p, cs.s, wait_limit);
    if (!st) st = cuda_status(cudaMemcpyAsync(out, d_out.p, count * sizeof(float), cudaMemcpyDeviceToHost, cs.s));
    if (!st) st = cuda_status(cudaStreamSynchronize(cs.s));
    return st;
} NQB_ABI_CATCH

int nqb_model_loss_grad(nqb_model* m, const nqb_state* states, const float* targets, uint64_t count, float* loss,
                        float* grad) try {
    if (!m || !states || !targets || !loss || !grad || count == 0) return NQB_E_INVALID;
    if (count > (1u << 20)) return NQB_E_RANGE;
    CallScope cs(m->device);
    if (cs.status) return cs.status;
    Work w(cs.s);
    DevBuf<nqb_state> d_st(cs.s);
    DevBuf<__half> d_X(cs.s);
    DevBuf<float> d_t(cs.s);
    int st = w.init((uint32_t)count, m->device);
    if (!st) st = d_st.alloc(count);
    if (!st) st = d_X.alloc(count * kIn);
    if (!st) st = d_t.alloc(count);
    if (!st) st = cuda_status(cudaMemcpyAsync(d_st.p, states, count * sizeof(nqb_state), cudaMemcpyHostToDevice, cs.s));
    if (!st) st = cuda_status(cudaMemcpyAsync(d_t.p, targets, count * sizeof(float), cudaMemcpyHostToDevice, cs.s));
    if (st) return st;
    features_kernel<<<blocks_for(count * kIn), 256, 0, cs.s>>>(reinterpret_cast<const uint4*>(d_st.p), count, d_X.p);
    cudaMemsetAsync(w.loss, 0, sizeof(float), cs.s);
    int slots = 0;
    if ((st = pass(m, w, d_X.p, d_t.p, nullptr, (uint32_t)count, &slots, cs.s))) return st;
    grad_kernel<<<blocks_for(kParams), 256, 0, cs.s>>>(w.parts, slots, m->grad, w.loss, w.err);
    if ((st = cuda_status(cudaGetLastError()))) return st;
    float l = 0;
    st = cuda_status(cudaMemcpyAsync(&l, w.loss, sizeof(float), cudaMemcpyDeviceToHost, cs.s));
    if (!st) st = cuda_status(cudaMemcpyAsync(grad, m->grad, kParams * sizeof(float), cudaMemcpyDeviceToHost, cs.s));
    if (!st) st = w.check(cs.s);
    *loss = l / (float)count;
    return st;
} NQB_ABI_CATCH

int nqb_model_train(nqb_model* m, const nqb_state* states, const float* targets, uint64_t count,
                    const nqb_train_opts* opts, float* epoch_loss) try {
    if (!m || !states || !targets || count == 0) return NQB_E_INVALID;
    if (count > 0xFFFFFFFFull) return NQB_E_RANGE;
    nqb_train_opts o;
    std::memset(&o, 0, sizeof(o));
    o.epochs = 8;
    o.batch = 4096;
    o.lr = 1e-3f;
    o.seed = 1;
    if (opts) o = *opts;
    if (o.epochs <= 0 || o.batch <= 0 || o.batch > (1 << 20) || !(o.lr > 0.0f)) return NQB_E_INVALID;
    EpochOrder order;  // before the scope, which waits for the stream on every way out
    CallScope cs(m->device);
    if (cs.status) return cs.status;
    const uint32_t B = (uint32_t)std::min<uint64_t>(o.batch, count);
    Work w(cs.s);
    DevBuf<nqb_state> d_st(cs.s);
    DevBuf<__half> d_X(cs.s);
    DevBuf<float> d_t(cs.s);
    DevBuf<uint32_t> d_perm(cs.s);
    int st = w.init(B, m->device);
    if (!st) st = d_st.alloc(count);
    if (!st) st = d_X.alloc(count * kIn);
    if (!st) st = d_t.alloc(count);
    if (!st) st = d_perm.alloc(count);
    if (!st) st = cuda_status(cudaMemcpyAsync(d_st.p, states, count * sizeof(nqb_state), cudaMemcpyHostToDevice, cs.s));
    if (!st) st = cuda_status(cudaMemcpyAsync(d_t.p, targets, count * sizeof(float), cudaMemcpyHostToDevice, cs.s));
    if (st) return st;
    features_kernel<<<blocks_for(count * kIn), 256, 0, cs.s>>>(reinterpret_cast<const uint4*>(d_st.p), count, d_X.p);
    order.start(count, o.seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int ep = 0; ep < o.epochs; ++ep) {
        st = cuda_status(cudaMemcpyAsync(d_perm.p, order.current(), count * sizeof(uint32_t), cudaMemcpyHostToDevice, cs.s));
        if (st) return st;
        cudaMemsetAsync(w.loss, 0, sizeof(float), cs.s);
        for (uint64_t off = 0; off < count; off += B) {
            const uint32_t rows = (uint32_t)std::min<uint64_t>(B, count - off);
            int slots = 0;
            if ((st = pass(m, w, d_X.p, d_t.p, d_perm.p + off, rows, &slots, cs.s))) return st;
            m->adam_step++;
            const float c1 = 1.0f - std::pow(b1, (float)m->adam_step), c2 = 1.0f - std::pow(b2, (float)m->adam_step);
            adam_kernel<<<blocks_for(kParams), 256, 0, cs.s>>>(m->params, w.parts, slots, m->m, m->v, o.lr, b1, b2, eps,
                                                                c1, c2, m->w1h, m->w2h, w.loss, w.err);
        }
        if (ep + 1 < o.epochs) order.prepare();  // while the device works on this epoch
        float l = 0;
        st = cuda_status(cudaMemcpyAsync(&l, w.loss, sizeof(float), cudaMemcpyDeviceToHost, cs.s));
        if (!st) st = w.check(cs.s);
        if (st) return st;
        if (epoch_loss) epoch_loss[ep] = l / (float)count;
        if (ep + 1 < o.epochs) order.advance();  // check() has waited for the stream
    }
    return cuda_status(cudaStreamSynchronize(cs.s));
} NQB_ABI_CATCH

}  // extern "C"

namespace nqb {

int model_predict_device(const nqb_model* m, const nqb_state* d_states, uint32_t count, float* d_out, cudaStream_t s,
                         uint32_t wait_limit) {
    if (count == 0) return NQB_OK;  // wait_limit 0: the default (suspending) bounded wait
    cudaError_t e = cudaFuncSetAttribute(predict_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPredictSmem);
    if (e != cudaSuccess) return cuda_status(e);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
    const uint64_t tiles = ((uint64_t)count + kTileRows - 1) / kTileRows;
    // at most 2 blocks per SM (shared memory), so their tensor memory (2 x 128 columns) fits
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)sms * 2));
    unsigned* d_err = nullptr;
    NQB_TRY(dev_alloc(&d_err, sizeof(unsigned), s));
    unsigned h_err = 0;
    int st = cuda_status(cudaMemsetAsync(d_err, 0, sizeof(unsigned), s));
    if (!st) {
        predict_kernel<<<grid, kPredictThreads, kPredictSmem, s>>>(reinterpret_cast<const uint4*>(d_states), count,
                                                                   m->w1h, m->w2h, m->params, d_out, wait_limit, d_err);
        st = cuda_status(cudaGetLastError());
    }
    if (!st) st = cuda_status(cudaMemcpyAsync(&h_err, d_err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    if (!st) st = cuda_status(cudaStreamSynchronize(s));
    dev_free(d_err, s);
    if (!st && h_err) st = (h_err & 2u) ? NQB_E_DEVICE : NQB_E_STALL;
    return st;
}

int model_device(const nqb_model* m) { return m->device; }

}  // namespace nqb
