// vbd_mlp_train_tc.cuh -- loss and parameter gradients of the warm-start MLP (64 -> 128 -> 128 -> 3,
// SiLU) in one pass over the samples on the 5th-generation tensor cores.  Included by vbd_mlp.cu only.
//
// One persistent CTA of 512 threads per SM takes 128-sample tiles.  A tile's activations and their
// gradients live in shared memory as BF16 operands and never reach HBM; the weight gradients
// accumulate over all tiles of the CTA in tensor memory (FP32), so that a CTA writes one partial of
// the parameter blob at its end, and a second kernel adds the partials in CTA order (deterministic).
// Per tile (thread: one row, a quarter of the 128 columns):
//   Z1 = X W1,  H1 = silu(Z1 + b1);  Z2 = H1 W2,  H2 = silu(Z2 + b2);  Y = H2 W3 + b3, loss, dY
//   dH2 = dY W3^T,  dZ2 = dH2 silu'(Z2);  dH1 = dZ2 W2^T,  dZ1 = dH1 silu'(Z1)
//   dW3 += H2^T dY,  dW2 += H1^T dZ2,  dW1^T += dZ1^T X,  db += dZ^T 1  (issued beside the products
//   that the next epilogue waits for)
// Rounding is that of a layer-by-layer BF16 pass: weights, inputs, activations, pre-activations (for
// silu') and gradients are rounded to BF16 as operands, every product accumulates in FP32, and
// biases, SiLU and its derivative are FP32 -- with the approximate FP32 division (__fdividef, 2 ulp) in the
// sigmoid, and the bias gradients summed by the tensor cores.  Against 64 bits over 1,000 to 131,072
// samples (42 passes) the gradients are off by 2.5599e-3 on average, at most 3.7793e-3; with the IEEE
// division 2.5599e-3 and 3.7810e-3 (and 64 us instead of 45), and the mma.sync passes 2.5599e-3 and
// 3.7807e-3.
//
// Operand views.  A tile operand of 128 rows by K columns is stored K-major without swizzle (as in
// vbd_mlp_tc.cuh): core matrices of 8 rows x 16 bytes, 8-row groups 128 bytes apart, groups of 8
// columns 2048 bytes apart.  Read with rows and columns exchanged, the same bytes are the canonical
// MN-major layout (8 columns contiguous, 8 rows 16 bytes apart): the products that contract over the
// samples (dW = A^T B) and those with a transposed weight take that view of the same buffer (the
// transpose bits of the instruction descriptor, stride offset = column groups, leading offset = row
// groups), so nothing is transposed or stored twice.
//
// What bounds it: two tiles per SM at 32,768 samples, each a serial chain of six products and
// epilogues; the epilogues' exponentials and reciprocals (4 x 16,384 of each per tile) are the
// largest part, so four warps share a row quarter's columns.  Measured, a training pass over 32,768
// samples: 45 us with 512 threads (51 with 256), against 195 us for mma.sync passes with their
// operands in HBM (tile kernel, three split-K products, column sums).
#pragma once

#include <cuda_bf16.h>

#include "vbd_mlp_tc.cuh"

namespace vbd {
namespace tct {

constexpr int kThreads = 512;
constexpr int kCols = 32;  // accumulator columns per thread
constexpr int kMaxCtas = 148;  // one per SM; partials of the workspace
constexpr int kRows = 128;
constexpr int kIn = 64, kHid = 128, kOutP = 8;
constexpr int kN3 = 16;  // MMA width of the 3 outputs (and of the column of ones)
// parameter blob offsets (as vbd_mlp.cu), then the loss
constexpr int kOffW1 = 0, kOffB1 = kIn * kHid, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
              kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kOutP, kParams = kOffB3 + kOutP;
constexpr int kPart = kParams + 8;  // floats per partial: parameters, loss, padding

// shared memory (bytes)
constexpr int kSW1 = 0;
constexpr int kSW2 = kSW1 + kHid * kIn * 2;
constexpr int kSW3 = kSW2 + kHid * kHid * 2;
constexpr int kSOnes = kSW3 + kN3 * kHid * 2;
constexpr int kSX = kSOnes + kN3 * kRows * 2;
constexpr int kSH1 = kSX + kRows * kIn * 2;
constexpr int kSH2 = kSH1 + kRows * kHid * 2;  // H2, then dZ1
constexpr int kSDZ2 = kSH2 + kRows * kHid * 2;
constexpr int kSDY = kSDZ2 + kRows * kHid * 2;
constexpr int kSBias = kSDY + kRows * kN3 * 2;  // b1, b2 [128] and b3 [8] float
constexpr int kSRed = kSBias + (2 * kHid + kOutP) * 4;  // per-warp sums of loss and db3
constexpr int kSBar = kSRed + (kThreads / 32) * 4 * 4;
constexpr int kSmemBytes = kSBar + 16 + 1024;  // + slack for aligning the base

// tensor memory columns
constexpr uint32_t kCWork = 0, kCW2 = 128, kCW1 = 256, kCW3 = 320, kCB1 = 336, kCB2 = 352, kTmemCols = 512;

struct TrainArgs {
    int n;
    const float* params;  // FP32 blob (biases)
    const uint16_t* w16;  // BF16 weights W1 [64][128], W2 [128][128], W3 [128][8]
    const float* X;       // [n][64]
    const float* T;       // [n][3]
    float grad_scale;     // dL/dY = grad_scale * 2 (y - t)
    float* part;          // [gridDim.x][kPart]
    unsigned* status;     // incremented on a wait that gave up
};

// kind::f16 with BF16 operands and FP32 accumulators; ta / tb: A / B read MN-major
__host__ __device__ constexpr uint32_t idesc(int N, bool ta, bool tb) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (ta ? 1u << 15 : 0u) | (tb ? 1u << 16 : 0u) |
           (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
}

// one product over `slices` steps of K = 16: operand start addresses, their step per slice, and the
// descriptors' leading / stride byte offsets
struct Op {
    uint32_t addr, step, lbo, sbo;
};
__device__ __forceinline__ Op k_major(uint32_t addr, int rows) {
    const uint32_t group = static_cast<uint32_t>(rows / 8) * 128;  // between groups of 8 columns
    return {addr, 2 * group, group, 128};
}
// contracts over the buffer's rows
__device__ __forceinline__ Op mn_major(uint32_t addr, int rows) {
    return {addr, 256, 128, static_cast<uint32_t>(rows / 8) * 128};
}
__device__ __forceinline__ void product(uint32_t d, Op a, Op b, uint32_t desc, int slices, bool accumulate) {
    for (int s = 0; s < slices; ++s)
        tc::mma_f16(d, tc::smem_desc(a.addr + s * a.step, a.lbo, a.sbo), tc::smem_desc(b.addr + s * b.step, b.lbo, b.sbo),
                    desc, (accumulate || s > 0) ? 1u : 0u);
}

__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float2 unpack2(unsigned u) {
    __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
    return __bfloat1622float2(v);
}
__device__ __forceinline__ float sigm(float z) { return __fdividef(1.0f, 1.0f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = sigm(z);
    return s * (1.0f + z * (1.0f - s));
}

__global__ void __launch_bounds__(kThreads, 1) mlp_train_tc_kernel(const __grid_constant__ TrainArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* sB = reinterpret_cast<float*>(smem + kSBias);
    float* sRed = reinterpret_cast<float*>(smem + kSRed);
    uint64_t* bar_slot = reinterpret_cast<uint64_t*>(smem + kSBar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kSBar + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quarter = warp & 3, part = warp >> 2;  // TMEM lanes of the warp, its quarter of the columns
    const int row = quarter * 32 + lane, c0 = part * kCols;

    // ---- weights [K][N] -> [N][K] operands, ones, biases, mbarrier, TMEM ----
    auto weights = [&](int dst, const uint16_t* src, int K, int N, int R) {
        for (int i = tid; i < (K / 8) * R; i += kThreads) {
            const int nn = i % R, kg = i / R;
            unsigned w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned lo = nn < N ? __ldg(src + (kg * 8 + 2 * j) * N + nn) : 0u;
                const unsigned hi = nn < N ? __ldg(src + (kg * 8 + 2 * j + 1) * N + nn) : 0u;
                w[j] = lo | (hi << 16);
            }
            *reinterpret_cast<uint4*>(smem + dst + tc::kmajor_offset(nn, kg * 8, R)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    };
    weights(kSW1, a.w16, kIn, kHid, kHid);
    weights(kSW2, a.w16 + kIn * kHid, kHid, kHid, kHid);
    weights(kSW3, a.w16 + kIn * kHid + kHid * kHid, kHid, kOutP, kN3);  // rows 8..15 zero
    {
        const unsigned one2 = pack2(1.0f, 1.0f);
        for (int i = tid; i < kN3 * kRows / 8; i += kThreads)
            *reinterpret_cast<uint4*>(smem + kSOnes + 16 * i) = make_uint4(one2, one2, one2, one2);
        for (int i = tid; i < kRows * kN3 / 8; i += kThreads)
            *reinterpret_cast<uint4*>(smem + kSDY + 16 * i) = make_uint4(0u, 0u, 0u, 0u);
    }
    for (int i = tid; i < kHid; i += kThreads) {
        sB[i] = a.params[kOffB1 + i];
        sB[kHid + i] = a.params[kOffB2 + i];
    }
    if (tid < kOutP) sB[2 * kHid + tid] = a.params[kOffB3 + tid];
    const uint32_t bar = tc::smem_u32(bar_slot);
    if (tid == 0) {
        tc::bar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc::fence_proxy_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tm = *tmem_slot, work = tm + kCWork;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t base = tc::smem_u32(smem);
    const uint32_t w1 = base + kSW1, w2 = base + kSW2, w3 = base + kSW3, ones = base + kSOnes, x = base + kSX,
                   h1 = base + kSH1, h2 = base + kSH2, dz2 = base + kSDZ2, dy = base + kSDY, dz1 = h2;
    const bool issuer = tid == 0;
    uint32_t phase = 0;
    bool ok = true;
    float loss = 0.f, db3[3] = {0.f, 0.f, 0.f};

    // operands written by all threads -> the issuer may start its products
    auto publish = [&]() {
        tc::fence_proxy_async();
        tc::fence_before();
        __syncthreads();
        if (issuer) tc::fence_after();
    };
    // all threads: the committed products are done (false: a wait gave up)
    auto await = [&]() {
        ok = __syncthreads_and(tc::bar_wait(bar, phase)) != 0;
        phase ^= 1u;
        tc::fence_after();
        return ok;
    };
    // this thread's part of a row of BF16 values into a 128-row operand, 8 at a time
    auto store8 = [&](int dst, int c, const unsigned (&w)[4]) {
        *reinterpret_cast<uint4*>(smem + dst + tc::kmajor_offset(row, c, kRows)) = make_uint4(w[0], w[1], w[2], w[3]);
    };
    // X rows of a tile: 8 rows x 64 contiguous bytes per load instruction
    float4 xv[4];
    const bool vec = (reinterpret_cast<uintptr_t>(a.X) & 15u) == 0;
    auto load_x = [&](int tile) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = warp * 8 + (lane & 7), c4 = 4 * j + (lane >> 3);
            const int s = tile * kRows + r;
            const float* src = a.X + static_cast<size_t>(s) * kIn + 4 * c4;
            xv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < a.n)
                xv[j] = vec ? __ldg(reinterpret_cast<const float4*>(src))
                            : make_float4(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3));
        }
    };

    const int tiles = (a.n + kRows - 1) / kRows;
    load_x(blockIdx.x);
    bool first = true;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int sample = tile * kRows + row;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = warp * 8 + (lane & 7), c4 = 4 * j + (lane >> 3);
            *reinterpret_cast<uint2*>(smem + kSX + tc::kmajor_offset(r, 4 * c4, kRows)) =
                make_uint2(pack2(xv[j].x, xv[j].y), pack2(xv[j].z, xv[j].w));
        }
        float tgt[3] = {0.f, 0.f, 0.f};
        if (part == 0 && sample < a.n) {
#pragma unroll
            for (int c = 0; c < 3; ++c) tgt[c] = __ldg(a.T + static_cast<size_t>(sample) * 3 + c);
        }
        // ---- forward ----
        publish();
        if (issuer) {
            product(work, k_major(x, kRows), k_major(w1, kHid), idesc(kHid, false, false), kIn / 16, false);
            tc::mma_commit(bar);
        }
        if (!await()) break;
        unsigned z1p[kCols / 2], z2p[kCols / 2];  // pre-activations as BF16 pairs, for silu'
        float acc[kCols];
        auto hidden = [&](const float* b, unsigned (&zp)[kCols / 2], int dst) {
            tc::tmem_ld32(work + lanes + c0, acc);
#pragma unroll
            for (int q = 0; q < kCols / 8; ++q) {
                unsigned w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 8 * q + 2 * j;
                    const float za = acc[c] + b[c0 + c], zb = acc[c + 1] + b[c0 + c + 1];
                    zp[c / 2] = pack2(za, zb);
                    w[j] = pack2(silu(za), silu(zb));
                }
                store8(dst, c0 + 8 * q, w);
            }
        };
        hidden(sB, z1p, kSH1);
        publish();
        if (issuer) {
            product(work, k_major(h1, kRows), k_major(w2, kHid), idesc(kHid, false, false), kHid / 16, false);
            tc::mma_commit(bar);
        }
        if (!await()) break;
        hidden(sB + kHid, z2p, kSH2);
        publish();
        if (issuer) {
            product(work, k_major(h2, kRows), k_major(w3, kN3), idesc(kN3, false, false), kHid / 16, false);
            tc::mma_commit(bar);
        }
        if (!await()) break;
        if (part == 0) {
            float y[16];
            tc::tmem_ld16(work + lanes, y);
            float d[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float e = sample < a.n ? y[c] + sB[2 * kHid + c] - tgt[c] : 0.f;
                loss += e * e;
                d[c] = a.grad_scale * 2.0f * e;
            }
            const unsigned w[4] = {pack2(d[0], d[1]), pack2(d[2], 0.f), 0u, 0u};
            db3[0] += unpack2(w[0]).x;
            db3[1] += unpack2(w[0]).y;
            db3[2] += unpack2(w[1]).x;
            store8(kSDY, 0, w);  // columns 8..15 stay zero
        }
        // ---- backward ----
        publish();
        if (issuer) {
            product(work, k_major(dy, kRows), mn_major(w3, kN3), idesc(kHid, false, true), 1, false);
            product(tm + kCW3, mn_major(h2, kRows), mn_major(dy, kRows), idesc(kN3, true, true), kRows / 16, !first);
            tc::mma_commit(bar);
        }
        if (!await()) break;
        auto gradient = [&](const unsigned (&zp)[kCols / 2], int dst) {
            tc::tmem_ld32(work + lanes + c0, acc);
#pragma unroll
            for (int q = 0; q < kCols / 8; ++q) {
                unsigned w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = 8 * q + 2 * j;
                    const float2 z = unpack2(zp[c / 2]);
                    w[j] = pack2(acc[c] * dsilu(z.x), acc[c + 1] * dsilu(z.y));
                }
                store8(dst, c0 + 8 * q, w);
            }
        };
        gradient(z2p, kSDZ2);
        publish();
        if (issuer) {
            product(work, k_major(dz2, kRows), mn_major(w2, kHid), idesc(kHid, false, true), kHid / 16, false);
            product(tm + kCW2, mn_major(h1, kRows), mn_major(dz2, kRows), idesc(kHid, true, true), kRows / 16, !first);
            product(tm + kCB2, mn_major(dz2, kRows), k_major(ones, kN3), idesc(kN3, true, false), kRows / 16, !first);
            tc::mma_commit(bar);
        }
        if (!await()) break;
        gradient(z1p, kSH2);  // dZ1: H2's last product has completed
        publish();
        if (issuer) {
            product(tm + kCW1, mn_major(dz1, kRows), mn_major(x, kRows), idesc(kIn, true, true), kRows / 16, !first);
            product(tm + kCB1, mn_major(dz1, kRows), k_major(ones, kN3), idesc(kN3, true, false), kRows / 16, !first);
            tc::mma_commit(bar);
        }
        first = false;
        if (tile + static_cast<int>(gridDim.x) < tiles) load_x(tile + gridDim.x);
        if (!await()) break;  // X and the operand buffers are free
    }
    // ---- the CTA's partial of the parameter blob ----
    float* out = a.part + static_cast<size_t>(blockIdx.x) * kPart;
    if (ok) {
        float acc[kCols];
        tc::tmem_ld32(tm + kCW2 + lanes + c0, acc);
        float4* o2 = reinterpret_cast<float4*>(out + kOffW2 + row * kHid + c0);
#pragma unroll
        for (int q = 0; q < kCols / 4; ++q) o2[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        float v[16];
        if (part < 2) {  // the inputs' 64 columns
            tc::tmem_ld32(tm + kCW1 + lanes + c0, acc);
#pragma unroll
            for (int f = 0; f < kCols; ++f) out[kOffW1 + (c0 + f) * kHid + row] = acc[f];
        } else if (part == 2) {
            tc::tmem_ld16(tm + kCW3 + lanes, v);
            float4* o3 = reinterpret_cast<float4*>(out + kOffW3 + row * kOutP);
            o3[0] = make_float4(v[0], v[1], v[2], v[3]);
            o3[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
            tc::tmem_ld16(tm + kCB1 + lanes, v);
            out[kOffB1 + row] = v[0];
            tc::tmem_ld16(tm + kCB2 + lanes, v);
            out[kOffB2 + row] = v[0];
        }
    } else {
        // a wait gave up: record it, wait (bounded) for the products in flight before freeing TMEM
        if (issuer) {
            if (a.status) atomicAdd(a.status, 1u);
            tc::bar_wait(bar, phase ^ 1u);
        }
        for (int i = tid; i < kPart; i += kThreads) out[i] = 0.f;
    }
    float red[4] = {loss, db3[0], db3[1], db3[2]};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        for (int off = 16; off > 0; off >>= 1) red[k] += __shfl_xor_sync(0xffffffffu, red[k], off);
        if (lane == 0) sRed[warp * 4 + k] = red[k];
    }
    tc::fence_before();
    __syncthreads();
    if (ok && tid < kOutP) {
        // part 0's four warps hold the sums
        auto sum = [&](int k) { return sRed[k] + sRed[4 + k] + sRed[8 + k] + sRed[12 + k]; };
        out[kOffB3 + tid] = tid < 3 ? sum(1 + tid) : 0.f;
        out[kParams + tid] = tid == 0 ? sum(0) : 0.f;
    }
    if (warp == 0) {
        tc::fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(kTmemCols));
    }
}

// grads[i] = the partials added in CTA order (four interleaved chains, then their sum: a fixed order);
// the loss is added to the caller's value
constexpr int kReduceWidth = 64, kReduceChains = 4;
__global__ void __launch_bounds__(kReduceWidth* kReduceChains)
    mlp_train_reduce_kernel(const float* part, int ctas, float* grads, float* loss) {
    __shared__ float s[kReduceChains][kReduceWidth];
    const int lane = threadIdx.x % kReduceWidth, chain = threadIdx.x / kReduceWidth;
    const int i = blockIdx.x * kReduceWidth + lane;
    float v = 0.f;
    if (i <= kParams) {
#pragma unroll 8
        for (int c = chain; c < ctas; c += kReduceChains) v += part[static_cast<size_t>(c) * kPart + i];
    }
    s[chain][lane] = v;
    __syncthreads();
    if (chain != 0 || i > kParams) return;
    for (int c = 1; c < kReduceChains; ++c) v += s[c][lane];
    if (i < kParams) grads[i] = v;
    else if (loss) *loss += v;
}

}  // namespace tct
}  // namespace vbd
