// The surrogate's network on the tensor cores: C = A B^T with BF16 operands and an FP32 accumulator in tensor memory
// (tcgen05.mma, kind::f16, one CTA a 128-row tile), and the element-wise kernels of training (activation, its
// gradient, transposes, the mean-square-error gradient, column sums, Adam).
//
// The products: C (M x N) = A B^T, 16 <= N <= 256, N and K multiples of 16, each operand K-major (row-major M x K or
// N x K) or MN-major (row-major K x M or K x N: what a backward pass has in hand, so nothing is transposed in memory).
// They are a few megaflops each, so latency bounds them: launches, one trip to L2 for the operands, one for the
// epilogue's. A CTA of 8 warps therefore takes a tile of 128 x 32 (a product of 256 x 256 is 16 CTAs), all of a K
// chunk's copies (cp.async, 16 B each) in flight at once, and the element-wise work that follows a product (bias and
// activation, the loss gradient, the activation's gradient, bias gradients, Adam) is its epilogue. A 256 x 256 x 256
// product takes 8.4 us where a CTA a 128-row tile, staging 128 of K at a time by loads through registers with
// 8-way bank conflicts, took 39 us; a training step at a batch of 256 is 9 launches and
// 94 us instead of 50 launches and 700 us.
// Operands sit in shared memory in the canonical layout without swizzle: core matrices of 8 rows of 16 bytes (K-major:
// 8 rows of 8 K; MN-major: 8 K of 8 rows), the next 8 of K 128 B on, the next 8 rows (K chunk / 8) x 128 B on, in both
// orders. Thread 0 issues one MMA per 16 of K against the accumulator in tensor memory and commits it to an mbarrier;
// the CTA waits (bounded) before the next chunk overwrites the tiles. The epilogue reads the accumulator with
// tcgen05.ld.32x32b (warp w owns tensor-memory lanes 32 (w mod 4) .. + 31, one row each, and half of the columns).
// A wait that gives up sets the status word, waits once more for the MMAs in flight, frees the tensor memory and
// returns.
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "w2b_common.cuh"
#include "w2b_tma.cuh"

namespace w2b {

constexpr int GEMM_M = 128, GEMM_N = 32;
constexpr int GEMM_KC = 256;  // K staged a chunk at a time
constexpr int GEMM_THREADS = 256;
constexpr int GEMM_SMEM = (GEMM_M + GEMM_N) * GEMM_KC * 2;  // 80 KB: two CTAs a SM

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    // shared-memory matrix descriptor: start address, leading and stride byte offsets (16-byte units), version 1 for
    // this architecture, no swizzle (cute/arch/mma_sm100_desc.hpp SmemDescriptor)
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 bytes into shared memory (asynchronously), zeros where valid is false.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// A K chunk (kw of it from k0) of `rows` rows of an operand, from row r0 on, into shared memory; rows at or past
// `limit` are zero. mn: the operand is K x ld row-major (ld its rows' count), else rows of ld = K. A warp's 32 copies
// are 8 rows (or 8 K) of 64 contiguous bytes each, and fill contiguous shared memory: no bank conflicts.
__device__ __forceinline__ void stage(uint32_t dst, const __nv_bfloat16* src, int ld, int rows, int r0, int limit,
                                      int k0, int kw, bool mn) {
    const int kc = kw / 8, sbo = kc * 128;
    const int inner = mn ? rows / 8 : kc, outer = mn ? kw : rows;  // 16-byte pieces of a source line; source lines
    const int spans = (inner + 3) / 4, items = spans * outer * 4;
    for (int idx = threadIdx.x; idx < items; idx += GEMM_THREADS) {
        const int lane = idx & 31, at = idx >> 5;
        const int line = (at / spans) * 8 + (lane & 7), piece = (at % spans) * 4 + (lane >> 3);
        if (piece >= inner) continue;
        if (mn) {
            const int r = r0 + piece * 8;
            copy16(dst + piece * sbo + (line >> 3) * 128 + (line & 7) * 16,
                   src + (r < limit ? (size_t)(k0 + line) * ld + r : 0), r < limit);
        } else {
            const int r = r0 + line;
            copy16(dst + (line >> 3) * sbo + piece * 128 + (line & 7) * 16,
                   src + (r < limit ? (size_t)r * ld + k0 + piece * 8 : 0), r < limit);
        }
    }
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// The row of the data set that row r of a batch is: its own, or the one this step's draw names.
__device__ __forceinline__ int64_t batch_row(const W2BMlpOp& G, int r) {
    return G.rows ? G.rows[(G.step ? *G.step : 0) * G.batch + r] : r;
}

// stage for the network's input: FP32 rows (the batch's rows of the data set, zero past its valid ones), rounded to
// BF16; the first column of CTAs also writes them out, for the backward pass.
__device__ __forceinline__ void stage_input(uint8_t* dst, const W2BMlpOp& G, int m0, int k0, int kw, bool write) {
    const int kc = kw / 8, sbo = kc * 128;
    for (int idx = threadIdx.x; idx < GEMM_M * kc; idx += GEMM_THREADS) {
        const int r = idx / kc, c = idx - r * kc;
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        if (m0 + r < G.valid) {
            const float4* x = reinterpret_cast<const float4*>(G.x + batch_row(G, m0 + r) * G.k + k0 + c * 8);
            lo = x[0];
            hi = x[1];
        }
        const uint4 v = make_uint4(pack2(lo.x, lo.y), pack2(lo.z, lo.w), pack2(hi.x, hi.y), pack2(hi.z, hi.w));
        *reinterpret_cast<uint4*>(dst + (r >> 3) * sbo + c * 128 + (r & 7) * 16) = v;
        if (write && m0 + r < G.m)
            *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(G.h0) + (size_t)(m0 + r) * G.k + k0 + c * 8) = v;
    }
}

// One Adam step of one weight (as adam_kernel takes it).
__device__ __forceinline__ void adam_one(float& w, float& m, float& v, float gi, float lr_t, float b1, float b2,
                                         float eps) {
    m = b1 * m + (1.0f - b1) * gi;
    v = b2 * v + (1.0f - b2) * gi * gi;
    w = w - lr_t * m / (sqrtf(v) + eps);
}

struct MlpGroup {
    W2BMlpOp op[W2B_MLP_OPS_MAX];
    int first[W2B_MLP_OPS_MAX + 1];  // each product's first CTA
    int count;
};

__global__ void __launch_bounds__(GEMM_THREADS) mlp_kernel(const __grid_constant__ MlpGroup P, int32_t* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ double red[GEMM_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int o = 0;
    while (o + 1 < P.count && (int)blockIdx.x >= P.first[o + 1]) ++o;
    const W2BMlpOp& G = P.op[o];
    const int M = G.m, N = G.n, K = G.k;
    const int ntn = (N + GEMM_N - 1) / GEMM_N;
    const int tile = (int)blockIdx.x - P.first[o];
    const int m0 = tile / ntn * GEMM_M, n0 = tile % ntn * GEMM_N;
    const int nt = N - n0 < GEMM_N ? N - n0 : GEMM_N;
    uint8_t* sA = smem;
    uint8_t* sB = smem + GEMM_M * GEMM_KC * 2;
    constexpr uint32_t NCOLS = 32;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(NCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    // instruction descriptor: FP32 accumulator, BF16 A and B, their orders, N / 8, M / 16
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((G.a_mn ? 1u : 0u) << 15) |
                           ((G.b_mn ? 1u : 0u) << 16) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(GEMM_M >> 4) << 24);
    const bool bias_grad = G.gb && n0 == 0;  // the column sums of A (K x M), rows in order
    float gb = 0.0f;
    uint32_t phase = 0;
    bool ok = true;
    for (int k0 = 0; k0 < K && ok; k0 += GEMM_KC) {
        const int kw = K - k0 < GEMM_KC ? K - k0 : GEMM_KC;  // this chunk's K, a multiple of 16
        const uint32_t sbo = (uint32_t)(kw / 8) * 128u;
        stage(smem_u32(sB), static_cast<const __nv_bfloat16*>(G.b), G.b_mn ? N : K, nt, n0, N, k0, kw, G.b_mn);
        if (G.x)
            stage_input(sA, G, m0, k0, kw, n0 == 0 && G.h0);
        else
            stage(smem_u32(sA), static_cast<const __nv_bfloat16*>(G.a), G.a_mn ? M : K, GEMM_M, m0, M, k0, kw, G.a_mn);
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async();  // these writes, before the tensor cores read the tiles
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
            for (int s = 0; s < kw / 16; ++s) {
                const uint64_t da = umma_desc(a0 + s * 256, 128, sbo);
                const uint64_t db = umma_desc(b0 + s * 256, 128, sbo);
                const uint32_t acc = (k0 > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&bar))
                         : "memory");
        }
        if (bias_grad && tid >= GEMM_M) {
            const int r = tid - GEMM_M;
            const __nv_bfloat16* col = reinterpret_cast<const __nv_bfloat16*>(sA + (r >> 3) * sbo) + (r & 7);
#pragma unroll 16
            for (int kk = 0; kk < kw; ++kk) gb += __bfloat162float(col[(kk >> 3) * 64 + (kk & 7) * 8]);
        }
        ok = mbar_wait(&bar, phase);
        if (!ok) mbar_wait(&bar, phase);  // once more for the MMAs in flight before anything is freed
        phase ^= 1u;
        ok = !__syncthreads_or(!ok);
        tc_fence_after();
    }
    if (ok) {
        // the tile through shared memory, so that the epilogue's loads and stores are whole row segments
        constexpr int PITCH = GEMM_N + 4;
        float* acc = reinterpret_cast<float*>(smem);
        const int c1 = (warp >> 2) * (nt / 2);  // this warp's columns of the tile: nt / 2 of them, 8 or 16
        for (int c = c1; c < c1 + nt / 2; c += 8) {
            uint32_t u[8];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            uint4* to = reinterpret_cast<uint4*>(acc + ((warp & 3) * 32 + lane) * PITCH + c);
            to[0] = make_uint4(u[0], u[1], u[2], u[3]);
            to[1] = make_uint4(u[4], u[5], u[6], u[7]);
        }
        __syncthreads();
        const float lr = G.lr_table ? G.lr_table[*G.step] : G.lr;
        double loss = 0.0;
        const int quads = nt / 4;
#pragma unroll 4
        for (int idx = tid; idx < GEMM_M * quads; idx += GEMM_THREADS) {
            const int r = idx / quads, row = m0 + r, col = n0 + (idx - r * quads) * 4;
            if (row >= M) continue;
            float v[4];
            const float4 q = *reinterpret_cast<const float4*>(acc + r * PITCH + col - n0);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
            if (G.bias)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += G.bias[col + j];
            const size_t at = (size_t)row * N + col;
            if (G.w) {  // the gradient of four weights: their Adam step
                const float4 w4 = *reinterpret_cast<const float4*>(G.w + at);
                const float4 m4 = *reinterpret_cast<const float4*>(G.mw + at);
                const float4 v4 = *reinterpret_cast<const float4*>(G.vw + at);
                float w[4] = {w4.x, w4.y, w4.z, w4.w}, m[4] = {m4.x, m4.y, m4.z, m4.w}, s[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) adam_one(w[j], m[j], s[j], v[j], lr, G.b1, G.b2, G.eps);
                *reinterpret_cast<float4*>(G.w + at) = make_float4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<float4*>(G.mw + at) = make_float4(m[0], m[1], m[2], m[3]);
                *reinterpret_cast<float4*>(G.vw + at) = make_float4(s[0], s[1], s[2], s[3]);
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(G.wb) + at) =
                    make_uint2(pack2(w[0], w[1]), pack2(w[2], w[3]));
            }
            if (G.c) {
                if (!((uintptr_t)G.c & 15)) {
                    *reinterpret_cast<float4*>(G.c + at) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
                    for (int j = 0; j < 4; ++j) G.c[at + j] = v[j];
                }
            }
            if (G.h) {  // the loss's gradient, the gradient behind an activation, or the next layer's input (relu)
                if (G.t) {
                    float4 t = make_float4(v[0], v[1], v[2], v[3]);
                    if (row < G.valid) t = *reinterpret_cast<const float4*>(G.t + batch_row(G, row) * N + col);
                    const float e[4] = {v[0] - t.x, v[1] - t.y, v[2] - t.z, v[3] - t.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        loss += row < G.valid ? (double)e[j] * (double)e[j] : 0.0;
                        v[j] = row < G.valid ? G.scale * e[j] : 0.0f;
                    }
                } else {
                    const float4 z = G.z ? *reinterpret_cast<const float4*>(G.z + at) : make_float4(v[0], v[1], v[2], v[3]);
                    v[0] = z.x > 0.0f ? v[0] : 0.0f;
                    v[1] = z.y > 0.0f ? v[1] : 0.0f;
                    v[2] = z.z > 0.0f ? v[2] : 0.0f;
                    v[3] = z.w > 0.0f ? v[3] : 0.0f;
                }
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(G.h) + at) =
                    make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
            }
        }
        if (G.t) {  // the CTA's share of the squared error
            for (int q = 16; q > 0; q >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, q);
            if (lane == 0) red[warp] = loss;
            __syncthreads();
            if (tid == 0) {
                for (int q = 1; q < GEMM_THREADS / 32; ++q) loss += red[q];
                G.partial[tile] = loss;
            }
        }
        if (bias_grad && tid >= GEMM_M && m0 + tid - GEMM_M < M) {
            const int r = m0 + tid - GEMM_M;
            if (G.w)
                adam_one(G.gb[r], G.mb[r], G.vb[r], gb, lr, G.b1, G.b2, G.eps);
            else
                G.gb[r] = gb;
        }
    } else if (tid == 0) {
        atomicExch(status, W2B_ETIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS) : "memory");
    }
}

// The end of a training step: its loss (the partial sums in order, over the outputs' count) into loss[*step],
// and the step counter moved on.
__global__ void mlp_tick_kernel(const double* __restrict__ partial, int n, double count, double* __restrict__ loss,
                                int64_t* __restrict__ step) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += partial[i];
    loss[*step] = s / count;
    *step += 1;
}

// The products of one launch; W2B_EINVAL if the shapes, orders or alignments are not what the kernel takes.
static int mlp_group(const W2BMlpOp* ops, int count, MlpGroup& P) {
    memset(&P, 0, sizeof(P));
    P.count = count;
    auto off = [](const void* p) { return ((uintptr_t)p & 15) != 0; };
    for (int i = 0; i < count; ++i) {
        const W2BMlpOp& G = ops[i];
        if (G.m < 1 || G.n < 16 || G.n > 256 || G.n % 16 || G.k < 16 || G.k % 16 || !G.b || off(G.b)) return W2B_EINVAL;
        if (G.x ? off(G.x) || off(G.h0) || G.a_mn : !G.a || off(G.a) || (G.a_mn && G.m % 8)) return W2B_EINVAL;
        if (off(G.h) || off(G.z) || off(G.t) || off(G.w) || off(G.mw) || off(G.vw) || off(G.wb)) return W2B_EINVAL;
        if ((G.t && (!G.partial || !G.h)) || (G.rows && G.batch < 1) || (G.lr_table && !G.step))
            return W2B_EINVAL;
        if (G.w && (!G.mw || !G.vw || !G.wb || (G.gb && (!G.mb || !G.vb)))) return W2B_EINVAL;
        if (G.gb && !G.a_mn) return W2B_EINVAL;
        P.op[i] = G;
        P.first[i + 1] = P.first[i] + (G.m + GEMM_M - 1) / GEMM_M * ((G.n + GEMM_N - 1) / GEMM_N);
    }
    return W2B_OK;
}

static int mlp_status(cudaError_t e) {
    if (e == cudaSuccess) return W2B_OK;
    fprintf(stderr, "libwadi_b200: mlp_kernel: %s\n", cudaGetErrorString(e));
    return W2B_ECUDA;
}

static int launch_mlp(const W2BMlpOp* ops, int count, int32_t* status, cudaStream_t s) {
    MlpGroup P;
    const int st = mlp_group(ops, count, P);
    if (st != W2B_OK) return st;
    if (cudaFuncSetAttribute(mlp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM) != cudaSuccess)
        return W2B_ECUDA;
    mlp_kernel<<<P.first[count], GEMM_THREADS, GEMM_SMEM, s>>>(P, status);
    return mlp_status(cudaGetLastError());
}

// ------------------------------------------------------------------ element-wise kernels of training

// out = bf16(relu(z)) (relu = 1) or bf16(z) (relu = 0)
__global__ void bf16_act_kernel(const float* __restrict__ z, int64_t n, int relu, __nv_bfloat16* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float v = z[i];
        out[i] = __float2bfloat16_rn(relu && !(v > 0.0f) ? 0.0f : v);
    }
}

// dz = bf16(g * [z > 0])
__global__ void relu_back_kernel(const float* __restrict__ g, const float* __restrict__ z, int64_t n,
                                 __nv_bfloat16* __restrict__ dz) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dz[i] = __float2bfloat16_rn(z[i] > 0.0f ? g[i] : 0.0f);
}

// xt (cols x rows) = x^T (x: rows x cols), BF16; zero-padded to rows_pad columns of xt
__global__ void transpose_bf16_kernel(const __nv_bfloat16* __restrict__ x, int rows, int cols, int rows_pad,
                                      __nv_bfloat16* __restrict__ xt) {
    __shared__ __nv_bfloat16 tile[32][33];
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = r0 + j, c = c0 + threadIdx.x;
        tile[j][threadIdx.x] = (r < rows && c < cols) ? x[(size_t)r * cols + c] : __float2bfloat16_rn(0.0f);
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int c = c0 + j, r = r0 + threadIdx.x;
        if (c < cols && r < rows_pad) xt[(size_t)c * rows_pad + r] = tile[threadIdx.x][j];
    }
}

// dy = bf16(scale (y - t)) over the m valid rows (zero for padded rows), and the loss partials sum (y - t)^2 in FP64
__global__ void mse_grad_kernel(const float* __restrict__ y, const float* __restrict__ t, int m, int m_pad, int n,
                                float scale, __nv_bfloat16* __restrict__ dy, double* __restrict__ partial) {
    __shared__ double red[256];
    double acc = 0.0;
    const int64_t total = (int64_t)m_pad * n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        float g = 0.0f;
        if (i / n < m) {
            const float d = y[i] - t[i];
            acc += (double)d * (double)d;
            g = scale * d;
        }
        dy[i] = __float2bfloat16_rn(g);
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// out[c] = sum over rows of bf16 x[r][c], FP32, rows in order
__global__ void colsum_kernel(const __nv_bfloat16* __restrict__ x, int rows, int cols, float* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    float s = 0.0f;
    for (int r = 0; r < rows; ++r) s += __bfloat162float(x[(size_t)r * cols + c]);
    out[c] = s;
}

// Adam on FP32 weights (bias-corrected steps lr_t = lr sqrt(1 - b2^t) / (1 - b1^t)), and their BF16 copy. With
// lr_table, the step size is lr_table[*step], read on the device (a captured training step replays with each step's
// own size).
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int64_t n, float lr_t, const float* __restrict__ lr_table,
                            const int64_t* __restrict__ step, float b1, float b2, float eps,
                            __nv_bfloat16* __restrict__ wb) {
    if (lr_table) lr_t = lr_table[*step];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        adam_one(w[i], m[i], v[i], gi, lr_t, b1, b2, eps);
        if (wb) wb[i] = __float2bfloat16_rn(w[i]);
    }
}

}  // namespace w2b

using namespace w2b;

extern "C" {

int32_t w2b_mma_gemm(const void* a, const void* b, int32_t m, int32_t n, int32_t k, const float* bias, float* c,
                     int32_t* status, void* stream) {
    if (!a || !b || !c || !status || m < 1 || n < 16 || n > 256 || n % 16 || k < 16 || k % 16) return W2B_EINVAL;
    if (((uintptr_t)a & 15) || ((uintptr_t)b & 15)) return W2B_EINVAL;
    W2BMlpOp G;
    memset(&G, 0, sizeof(G));
    G.a = a;
    G.b = b;
    G.m = m;
    G.n = n;
    G.k = k;
    G.bias = bias;
    G.c = c;
    return launch_mlp(&G, 1, status, (cudaStream_t)stream);
}

int32_t w2b_mlp_ops(const W2BMlpOp* ops, int32_t count, int32_t* status, void* stream) {
    if (!ops || !status || count < 1 || count > W2B_MLP_OPS_MAX) return W2B_EINVAL;
    return launch_mlp(ops, count, status, (cudaStream_t)stream);
}

int32_t w2b_mlp_train(const W2BMlpOp* ops, const int32_t* sizes, int32_t launches, int32_t iters,
                      const double* partial, int32_t n, double count, double* loss, int64_t* step, int32_t* status,
                      void* stream) {
    if (!ops || !sizes || launches < 1 || iters < 0 || !partial || n < 1 || !(count > 0.0) || !loss || !step || !status)
        return W2B_EINVAL;
    try {
        std::vector<MlpGroup> groups(launches);
        for (int l = 0; l < launches; ops += sizes[l], ++l) {
            if (sizes[l] < 1 || sizes[l] > W2B_MLP_OPS_MAX) return W2B_EINVAL;
            const int st = mlp_group(ops, sizes[l], groups[l]);
            if (st != W2B_OK) return st;
        }
        if (cudaFuncSetAttribute(mlp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM) != cudaSuccess)
            return W2B_ECUDA;
        cudaStream_t s = (cudaStream_t)stream;
        for (int it = 0; it < iters; ++it) {
            for (const MlpGroup& P : groups) mlp_kernel<<<P.first[P.count], GEMM_THREADS, GEMM_SMEM, s>>>(P, status);
            mlp_tick_kernel<<<1, 1, 0, s>>>(partial, n, count, loss, step);
            const int st = mlp_status(cudaGetLastError());
            if (st != W2B_OK) return st;
        }
    } catch (const std::bad_alloc&) {
        return W2B_EINVAL;
    }
    return W2B_OK;
}

int32_t w2b_mlp_tick(const double* partial, int32_t n, double count, double* loss, int64_t* step, void* stream) {
    if (!partial || !loss || !step || n < 1 || !(count > 0.0)) return W2B_EINVAL;
    mlp_tick_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(partial, n, count, loss, step);
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_bf16_act(const float* z, int64_t n, int32_t relu, void* out, void* stream) {
    if (!z || !out || n < 0) return W2B_EINVAL;
    bf16_act_kernel<<<296, 256, 0, (cudaStream_t)stream>>>(z, n, relu, static_cast<__nv_bfloat16*>(out));
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_relu_back(const float* g, const float* z, int64_t n, void* dz, void* stream) {
    if (!g || !z || !dz || n < 0) return W2B_EINVAL;
    relu_back_kernel<<<296, 256, 0, (cudaStream_t)stream>>>(g, z, n, static_cast<__nv_bfloat16*>(dz));
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_transpose_bf16(const void* x, int32_t rows, int32_t cols, int32_t rows_pad, void* xt, void* stream) {
    if (!x || !xt || rows < 1 || cols < 1 || rows_pad < rows) return W2B_EINVAL;
    const dim3 grid((cols + 31) / 32, (rows_pad + 31) / 32);
    transpose_bf16_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>(
        static_cast<const __nv_bfloat16*>(x), rows, cols, rows_pad, static_cast<__nv_bfloat16*>(xt));
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_mse_grad(const float* y, const float* t, int32_t m, int32_t m_pad, int32_t n, float scale, void* dy,
                     double* partial, void* stream) {
    if (!y || !t || !dy || !partial || m < 0 || m_pad < m || n < 1) return W2B_EINVAL;
    mse_grad_kernel<<<64, 256, 0, (cudaStream_t)stream>>>(y, t, m, m_pad, n, scale, static_cast<__nv_bfloat16*>(dy),
                                                          partial);
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_colsum_bf16(const void* x, int32_t rows, int32_t cols, float* out, void* stream) {
    if (!x || !out || rows < 0 || cols < 1) return W2B_EINVAL;
    colsum_kernel<<<(cols + 127) / 128, 128, 0, (cudaStream_t)stream>>>(static_cast<const __nv_bfloat16*>(x), rows,
                                                                        cols, out);
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_adam(float* w, const float* g, float* m, float* v, int64_t n, float lr_t, float b1, float b2, float eps,
                 void* wb, void* stream) {
    if (!w || !g || !m || !v || n < 0) return W2B_EINVAL;
    adam_kernel<<<296, 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr_t, nullptr, nullptr, b1, b2, eps,
                                                       static_cast<__nv_bfloat16*>(wb));
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

int32_t w2b_adam_table(float* w, const float* g, float* m, float* v, int64_t n, const float* lr_table,
                       const int64_t* step, float b1, float b2, float eps, void* wb, void* stream) {
    if (!w || !g || !m || !v || !lr_table || !step || n < 0) return W2B_EINVAL;
    adam_kernel<<<296, 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, 0.0f, lr_table, step, b1, b2, eps,
                                                       static_cast<__nv_bfloat16*>(wb));
    return cudaGetLastError() == cudaSuccess ? W2B_OK : W2B_ECUDA;
}

}  // extern "C"
