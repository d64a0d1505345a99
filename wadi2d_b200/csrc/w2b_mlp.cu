// The surrogate's network on the tensor cores: C = A B^T with BF16 operands and an FP32 accumulator in tensor memory
// (tcgen05.mma, kind::f16, a CTA a tile of 64 or 128 rows), and the element-wise kernels of training (activation, its
// gradient, transposes, the mean-square-error gradient, column sums, Adam).
//
// The products: C (M x N) = A B^T, 16 <= N <= 256, N and K multiples of 16, each operand K-major (row-major M x K or
// N x K) or MN-major (row-major K x M or K x N: what a backward pass has in hand, so nothing is transposed in memory).
// They are a few megaflops each, so latency bounds them: launches, one trip to L2 for the operands, one for the
// epilogue's. A CTA of 8 warps therefore takes a tile of 64 x 32 (a product of 256 x 256 is 32 CTAs), all of a K
// chunk's copies (cp.async, 16 B each) in flight at once, and the element-wise work that follows a product (bias and
// activation, the loss gradient, the activation's gradient, bias gradients, Adam) is its epilogue. A 256 x 256 x 256
// product takes 7.8 us where a CTA a 128-row tile, staging 128 of K at a time by loads through registers with
// 8-way bank conflicts, took 39 us; a training step at a batch of 256 is 50 us (mlp_train_kernel; as 9 launches 94 us)
// instead of 50 launches and 700 us.
// Operands sit in shared memory in the canonical layout without swizzle: core matrices of 8 rows of 16 bytes (K-major:
// 8 rows of 8 K; MN-major: 8 K of 8 rows), core_strides apart. Thread 0 issues one MMA per 16 of K against the
// accumulator in tensor memory and commits it to an mbarrier; the CTA waits (bounded) before the next chunk overwrites
// the tiles. The epilogue reads the accumulator with tcgen05.ld.32x32b (warp w sees tensor-memory lanes 32 (w mod 4) ..
// + 31, one row a lane, of a tile of 64 rows in the first 16 of them, and takes half of the columns).
// A wait that gives up sets the status word, waits once more for the MMAs in flight, frees the tensor memory and
// returns.
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "w2b_common.cuh"
#include "w2b_loop.cuh"
#include "w2b_tma.cuh"

namespace w2b {

constexpr int GEMM_N = 32;  // a tile's columns; its rows (TM) are 64 or 128: tile_rows
constexpr int GEMM_KC = 256;  // K staged a chunk at a time
constexpr int GEMM_THREADS = 256;
// bytes of `rows` rows of an operand in shared memory (core_strides; the other order takes less)
__host__ __device__ constexpr int gemm_bytes(int rows) { return rows / 8 * (GEMM_KC / 8) * 144; }
__host__ __device__ constexpr int gemm_smem(int tm) { return gemm_bytes(tm) + gemm_bytes(GEMM_N); }  // 54 or 90 KB: two CTAs a SM

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

// Where an operand's core matrices lie in shared memory: their stride from one 8 of K to the next (lead) and from 8 rows
// to the next (step), for a chunk of kc pieces of 8 K. A warp copies whole source lines, which run along K (K-major) or
// along the rows (MN-major): the stride in that direction is 16 bytes over a multiple of 128, so that a line's pieces
// fall into different banks.
struct CoreStrides {
    int lead, step;
};
__device__ __forceinline__ CoreStrides core_strides(int kc, bool mn) {
    return mn ? CoreStrides{128, kc * 128 + 16} : CoreStrides{144, kc * 144};
}

// A K chunk (kw of it from k0) of `rows` rows of an operand, from row r0 on, into shared memory; rows at or past
// `limit` are zero. mn: the operand is K x ld row-major (ld its rows' count), else rows of ld = K. The threads take a
// line's 16-byte pieces one after another, line after line, stepped without a division.
__device__ __forceinline__ void stage(uint32_t dst, const __nv_bfloat16* src, int ld, int rows, int r0, int limit,
                                      int k0, int kw, bool mn) {
    const CoreStrides S = core_strides(kw / 8, mn);
    const int inner = (mn ? rows : kw) / 8, lines = mn ? kw : rows;
    const int across = mn ? S.step : S.lead, down = mn ? S.lead : S.step;  // from a piece, from 8 lines to the next
    const int by = GEMM_THREADS / inner, rest = GEMM_THREADS - by * inner;
    int line = threadIdx.x / inner, piece = threadIdx.x - line * inner;
    const __nv_bfloat16* base = src + (size_t)(mn ? k0 : r0) * ld + (mn ? r0 : k0);
    while (line < lines) {
        const bool valid = (mn ? r0 + piece * 8 : r0 + line) < limit;
        copy16(dst + piece * across + (line >> 3) * down + (line & 7) * 16,
               valid ? base + (size_t)line * ld + piece * 8 : src, valid);
        line += by;
        piece += rest;
        if (piece >= inner) piece -= inner, ++line;
    }
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// The row of the data set that row r of a batch is: its own, or the one this step's draw names.
__device__ __forceinline__ int64_t batch_row(const W2BMlpOp& G, int64_t at, int r) {
    return G.rows ? G.rows[at * G.batch + r] : r;
}

// stage for the network's input: FP32 rows (the batch's rows of the data set, zero past its valid ones), rounded to
// BF16; the first column of CTAs also writes them out, for the backward pass.
template <int TM>
__device__ __forceinline__ void stage_input(uint8_t* dst, const W2BMlpOp& G, int64_t at, int m0, int k0, int kw,
                                            bool write) {
    const int kc = kw / 8;
    const CoreStrides S = core_strides(kc, false);
    for (int idx = threadIdx.x; idx < TM * kc; idx += GEMM_THREADS) {
        const int r = idx / kc, c = idx - r * kc;
        float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
        if (m0 + r < G.valid) {
            const float4* x = reinterpret_cast<const float4*>(G.x + batch_row(G, at, m0 + r) * G.k + k0 + c * 8);
            lo = x[0];
            hi = x[1];
        }
        const uint4 v = make_uint4(pack2(lo.x, lo.y), pack2(lo.z, lo.w), pack2(hi.x, hi.y), pack2(hi.z, hi.w));
        *reinterpret_cast<uint4*>(dst + (r >> 3) * S.step + c * S.lead + (r & 7) * 16) = v;
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

// Products of one launch: their first tiles, and where the last one's end.
struct MlpGroup {
    W2BMlpOp op[W2B_MLP_OPS_MAX];
    int first[W2B_MLP_OPS_MAX + 1];  // for tiles of tm rows
    int count, tm;
};

// What a CTA works in: shared memory (B's tile, then A's), the barrier its MMAs commit to with its phase, a scratch of
// one double a warp, and its accumulator in tensor memory.
struct MlpCta {
    uint8_t* smem;
    uint64_t* bar;
    double* red;
    uint32_t phase, tmem;
};
constexpr uint32_t MLP_COLS = 32;

// Tensor memory and the barrier of a CTA; and back (every thread, on every way out).
__device__ __forceinline__ void mlp_begin(MlpCta& C, uint32_t* tmem_base) {
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base)),
                     "r"(MLP_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        mbar_init(C.bar, 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    C.phase = 0;
    C.tmem = *tmem_base;
}
__device__ __forceinline__ void mlp_end(MlpCta& C) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(C.tmem), "r"(MLP_COLS) : "memory");
}

// The first K chunk of B of a product's tile into shared memory (asynchronously).
__device__ __forceinline__ void stage_b(const MlpCta& C, const W2BMlpOp& G, int tile, int k0) {
    const int ntn = (G.n + GEMM_N - 1) / GEMM_N, n0 = tile % ntn * GEMM_N;
    const int nt = G.n - n0 < GEMM_N ? G.n - n0 : GEMM_N, kw = G.k - k0 < GEMM_KC ? G.k - k0 : GEMM_KC;
    stage(smem_u32(C.smem), static_cast<const __nv_bfloat16*>(G.b), G.b_mn ? G.n : G.k, nt, n0, G.n, k0, kw, G.b_mn);
}

// One tile of a product. at: the training step (what *G.step holds); b_staged: stage_b has begun for it. False: a wait
// gave up (reported; the caller frees the tensor memory and leaves).
template <int TM>
__device__ __forceinline__ bool mlp_tile(MlpCta& C, const W2BMlpOp& G, int tile, int64_t at, bool b_staged,
                                         int32_t* status) {
    uint8_t* const smem = C.smem;
    double* const red = C.red;
    const uint32_t tmem = C.tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int M = G.m, N = G.n, K = G.k;
    const int ntn = (N + GEMM_N - 1) / GEMM_N;
    const int m0 = tile / ntn * TM, n0 = tile % ntn * GEMM_N;
    const int nt = N - n0 < GEMM_N ? N - n0 : GEMM_N;
    uint8_t* sB = smem;
    uint8_t* sA = smem + gemm_bytes(GEMM_N);
    // instruction descriptor: FP32 accumulator, BF16 A and B, their orders, N / 8, M / 16
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((G.a_mn ? 1u : 0u) << 15) |
                           ((G.b_mn ? 1u : 0u) << 16) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    const bool bias_grad = G.gb && n0 == 0;  // the column sums of A (K x M), rows in order
    float gb = 0.0f;
    bool ok = true;
    // what the epilogue reads: a thread's quads of four columns, 32 rows (or 64) apart, the same columns in each; loaded
    // while A lands
    const int shift = nt == GEMM_N ? 3 : 2;  // quads of columns in a row of the tile: 8, or 4
    const int c = (tid & ((1 << shift) - 1)) * 4;
    constexpr int QUADS = TM * GEMM_N / 4 / GEMM_THREADS;
    float4 z[QUADS], m4[QUADS], v4[QUADS];
    float bias[4], lr = G.lr;
    const float* zs = G.w ? G.w : (G.h && !G.t ? G.z : nullptr);
    auto ahead = [&] {
        if (G.lr_table) lr = G.lr_table[at];
        if (G.bias)
#pragma unroll
            for (int j = 0; j < 4; ++j) bias[j] = G.bias[n0 + c + j];
#pragma unroll
        for (int x = 0; x < QUADS; ++x) {
            const int r = (tid + x * GEMM_THREADS) >> shift, row = m0 + r;
            if (r >= TM || row >= M) continue;
            const size_t e0 = (size_t)row * N + n0 + c;
            if (zs) z[x] = *reinterpret_cast<const float4*>(zs + e0);
            if (G.w) {
                m4[x] = *reinterpret_cast<const float4*>(G.mw + e0);
                v4[x] = *reinterpret_cast<const float4*>(G.vw + e0);
            }
            if (G.t && row < G.valid)
                z[x] = *reinterpret_cast<const float4*>(G.t + batch_row(G, at, row) * N + n0 + c);
        }
    };
    for (int k0 = 0; k0 < K && ok; k0 += GEMM_KC) {
        const int kw = K - k0 < GEMM_KC ? K - k0 : GEMM_KC;  // this chunk's K, a multiple of 16
        const CoreStrides SA = core_strides(kw / 8, G.a_mn), SB = core_strides(kw / 8, G.b_mn);
        if (k0 > 0 || !b_staged) stage_b(C, G, tile, k0);
        if (G.x)
            stage_input<TM>(sA, G, at, m0, k0, kw, n0 == 0 && G.h0);
        else
            stage(smem_u32(sA), static_cast<const __nv_bfloat16*>(G.a), G.a_mn ? M : K, TM, m0, M, k0, kw, G.a_mn);
        if (k0 + GEMM_KC >= K) ahead();
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async();  // these writes, before the tensor cores read the tiles
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            // (a step of 16 K is two core matrices on; a descriptor's address field counts 16 bytes)
            const uint64_t a0 = umma_desc(smem_u32(sA), SA.lead, SA.step), b0 = umma_desc(smem_u32(sB), SB.lead, SB.step);
            for (int s = 0; s < kw / 16; ++s) {
                const uint64_t da = a0 + s * SA.lead / 8, db = b0 + s * SB.lead / 8;
                const uint32_t acc = (k0 > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(C.bar))
                         : "memory");
        }
        if (bias_grad && tid >= GEMM_THREADS - TM) {
            // a thread a row, in the order of K
            const int r = tid - (GEMM_THREADS - TM);
            const __nv_bfloat16* col = reinterpret_cast<const __nv_bfloat16*>(sA + (r >> 3) * SA.step) + (r & 7);
#pragma unroll 16
            for (int kk = 0; kk < kw; ++kk) gb += __bfloat162float(col[kk * 8]);
        }
        ok = mbar_wait(C.bar, C.phase);
        if (!ok) mbar_wait(C.bar, C.phase);  // once more for the MMAs in flight before anything is freed
        C.phase ^= 1u;
        ok = !__syncthreads_or(!ok);
        tc_fence_after();
    }
    if (ok) {
        // the tile through shared memory, so that the epilogue's loads and stores are whole row segments
        constexpr int PITCH = GEMM_N + 4;
        float* acc = reinterpret_cast<float*>(sA);
        const int c1 = (warp >> 2) * (nt / 2);  // this warp's columns of the tile: nt / 2 of them, 8 or 16
        for (int d = c1; d < c1 + nt / 2; d += 8) {
            uint32_t u[8];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)d));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (lane < TM / 4) {  // 64 rows are in the first 16 lanes of each warp's 32
                uint4* to = reinterpret_cast<uint4*>(acc + ((warp & 3) * (TM / 4) + lane) * PITCH + d);
                to[0] = make_uint4(u[0], u[1], u[2], u[3]);
                to[1] = make_uint4(u[4], u[5], u[6], u[7]);
            }
        }
        __syncthreads();
        double loss[TM / 64] = {};  // of each 64 rows: the sums are the same for either tile
#pragma unroll
        for (int x = 0; x < QUADS; ++x) {
            const int r = (tid + x * GEMM_THREADS) >> shift, row = m0 + r;
            if (r >= TM || row >= M) continue;
            const size_t e0 = (size_t)row * N + n0 + c;
            const float4 q = *reinterpret_cast<const float4*>(acc + r * PITCH + c);
            float v[4] = {q.x, q.y, q.z, q.w};
            if (G.bias)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += bias[j];
            if (G.w) {  // the gradient of four weights: their Adam step
                float w[4] = {z[x].x, z[x].y, z[x].z, z[x].w}, m[4] = {m4[x].x, m4[x].y, m4[x].z, m4[x].w};
                float s[4] = {v4[x].x, v4[x].y, v4[x].z, v4[x].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) adam_one(w[j], m[j], s[j], v[j], lr, G.b1, G.b2, G.eps);
                *reinterpret_cast<float4*>(G.w + e0) = make_float4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<float4*>(G.mw + e0) = make_float4(m[0], m[1], m[2], m[3]);
                *reinterpret_cast<float4*>(G.vw + e0) = make_float4(s[0], s[1], s[2], s[3]);
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(G.wb) + e0) =
                    make_uint2(pack2(w[0], w[1]), pack2(w[2], w[3]));
            }
            if (G.c) {
                if (!((uintptr_t)G.c & 15)) {
                    *reinterpret_cast<float4*>(G.c + e0) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
                    for (int j = 0; j < 4; ++j) G.c[e0 + j] = v[j];
                }
            }
            if (G.h) {  // the loss's gradient, the gradient behind an activation, or the next layer's input (relu)
                if (G.t) {
                    const float e[4] = {v[0] - z[x].x, v[1] - z[x].y, v[2] - z[x].z, v[3] - z[x].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const double sq = row < G.valid ? (double)e[j] * (double)e[j] : 0.0;
                        if (TM == 64 || r < 64)
                            loss[0] += sq;
                        else
                            loss[TM / 64 - 1] += sq;
                        v[j] = row < G.valid ? G.scale * e[j] : 0.0f;
                    }
                } else {
                    const float4 y = zs ? z[x] : make_float4(v[0], v[1], v[2], v[3]);
                    v[0] = y.x > 0.0f ? v[0] : 0.0f;
                    v[1] = y.y > 0.0f ? v[1] : 0.0f;
                    v[2] = y.z > 0.0f ? v[2] : 0.0f;
                    v[3] = y.w > 0.0f ? v[3] : 0.0f;
                }
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(G.h) + e0) =
                    make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
            }
        }
        if (G.t) {  // the CTA's share of the squared error
#pragma unroll
            for (int b = 0; b < TM / 64; ++b) {
                for (int q = 16; q > 0; q >>= 1) loss[b] += __shfl_down_sync(0xffffffffu, loss[b], q);
                if (lane == 0) red[b * (GEMM_THREADS / 32) + warp] = loss[b];
            }
            __syncthreads();
            if (tid < TM / 64 && m0 + tid * 64 < M) {
                const double* part = red + tid * (GEMM_THREADS / 32);
                double sum = part[0];
                for (int q = 1; q < GEMM_THREADS / 32; ++q) sum += part[q];
                G.partial[(m0 / 64 + tid) * ntn + n0 / GEMM_N] = sum;
            }
        }
        if (bias_grad && tid >= GEMM_THREADS - TM && m0 + tid - (GEMM_THREADS - TM) < M) {
            const int r = m0 + tid - (GEMM_THREADS - TM);
            if (G.w)
                adam_one(G.gb[r], G.mb[r], G.vb[r], gb, lr, G.b1, G.b2, G.eps);
            else
                G.gb[r] = gb;
        }
        tc_fence_before();
        __syncthreads();  // the accumulator and the tile in shared memory are read: the next tile may write them
        tc_fence_after();
    } else if (tid == 0) {
        atomicExch(status, W2B_ETIMEOUT);
    }
    return ok;
}

__device__ __forceinline__ const W2BMlpOp& mlp_op(const MlpGroup& P, int tile, int& local) {
    int o = 0;
    while (o + 1 < P.count && tile >= P.first[o + 1]) ++o;
    local = tile - P.first[o];
    return P.op[o];
}

template <int TM>
__global__ void __launch_bounds__(GEMM_THREADS) mlp_kernel(const __grid_constant__ MlpGroup P, int32_t* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ double red[TM / 64 * (GEMM_THREADS / 32)];
    MlpCta C{smem, &bar, red};
    mlp_begin(C, &tmem_base);
    int tile;
    const W2BMlpOp& G = mlp_op(P, blockIdx.x, tile);
    mlp_tile<TM>(C, G, tile, G.step ? *G.step : 0, false, status);
    mlp_end(C);
}

// Training steps in one cooperative launch: each step's groups of products in order, a grid barrier after each. A group is
// a few tiles and as kernels of their own cost 8.4 us and a gap of 1.8 each, most of it starting up; here a CTA keeps its
// tensor memory and its code, and while it waits at the barrier its next tile's B is on its way (b_early).
// A step at a batch of 256 (four products of 256 x 256 among them) is 8 groups and 50 us instead of 94. Of a group's 6 us
// 1.6 are A's 32 KB on their way from L2 (one SM takes in 26 B a clock), 0.9 the MMAs, 0.9 the epilogue, 2.2 the barrier.
constexpr int TRAIN_GROUPS_MAX = 12;
constexpr int TRAIN_ITERS_MAX = 512;  // steps a launch, so that none holds the GPU for long
struct MlpTrain {
    MlpGroup group[TRAIN_GROUPS_MAX];
    int groups, iters, partials;
    const double* partial;
    double count;
    double* loss;
    int64_t* step;
    int32_t* status;  // [1], [2]: the barrier's arrivals, the CTAs that have left
};
template <int TM>
__global__ void __launch_bounds__(GEMM_THREADS, 2) mlp_train_kernel(const __grid_constant__ MlpTrain T) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ double red[TM / 64 * (GEMM_THREADS / 32)];
    if (*T.status) return;  // a wait before this launch gave up: the barrier's counters may be anything
    MlpCta C{smem, &bar, red};
    mlp_begin(C, &tmem_base);
    const int64_t step0 = *T.step;
    uint32_t* const arrived = reinterpret_cast<uint32_t*>(T.status + 1);
    uint32_t met = 0;
    bool staged = false, ok = true;  // staged: the B of this CTA's first tile of the group has begun
    for (int it = 0; it < T.iters && ok; ++it) {
        for (int g = 0; g < T.groups && ok; ++g) {
            const MlpGroup& P = T.group[g];
            const int tiles = P.first[P.count];
            for (int x = blockIdx.x; x < tiles && ok; x += gridDim.x) {
                int tile;
                const W2BMlpOp& G = mlp_op(P, x, tile);
                ok = mlp_tile<TM>(C, G, tile, G.step ? step0 + it : 0, staged && x == (int)blockIdx.x, T.status);
            }
            if (ok && g == T.groups - 1 && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
                double s = 0.0;
                for (int i = 0; i < T.partials; ++i) s += __ldcg(T.partial + i);
                T.loss[step0 + it] = s / T.count;
            }
            if (!ok) break;
            ok = grid_barrier(arrived, T.status, met, [&] {
                const MlpGroup& Q = T.group[g + 1 < T.groups ? g + 1 : 0];
                staged = (int)blockIdx.x < Q.first[Q.count];
                if (!staged) return;
                int tile;
                const W2BMlpOp& G = mlp_op(Q, blockIdx.x, tile);
                staged = G.b_early;
                if (staged) stage_b(C, G, tile, 0);
            });
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (ok && threadIdx.x == 0 && atomicAdd(arrived + 1, 1u) == gridDim.x - 1) {  // the last CTA to leave
        *T.step = step0 + T.iters;
        arrived[0] = 0;
        arrived[1] = 0;
    }
    mlp_end(C);
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

// The tiles of a launch's products, at tm rows each.
static int tile_rows(MlpGroup& P, int tm) {
    P.tm = tm;
    for (int i = 0; i < P.count; ++i)
        P.first[i + 1] = P.first[i] + (P.op[i].m + tm - 1) / tm * ((P.op[i].n + GEMM_N - 1) / GEMM_N);
    return P.first[P.count];
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
        if (G.w && (G.h || G.t)) return W2B_EINVAL;
        if (G.gb && !G.a_mn) return W2B_EINVAL;
        P.op[i] = G;
    }
    tile_rows(P, 128);
    return W2B_OK;
}

static int mlp_status(cudaError_t e) {
    if (e == cudaSuccess) return W2B_OK;
    fprintf(stderr, "libwadi_b200: mlp_kernel: %s\n", cudaGetErrorString(e));
    return W2B_ECUDA;
}

// The rows of a tile: 64 while tiles of 128 would leave SMs without one, for a CTA is bound by what one SM takes in of A
// and by its share of the epilogue. A product of 256 x 256 x 256 takes 7.8 us against 8.7 (1024 rows 8.2
// against 9.2, 2304 rows the same 10.3), a training step at a batch of 256 50 us against 66, 1024 63 against 84, 2304 117
// against 121.
static int pick_rows(int tiles128, int* sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return tiles128 <= *sms ? 64 : 128;
}

template <int TM>
static cudaError_t launch_group(const MlpGroup& P, int32_t* status, cudaStream_t s) {
    const cudaError_t e =
        cudaFuncSetAttribute(mlp_kernel<TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem(TM));
    if (e != cudaSuccess) return e;
    mlp_kernel<TM><<<P.first[P.count], GEMM_THREADS, gemm_smem(TM), s>>>(P, status);
    return cudaGetLastError();
}

static int launch_group(MlpGroup& P, int32_t* status, cudaStream_t s) {
    int sms = 0;
    const int tm = pick_rows(tile_rows(P, 128), &sms);
    if (!tm) return W2B_ECUDA;
    tile_rows(P, tm);
    return mlp_status(tm == 64 ? launch_group<64>(P, status, s) : launch_group<128>(P, status, s));
}

static int launch_mlp(const W2BMlpOp* ops, int count, int32_t* status, cudaStream_t s) {
    MlpGroup P;
    const int st = mlp_group(ops, count, P);
    return st != W2B_OK ? st : launch_group(P, status, s);
}

// Every step of T in cooperative launches of at most TRAIN_ITERS_MAX.
template <int TM>
static int launch_train(MlpTrain& T, int iters, int sms, cudaStream_t s) {
    int widest = 1, occ = 0;
    for (int l = 0; l < T.groups; ++l) {
        const int tiles = tile_rows(T.group[l], TM);
        widest = tiles > widest ? tiles : widest;
    }
    // (the largest carveout, as the resident loop's: a SM set up for one of them has room for the other)
    if (cudaFuncSetAttribute(mlp_train_kernel<TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemm_smem(TM)) !=
            cudaSuccess ||
        cudaFuncSetAttribute(mlp_train_kernel<TM>, cudaFuncAttributePreferredSharedMemoryCarveout, 100) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mlp_train_kernel<TM>, GEMM_THREADS, gemm_smem(TM)) !=
            cudaSuccess)
        return mlp_status(cudaGetLastError());
    if (occ < 1) return W2B_ECUDA;
    const int ctas = widest < sms * occ ? widest : sms * occ;
    for (int done = 0; done < iters; done += T.iters) {
        T.iters = iters - done < TRAIN_ITERS_MAX ? iters - done : TRAIN_ITERS_MAX;
        void* params[] = {&T};
        const int st = mlp_status(
            launch_in_turn((const void*)mlp_train_kernel<TM>, ctas, GEMM_THREADS, params, gemm_smem(TM), occ, s));
        if (st != W2B_OK) return st;
    }
    return W2B_OK;
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
    cudaStream_t s = (cudaStream_t)stream;
    try {
        std::vector<MlpGroup> groups(launches);
        int widest = 1;
        bool counted = true;  // every product's step is this call's, or none
        bool summed = true;   // no loss in the last launch: its sums are there when that one begins
        for (int l = 0; l < launches; ops += sizes[l], ++l) {
            if (sizes[l] < 1 || sizes[l] > W2B_MLP_OPS_MAX) return W2B_EINVAL;
            const int st = mlp_group(ops, sizes[l], groups[l]);
            if (st != W2B_OK) return st;
            for (int o = 0; o < sizes[l]; ++o) {
                counted = counted && (!ops[o].step || ops[o].step == step);
                summed = summed && !(ops[o].t && l == launches - 1);
            }
            const int tiles = tile_rows(groups[l], 128);
            widest = tiles > widest ? tiles : widest;
        }
        if (!iters) return W2B_OK;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (mlp_status(cudaStreamIsCapturing(s, &cap)) != W2B_OK) return W2B_ECUDA;
        if (launches <= TRAIN_GROUPS_MAX && counted && summed && cap == cudaStreamCaptureStatusNone) {
            // one launch of every step, which counts the steps itself and adds up the loss beside the last group; a stream
            // being captured cannot wait for another stream's
            MlpTrain T;
            memset(&T, 0, sizeof(T));
            memcpy(T.group, groups.data(), sizeof(MlpGroup) * launches);
            T.groups = launches;
            T.partials = n;
            T.partial = partial;
            T.count = count;
            T.loss = loss;
            T.step = step;
            T.status = status;
            int sms = 0;
            const int tm = pick_rows(widest, &sms);
            if (!tm) return W2B_ECUDA;
            return tm == 64 ? launch_train<64>(T, iters, sms, s) : launch_train<128>(T, iters, sms, s);
        }
        for (int it = 0; it < iters; ++it) {
            for (MlpGroup& P : groups) {
                const int st = launch_group(P, status, s);
                if (st != W2B_OK) return st;
            }
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
