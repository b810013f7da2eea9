// The f32 matrix products of the path, behind the entry points rusty-backend's ComputeEngine exposes, and the f32 Linear
// with a LoRA branch that is built from them:
//   matmul     (WGSL matmul_tiled, kernels.wgsl:16-54)      out[M,N] = a[M,K] . b[K,N]
//   matmul_bt  (WGSL matmul_bt,    kernels.wgsl:234-242)    out[M,N] = a[M,K] . b[N,K]^T
//   Linear::forward with an adapter (rusty-graph/src/lib.rs:69-80)   y = x . W + (x . A) . B
//
// Numerics contract of the two matmuls: ONE accumulator per output, the products added in ascending k with fused
// multiply-add, exactly the shaders' order: bit-identical to the shader arithmetic evaluated with FMA contraction (which
// WGSL permits).  So K is never split: an output is a chain of K dependent FMAs, and a small product is bound by that
// chain and by the shared-memory pipe, not by arithmetic or HBM.
#include <cooperative_groups.h>

#include "internal.h"
#include "tc_common.cuh"

using namespace rusty;
using namespace rusty_tc;
namespace cg = cooperative_groups;

namespace {

// The adapter's second product rides behind the first as more k: y = [x | t] . [W ; B], t = x . A (rows r4 floats long,
// zeros behind the r real ones), B [r, N].  r = 0: none.
struct LoraTail {
    const float* t;
    const float* b;
    int r, r4;
};

// 16 (VEC) or 4 bytes global -> shared; bytes = 0: nothing is read, zeros are stored
template <bool VEC>
__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, uint32_t bytes) {
    if constexpr (VEC)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// ROWS x COLS floats of a row-major matrix into shared memory rows LDS_ floats apart, by T threads; what lies outside
// rows x cols becomes zero.  A thread's copies lie in one column and a fixed number of rows apart where the shape allows
// (16-byte copies always do), so that a copy costs one addition: with an address worked out per copy a row times 4096 x 4096
// took 36 us instead of 20.
template <bool VEC, int T, int ROWS, int COLS, int LDS_>
__device__ __forceinline__ void copy_tile(uint32_t dst, const float* src, uint32_t ld, uint32_t rows, uint32_t cols) {
    constexpr int W = VEC ? 4 : 1, PER_ROW = COLS / W, N_COPY = ROWS * PER_ROW;
    const int tid = threadIdx.x;
    if constexpr (T % PER_ROW == 0 && N_COPY % T == 0) {
        constexpr int STEP = T / PER_ROW;
        const uint32_t r0 = tid / PER_ROW, c0 = (tid % PER_ROW) * W;
        const float* p = src + (size_t)r0 * ld + c0;
        const size_t hop = (size_t)STEP * ld;
        uint32_t d = dst + (r0 * LDS_ + c0) * 4;
        const uint32_t bytes = c0 < cols ? 4 * W : 0;
        if (rows >= (uint32_t)ROWS) {
#pragma unroll
            for (int u = 0; u < N_COPY / T; ++u, p += hop, d += STEP * LDS_ * 4) cp_async<VEC>(d, p, bytes);
        } else {
#pragma unroll
            for (int u = 0; u < N_COPY / T; ++u, p += hop, d += STEP * LDS_ * 4) cp_async<VEC>(d, p, r0 + u * STEP < rows ? bytes : 0u);
        }
    } else {
        for (int i = tid; i < N_COPY; i += T) {
            const uint32_t r = i / PER_ROW, c = (i % PER_ROW) * W;
            const bool in = r < rows && c < cols;
            cp_async<VEC>(dst + (r * LDS_ + c) * 4, in ? src + (size_t)r * ld + c : src, in ? 4 * W : 0u);
        }
    }
}

// Shared-memory reads as volatile asm: written as plain loads they were moved down to their first use, which undid the reading
// ahead below.
__device__ __forceinline__ float4 lds_f4(const float* p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(smem_u32(p)));
    return v;
}
__device__ __forceinline__ float2 lds_f2(const float* p) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_u32(p)));
    return v;
}
__device__ __forceinline__ float lds_f1(const float* p) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(smem_u32(p)));
    return v;
}
// Global loads as volatile asm, for the same reason.
__device__ __forceinline__ float4 ldg_f4(const float* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
// two FMAs an instruction, each half rounded like fmaf
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void fma2(float& c0, float& c1, unsigned long long a, unsigned long long b) {
    unsigned long long c = pack2(c0, c1);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(c));
}

// A block's WM warps are stacked along M; a warp's lanes form LM rows x LN columns, a thread owns TM x TN outputs.  What bounds
// these kernels is the shared-memory pipe (counted on the device: a pass returns 128 bytes of distinct columns, 256 where the
// eight lanes of a quarter warp read the same address): per k a warp spends TM / 2 passes on a and TN on b for TM TN FMA
// instructions, of which an SM issues four a cycle.  Only 8 x 8 comes near the FMA rate; the small tiles exist because a small
// product has too few outputs to give every scheduler a warp of more than a few.
// K is walked in chunks of BK through a ring of ST chunks filled with cp.async; a sits in shared memory as [m][k] (padded
// rows), b as [k][n] or, NK, as [n][k].
template <int WM_, int LM_, int TM_, int TN_, int BK_, int ST_>
struct Tile {
    static constexpr int LM = LM_, LN = 32 / LM_, TM = TM_, TN = TN_, BK = BK_, ST = ST_;
    static constexpr int BM = WM_ * LM * TM, BN = LN * TN, THREADS = 32 * WM_;
    static constexpr int LDA = BK + 4;
    static constexpr int B_KN = BK * BN, B_NK = BN * LDA;   // floats of b in a chunk
};

template <typename TL, bool NK, bool VEC>
__global__ void __launch_bounds__(TL::THREADS, 1) matmul_f32_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out,
                                                                    uint32_t M, uint32_t K, uint32_t N, const LoraTail lora) {
    constexpr int BM = TL::BM, BN = TL::BN, TM = TL::TM, TN = TL::TN, BK = TL::BK, ST = TL::ST, T = TL::THREADS, LDA = TL::LDA;
    constexpr int BFL = NK ? TL::B_NK : TL::B_KN;
    extern __shared__ __align__(16) float mm_smem[];
    float* sa = mm_smem;                       // [ST][BM][LDA]
    float* sb = mm_smem + ST * BM * LDA;       // [ST][BK][BN] or [ST][BN][LDA]
    const int tid = threadIdx.x;
    constexpr int LM = TL::LM, LN = TL::LN;
    const int ln = (tid & 31) % LN, lm = (tid & 31) / LN;
    // this thread's rows: row0 + i * LM; its columns: four neighbours at a time, NK: j * LN + ln (both free of bank conflicts)
    const int row0 = (tid >> 5) * (LM * TM) + lm;
    auto col = [&](int j) { return NK ? j * LN + ln : (j / 4) * (LN * 4) + ln * (TN < 4 ? TN : 4) + j % 4; };
    const uint32_t n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int chunks_k = (int)((K + BK - 1) / BK), chunks = chunks_k + (lora.r + BK - 1) / BK;
    // No early launch_dependents here: grids of fewer blocks than SMs are common, and the next grid's blocks would pile up on
    // the idle SMs (back to back, 64 x 4096 x 4096 took 280 us instead of 105).  With an adapter the kernel in front of this
    // one only computes t, and it lets this one start after its own griddepcontrol.wait (lora_down_kernel): x and W are final
    // by then, so only the chunks that hold t have to wait for it.
    if (lora.r == 0) pdl_wait();
    auto fetch = [&](int c) {
        const uint32_t da = smem_u32(sa + (c % ST) * BM * LDA), db = smem_u32(sb + (c % ST) * BFL);
        if (c < chunks_k) {
            const uint32_t k0 = (uint32_t)c * BK;
            copy_tile<VEC, T, BM, BK, LDA>(da, a + (size_t)m0 * K + k0, K, M - m0, K - k0);
            if constexpr (NK) copy_tile<VEC, T, BN, BK, LDA>(db, b + (size_t)n0 * K + k0, K, N - n0, K - k0);
            else copy_tile<VEC, T, BK, BN, BN>(db, b + (size_t)k0 * N + n0, N, K - k0, N - n0);
        } else if (!NK && c < chunks) {
            if (c == chunks_k) pdl_wait();
            const uint32_t k0 = (uint32_t)(c - chunks_k) * BK;
            copy_tile<VEC, T, BM, BK, LDA>(da, lora.t + (size_t)m0 * lora.r4 + k0, lora.r4, M - m0, lora.r4 - k0);
            copy_tile<VEC, T, BK, BN, BN>(db, lora.b + (size_t)k0 * N + n0, N, lora.r - k0, N - n0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int c = 0; c < ST - 1; ++c) fetch(c);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();                       // chunk c has landed for everybody, and chunk c - 1 has been read by everybody
        fetch(c + ST - 1);
        const float* pa = sa + (c % ST) * BM * LDA + row0 * LDA;
        const float* pb = sb + (c % ST) * BFL;
        // shared memory -> registers two steps (of four k) ahead of the FMAs: the reads of a step keep the shared-memory pipe
        // busy for about the step's own time, so one step ahead would still wait for the trip itself
        float av[3][TM][4], bv[3][4][TN];
        auto load = [&](int k, float (&va)[TM][4], float (&vb)[4][TN]) {
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 v = lds_f4(pa + i * LM * LDA + k);
                va[i][0] = v.x; va[i][1] = v.y; va[i][2] = v.z; va[i][3] = v.w;
            }
            if constexpr (NK) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float4 v = lds_f4(pb + col(j) * LDA + k);
                    vb[0][j] = v.x; vb[1][j] = v.y; vb[2][j] = v.z; vb[3][j] = v.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (TN == 1) {
                        vb[q][0] = lds_f1(pb + (k + q) * BN + col(0));
                    } else if constexpr (TN == 2) {
                        const float2 v = lds_f2(pb + (k + q) * BN + col(0));
                        vb[q][0] = v.x; vb[q][1] = v.y;
                    } else {
#pragma unroll
                        for (int j = 0; j < TN; j += 4) {
                            const float4 v = lds_f4(pb + (k + q) * BN + col(j));
                            vb[q][j] = v.x; vb[q][j + 1] = v.y; vb[q][j + 2] = v.z; vb[q][j + 3] = v.w;
                        }
                    }
                }
            }
        };
        load(0, av[0], bv[0]);
        load(4, av[1], bv[1]);
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            const int cur = (k >> 2) % 3;
            if (k + 8 < BK) load(k + 8, av[(cur + 2) % 3], bv[(cur + 2) % 3]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    if constexpr (!NK && TN >= 4) {   // (NK: the two columns' values do not come in neighbouring registers)
                        const unsigned long long aa = pack2(av[cur][i][q], av[cur][i][q]);
#pragma unroll
                        for (int j = 0; j < TN; j += 2) fma2(acc[i][j], acc[i][j + 1], aa, pack2(bv[cur][q][j], bv[cur][q][j + 1]));
                    } else {
#pragma unroll
                        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[cur][i][q], bv[cur][q][j], acc[i][j]);
                    }
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const uint32_t gm = m0 + row0 + i * LM;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const uint32_t gn = n0 + col(j);
            if (gn < N) out[(size_t)gm * N + gn] = acc[i][j];
        }
    }
}

using TileRow = Tile<1, 1, 1, 1, 128, 6>;    //  1 x 32
using Tile4 = Tile<2, 2, 1, 2, 128, 4>;      //  4 x 32
using Tile8 = Tile<4, 2, 1, 2, 64, 8>;       //  8 x 32
using Tile16 = Tile<4, 2, 2, 2, 64, 8>;      // 16 x 32
using Tile32 = Tile<4, 4, 2, 4, 64, 4>;      // 32 x 32
using Tile64 = Tile<4, 4, 4, 4, 32, 4>;      // 64 x 32
using TileBig = Tile<2, 4, 8, 8, 16, 4>;     // 64 x 64

template <typename TL, bool NK>
int launch_tile(rusty_cuda_ctx* ctx, const float* a, const float* b, float* out, uint32_t M, uint32_t K, uint32_t N, const LoraTail& lora) {
    const dim3 grid((N + TL::BN - 1) / TL::BN, (M + TL::BM - 1) / TL::BM);
    const bool vec = K % 4 == 0 && (NK || N % 4 == 0) &&
                     ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(lora.b)) & 15) == 0;
    auto kern = vec ? matmul_f32_kernel<TL, NK, true> : matmul_f32_kernel<TL, NK, false>;
    size_t smem = (size_t)TL::ST * (TL::BM * TL::LDA + (NK ? TL::B_NK : TL::B_KN)) * 4;
    // no more blocks than SMs: more than half an SM's shared memory each keeps two from sharing one SM while others idle
    if ((uint64_t)grid.x * grid.y <= (uint64_t)ctx->sm_count && smem < ctx->smem_optin / 2 + 2048) smem = ctx->smem_optin / 2 + 2048;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, ctx->device, smem);
    if (e == cudaSuccess) e = launch_pdl(kern, grid, dim3(TL::THREADS), smem, ctx->stream, a, b, out, M, K, N, lora);
    if (e != cudaSuccess) return check_cuda(ctx, e, NK ? "matmul_bt_f32" : "matmul_f32");
    return after_launch(ctx, NK ? "matmul_bt_f32" : "matmul_f32");
}
template <bool NK>
int launch_matmul(rusty_cuda_ctx* ctx, const float* a, const float* b, float* out, uint32_t M, uint32_t K, uint32_t N, const LoraTail& lora) {
    // Few rows: the tile that holds them, so that b is read once.  Otherwise by the outputs an SM gets: many threads of few
    // outputs while the chain is what bounds an SM, more outputs a thread (fewer shared-memory passes each) once the SMs are
    // full; 64 x 64 only where it still gives every SM two blocks.  K = 4096, us, by outputs an SM and tile:
    //                 4     8    16    32    64   big
    //      86       20.1  30.6  37.2  56.6  78.1   208     (64 x 200)
    //     221       29.6  29.7  35.7  55.5  76.8   208     (64 x 512)
    //     332       38.7  49.1  36.0  55.5  77.7   208     (128 x 384)
    //     554       64.9  76.9  59.2  55.6  77.2   208     (128 x 640)
    //     886       87.7  96.2  59.0  55.7  77.3   210     (128 x 1024)
    //    1384        133   143  92.3  94.3  77.6   210     (64 x 3200)
    //    7085        656   661   400   320   243   224     (256 x 4096)
    //   14170       1295  1317   795   632   415   402     (512 x 4096)
    // The lines are drawn by outputs alone; a tile whose blocks just miss one wave is chosen all the same (277, 64 x 640: 8 rows
    // 49.3, 16 rows 36.1; 1124, 64 x 2600: 32 rows 97.1, 64 rows 78.5).
    const uint64_t outputs = (uint64_t)M * N, sms = (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    if (M == 1) return launch_tile<TileRow, NK>(ctx, a, b, out, M, K, N, lora);
    if (M <= 4 || outputs <= 128 * sms) return launch_tile<Tile4, NK>(ctx, a, b, out, M, K, N, lora);
    if (M <= 8 || outputs <= 300 * sms) return launch_tile<Tile8, NK>(ctx, a, b, out, M, K, N, lora);
    if (M <= 16 || outputs <= 600 * sms) return launch_tile<Tile16, NK>(ctx, a, b, out, M, K, N, lora);
    if (M <= 32 || outputs <= 1300 * sms) return launch_tile<Tile32, NK>(ctx, a, b, out, M, K, N, lora);
    if (outputs < 8192 * sms) return launch_tile<Tile64, NK>(ctx, a, b, out, M, K, N, lora);
    return launch_tile<TileBig, NK>(ctx, a, b, out, M, K, N, lora);
}

// t[M, r4] = x[M, K] . A[K, r] (zeros in columns r .. r4), the adapter's first product.  Here the order of the sum is free (f32
// throughout): a block takes MT rows of x and four columns of A, its threads cut K between them, so that the product costs
// two trips to L2 instead of a chain of K links.  (No read-only loads here and in the kernel below: what they read may be the work
// of kernels that still run when these start.)
// LD_THREADS: 512 from K = 2048 on, so that a thread's loads are all in flight at once at K = 4096 (with 256 threads and four at a time a call on a
// quantised 4096 x 4096 weight took 34 instead of 26 us at 16 rows of rank 64, 11.3 instead of 10.6 at one of rank 8), 256 below.
template <int MT, int LD_THREADS>
__global__ void __launch_bounds__(LD_THREADS) lora_down_kernel(const float* x, const float* A, float* t,
                                                               uint32_t M, uint32_t K, uint32_t r, uint32_t r4, uint32_t col0) {
    __shared__ float red[LD_THREADS / 32][MT * 4];
    pdl_wait();
    pdl_launch_dependents();   // after the wait: the matmul that follows may read x and W at once
    const uint32_t m0 = blockIdx.x * MT, c0 = col0 + blockIdx.y * 4;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float acc[MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    const bool vec = r % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
#pragma unroll(MT == 1 ? 8 : 4)
    for (uint32_t k = tid; k < K; k += LD_THREADS) {
        float av[4];
        const float* pa = A + (size_t)k * r + c0;
        if (vec) {
            const float4 q = *reinterpret_cast<const float4*>(pa);
            av[0] = q.x; av[1] = q.y; av[2] = q.z; av[3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) av[j] = c0 + j < r ? pa[j] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            const float xv = m0 + i < M ? x[(size_t)(m0 + i) * K + k] : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv, av[j], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], off);
            if (lane == 0) red[warp][i * 4 + j] = acc[i][j];
        }
    __syncthreads();
    if (tid < MT * 4) {
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < LD_THREADS / 32; ++w) s += red[w][tid];
        const uint32_t m = m0 + tid / 4, c = c0 + tid % 4;
        if (m < M) t[(size_t)m * r4 + c] = c < r ? s : 0.0f;
    }
}

// y[M, N] += t[M, r4] . b[r, N], behind a quantised Linear that has written y.  One thread per column, the block's rows one
// after the other: b stays in registers up to rank 16.
constexpr int LU_THREADS = 256, LU_KEEP = 16;
__global__ void __launch_bounds__(LU_THREADS) lora_up_add_kernel(const float* t, const float* b, float* y, uint32_t M,
                                                                 uint32_t N, int r, uint32_t r4, uint32_t rows) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t n = blockIdx.x * LU_THREADS + threadIdx.x;
    if (n >= N) return;
    float bv[LU_KEEP];
#pragma unroll
    for (int q = 0; q < LU_KEEP; ++q) bv[q] = q < r ? b[(size_t)q * N + n] : 0.0f;
    const uint32_t m1 = min(M, (blockIdx.y + 1) * rows);
    for (uint32_t m = blockIdx.y * rows; m < m1; ++m) {
        const float* tr = t + (size_t)m * r4;
        const float v = y[(size_t)m * N + n];
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < LU_KEEP; ++q)
            if (q < r) s = fmaf(tr[q], bv[q], s);
        for (int q = LU_KEEP; q < r; ++q) s = fmaf(tr[q], b[(size_t)q * N + n], s);
        y[(size_t)m * N + n] = __fadd_rn(v, s);
    }
}

int launch_lora_down(rusty_cuda_ctx* ctx, const float* x, const float* A, float* t, uint32_t M, uint32_t K, uint32_t r, uint32_t r4) {
    // rows per block: enough blocks for the SMs first (one row each), then fewer passes over A; once x is re-read for so many
    // columns that the blocks fill the chip twice over, the chain of the matmul is shorter than the re-reading.  Whole calls, K =
    // 4096, N = 512, us, with 1, 4, 8 rows a block and with the matmul: 128 rows of rank 8 38.8 / 39.9 / 41.8 / 55.6, 256 of 8 60.0 /
    // 60.2 / 61.9 / 75.9, 64 of 64 46.9 / 36.5 / 36.4 / 49.3, 100 of 64 62.1 / 45.3 / 44.6 / 55.5, 256 of 64 121 / 77 / 73 / 76, 600
    // of 16 263 / 250 / 250 / 154, 1024 of 8 254 / 248 / 250 / 157.  (The line is drawn by blocks alone: 100 and 256 of 64 lie
    // behind it all the same.)
    const uint32_t cols = r4 / 4;
    const uint64_t want = 2ull * (unsigned)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    const uint32_t mt = (uint64_t)M * cols <= want ? 1 : (uint64_t)(M / 4) * cols <= want ? 4 : 8;
    if (mt == 8 && r == r4 && (uint64_t)(M / 8) * cols > want / 2) return launch_matmul<false>(ctx, x, A, t, M, K, r, LoraTail{});
    const unsigned threads = K >= 2048 ? 512 : 256;
    auto kern = threads == 512 ? (mt == 1 ? lora_down_kernel<1, 512> : mt == 4 ? lora_down_kernel<4, 512> : lora_down_kernel<8, 512>)
                               : (mt == 1 ? lora_down_kernel<1, 256> : mt == 4 ? lora_down_kernel<4, 256> : lora_down_kernel<8, 256>);
    cudaError_t e = cudaSuccess;
    for (uint32_t c = 0; c < cols && e == cudaSuccess; c += 65535u)
        e = launch_pdl(kern, dim3((M + mt - 1) / mt, cols - c < 65535u ? cols - c : 65535u), dim3(threads), 0, ctx->stream, x, A, t, M, K, r, r4, c * 4u);
    if (e != cudaSuccess) return check_cuda(ctx, e, "lora_down");
    return after_launch(ctx, "lora_down");
}

// ---- f32 Linear with an adapter ----------------------------------------------------------------------------------------
// y[M, N] = [x | t] . [W ; B].  No shader gives the order of this sum (the reference adds two products), so it may be cut, and it
// may run on the tensor cores as long as nothing is lost.  An f32 is a tf32 (11 bits, to nearest) plus a tf32 of what is left, off by
// 2^-23 of it at most and to either side; of the four products the smallest, below 2^-24, is left out.  The three others of sixteen k go
// into one mma.sync chain that starts at zero, the smaller ones first, and its result is added in f32 to the lane's accumulators: the
// tensor core's own, truncating, additions stay inside sixteen k.  Against float64, 2-norm, K = 4096: 1.4e-7 where one f32 chain is off by
// 1.1e-6; K = 512: 1.3e-7 and 3.7e-7.
// An infinity, or a sum beyond the largest float, comes out of the split as a NaN: outputs that are not finite are computed once
// more, in one f32 chain.
//
// A warp owns 64 columns x 8 NT rows x a range of K, in units of sixteen k.  Its loads go straight into fragments, one unit ahead: a
// lane's four neighbouring columns of W are rows g and g + 8 of two tiles (a register each, nothing to pack), its four
// neighbouring k of a row of x the k it owns in W.  The ranges of a CTA's warps are summed in shared memory, those of a cluster's
// CTAs in distributed shared memory, in a fixed order.  What bounds it: up to 16 rows waiting for W (48 KB in flight an SM; a warp's
// loads, its split and its MMAs take turns, three warps a scheduler), beyond them the split and the MMAs (24 NT of 8 cycles a unit).
// 4096 x 4096, rank 8, whole call in a graph: 8 rows 31.9 -> 22.3, 16 rows 41.4 -> 29.1, 64 rows 82.7 -> 60.8, 256 rows 251 -> 215 us;
// 8192 x 512: 8 rows 39.7 -> 14.5, 64 rows 65.9 -> 44.8; 8192 x 8192, rank 64: 8 rows 108 -> 72.5, 64 rows 500 -> 226.
// Tried: FMAs with x from shared memory (the reads and the copies of a weight into both halves of a pair: 16 rows 27, 256 rows 269),
// three bf16 instead of two tf32 (more to split and to pack: 28, 223), copies by cp.async (whole lines torn apart on their way into
// fragment order: 33), 256 columns a CTA (clusters of eight, of which 15 fit: 47).
constexpr int SP_BN = 64;
template <int NT>
constexpr int SP_WARPS = NT == 4 ? 8 : 12;

// D = A[16x8] . B[8x8] + C, tf32 -> f32
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], float c0, float c1, float c2, float c3) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
// v = big + small, both with the lower 13 bits clear
__device__ __forceinline__ void split2(float v, uint32_t& big, uint32_t& small) {
    big = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
    small = __float_as_uint(v - __uint_as_float(big)) & 0xffffe000u;
}

template <int NT>
__global__ void __launch_bounds__(32 * SP_WARPS<NT>, 1) linear_splitk_f32_kernel(const float* x, const float* W, float* y, uint32_t M, uint32_t K, uint32_t N,
                                                                                 const LoraTail lora, int ways, uint32_t row_tiles) {
    constexpr int TM = 8 * NT, WARPS = SP_WARPS<NT>, THREADS = 32 * WARPS;
    extern __shared__ __align__(16) float sp_smem[];
    const int warp = warp_id(), lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const uint32_t way = blockIdx.x % (uint32_t)ways, tile = blockIdx.x / (uint32_t)ways;
    const uint32_t m0 = (tile % row_tiles) * TM, n0 = (tile / row_tiles) * SP_BN;
    // this lane's columns, 4 g .. 4 g + 3 of each half of 32 (N % 4 == 0: they exist together, or are others' and not stored)
    const uint32_t c0 = min(n0 + 4 * g, N - 4), c1 = min(n0 + 32 + 4 * g, N - 4);
    float acc[4][NT][4];     // [tile of 16 columns][rows 8 at a time]
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < NT; ++i) acc[t][i][0] = acc[t][i][1] = acc[t][i][2] = acc[t][i][3] = 0.0f;

    // the K + r links in units of sixteen, the same number for every warp; the last ones hold t . B
    const uint32_t units_k = (K + 15) / 16, units = units_k + ((uint32_t)lora.r + 15) / 16;
    const uint32_t parts = (uint32_t)(ways * WARPS), mine = way * WARPS + warp;
    const uint32_t u0 = (uint32_t)((uint64_t)units * mine / parts), u1 = (uint32_t)((uint64_t)units * (mine + 1) / parts);
    // The kernel in front of this one only computes t, and it lets this one start after its own griddepcontrol.wait
    // (lora_down_kernel): x, W and y are free by then, only t has to be waited for.
    bool t_ready = false;
    struct Unit {
        float4 w[8];      // links 4 j .. 4 j + 3: columns c0, then c1
        float4 x[NT];     // the same links of row g
    };
    auto fetch = [&](Unit& v, uint32_t u) {
        if (u >= u1) return;
        const bool second = u >= units_k;
        if (second && !t_ready) {
            pdl_wait();
            t_ready = true;
        }
        const float* a = second ? lora.t : x;
        const uint32_t lda = second ? (uint32_t)lora.r4 : K, len = second ? (uint32_t)lora.r : K;
        const uint32_t k = (second ? u - units_k : u) * 16 + 4 * j;
        const float* p = (second ? lora.b : W) + (size_t)k * N;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool whole = k - 4 * j + 16 <= len;       // (the same for all lanes)
#pragma unroll
        for (int h = 0; h < 4; ++h, p += N) {
            if (whole) {
                v.w[h] = ldg_f4(p + c0);
                v.w[4 + h] = ldg_f4(p + c1);
            } else {                                     // links that do not exist are zeros
                v.w[h] = k + h < len ? ldg_f4(p + c0) : zero;
                v.w[4 + h] = k + h < len ? ldg_f4(p + c1) : zero;
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)                     // (rows that do not exist repeat the last one)
            v.x[i] = whole || k < len ? ldg_f4(a + (size_t)min(m0 + 8 * i + g, M - 1) * lda + k) : zero;
        if (!whole && k < len && k + 4 > len)            // t's rows are padded with zeros, x's (K % 4 == 0) end with a lane's four
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                if (k + 1 >= len) v.x[i].y = 0.0f;
                if (k + 2 >= len) v.x[i].z = 0.0f;
                v.x[i].w = 0.0f;
            }
    };
    auto multiply = [&](const Unit& v) {
        uint32_t xb[2][2][NT][2];                        // [big, small][eight of the sixteen k][rows][fragment]
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            split2(v.x[i].x, xb[0][0][i][0], xb[1][0][i][0]);
            split2(v.x[i].y, xb[0][0][i][1], xb[1][0][i][1]);
            split2(v.x[i].z, xb[0][1][i][0], xb[1][1][i][0]);
            split2(v.x[i].w, xb[0][1][i][1], xb[1][1][i][1]);
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                uint32_t wa[2][2][4];                    // [big, small][eight k][row g, g + 8 (columns 2 t, 2 t + 1) of k and of k + 1]
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float4& f = v.w[4 * half + h];
                    split2(t == 0 ? f.x : f.z, wa[0][h >> 1][2 * (h & 1)], wa[1][h >> 1][2 * (h & 1)]);
                    split2(t == 0 ? f.y : f.w, wa[0][h >> 1][2 * (h & 1) + 1], wa[1][h >> 1][2 * (h & 1) + 1]);
                }
                float d[NT][4];
#pragma unroll
                for (int i = 0; i < NT; ++i) mma_tf32(d[i], wa[1][0], xb[0][0][i], 0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int m = 1; m < 6; ++m)              // small x big, big x small, big x big
#pragma unroll
                    for (int i = 0; i < NT; ++i) mma_tf32(d[i], wa[m < 2 ? 1 : 0][m & 1], xb[m >> 1 == 1 ? 1 : 0][m & 1][i], d[i][0], d[i][1], d[i][2], d[i][3]);
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[2 * half + t][i][e] += d[i][e];
            }
    };
    Unit ua, ub;
    fetch(ua, u0);
#pragma unroll 1
    for (uint32_t u = u0; u < u1; u += 2) {
        fetch(ub, u + 1);
        multiply(ua);
        fetch(ua, u + 2);
        if (u + 1 < u1) multiply(ub);
    }
    // ---- the warps' sums: [warp][TM][64], then this CTA's in the first warp's place ----
    float* part = sp_smem;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 2; ++e)      // row 2 j + e of these eight, the lane's four columns of half h
                *reinterpret_cast<float4*>(part + ((size_t)warp * TM + 8 * i + 2 * j + e) * SP_BN + 32 * h + 4 * g) =
                    make_float4(acc[2 * h][i][e], acc[2 * h][i][2 + e], acc[2 * h + 1][i][e], acc[2 * h + 1][i][2 + e]);
    __syncthreads();
    constexpr int ITEMS = TM * SP_BN / 4;      // four columns of a row each
    float4* p4 = reinterpret_cast<float4*>(part);
    cg::cluster_group cl = cg::this_cluster();
    auto put = [&](int i, float4 s) {
        const uint32_t m = m0 + (uint32_t)(i / (SP_BN / 4)), c = n0 + (uint32_t)(i % (SP_BN / 4)) * 4;
        if (m >= M || c >= N) return;
        if (!(fabsf(s.x) <= 3.0e38f && fabsf(s.y) <= 3.0e38f && fabsf(s.z) <= 3.0e38f && fabsf(s.w) <= 3.0e38f)) {
            pdl_wait();
            s = make_float4(0.f, 0.f, 0.f, 0.f);
            auto chain = [&](const float* a, const float* b, uint32_t len) {
                for (uint32_t k = 0; k < len; ++k, b += N) {
                    const float4 v = *reinterpret_cast<const float4*>(b + c);
                    s.x = fmaf(a[k], v.x, s.x); s.y = fmaf(a[k], v.y, s.y); s.z = fmaf(a[k], v.z, s.z); s.w = fmaf(a[k], v.w, s.w);
                }
            };
            chain(x + (size_t)m * K, W, K);
            chain(lora.t + (size_t)m * lora.r4, lora.b, (uint32_t)lora.r);
        }
        *reinterpret_cast<float4*>(y + (size_t)m * N + c) = s;
    };
    for (int i = threadIdx.x; i < ITEMS; i += THREADS) {
        float4 s = p4[i];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) {
            const float4 v = p4[w * ITEMS + i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (ways == 1) put(i, s);
        else p4[i] = s;                        // (an item is one thread's)
    }
    if (ways == 1) return;
    cl.sync();
    for (int i = (int)way * THREADS + threadIdx.x; i < ITEMS; i += ways * THREADS) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int w = 0; w < ways; ++w) {
            const float4 v = cl.map_shared_rank(p4, w)[i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        put(i, s);
    }
    cl.sync();                                 // the others have read this CTA's sums
}

template <int NT>
int launch_splitk(rusty_cuda_ctx* ctx, const float* x, const float* W, float* y, uint32_t M, uint32_t K, uint32_t N, const LoraTail& lora) {
    constexpr int TM = 8 * NT, WARPS = SP_WARPS<NT>;
    const uint32_t groups = (N + SP_BN - 1) / SP_BN, row_tiles = (M + TM - 1) / TM;
    const uint64_t tiles = (uint64_t)groups * row_tiles, sms = (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    // K ranges: what fills the SMs with one CTA each, of a unit a warp at least.  Clusters lie in one GPC: of more than two CTAs not as
    // many fit as there are SMs (of 148: 132 in clusters of four, 120 of eight), so beyond two an eighth of them is left out.
    uint64_t ways = sms / tiles >= 3 ? sms * 7 / 8 / tiles : sms / tiles;
    const uint64_t most = K / (16 * WARPS);
    if (ways > most) ways = most;
    ways = ways < 1 ? 1 : ways > 4 ? (ways < 8 ? 4 : 8) : ways;
    constexpr size_t smem = (size_t)WARPS * TM * SP_BN * 4;
    auto kern = linear_splitk_f32_kernel<NT>;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, ctx->device, smem);
    if (e == cudaSuccess)
        e = launch_pdl_cluster(kern, dim3((unsigned)(tiles * ways)), dim3(32 * WARPS), (unsigned)ways, smem, ctx->stream, x, W, y, M, K, N, lora, (int)ways, row_tiles);
    if (e != cudaSuccess) return check_cuda(ctx, e, "linear_splitk_f32");
    return after_launch(ctx, "linear_splitk_f32");
}

int need(rusty_cuda_ctx* ctx, const char* op, const char* name, const rusty_cuda_buf* b, size_t bytes) {
    if (!b) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: buffer '%s' is null", op, name);
    if (b->bytes < bytes)
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: buffer '%s' holds %zu bytes, the given dimensions need %zu",
                    op, name, b->bytes, bytes);
    return RUSTY_CUDA_OK;
}

// A launch holds 65535 row tiles, of 4 rows in the worst case; a call as many as of 64 rows.
constexpr uint32_t PASS_ROWS = 65535u * 4u;
bool too_many_rows(uint32_t M) { return M > 65535u * 64u; }

template <bool NK>
int matmul_entry(rusty_cuda_ctx* ctx, const char* op, const rusty_cuda_buf* a, const rusty_cuda_buf* b, rusty_cuda_buf* out, uint32_t M,
                 uint32_t K, uint32_t N) {
    int rc;
    if ((rc = need(ctx, op, "a", a, (size_t)M * K * 4))) return rc;
    if ((rc = need(ctx, op, "b", b, (size_t)K * N * 4))) return rc;
    if ((rc = need(ctx, op, "out", out, (size_t)M * N * 4))) return rc;
    if (M == 0 || N == 0) return RUSTY_CUDA_OK;
    if (too_many_rows(M)) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: M=%u too large", op, M);
    DeviceGuard g(ctx->device);
    for (uint32_t m0 = 0; m0 < M; m0 += PASS_ROWS) {
        const uint32_t rows = M - m0 < PASS_ROWS ? M - m0 : PASS_ROWS;
        if ((rc = launch_matmul<NK>(ctx, (const float*)a->ptr + (size_t)m0 * K, (const float*)b->ptr, (float*)out->ptr + (size_t)m0 * N, rows, K, N,
                                    LoraTail{})))
            return rc;
    }
    return RUSTY_CUDA_OK;
}

}  // namespace

extern "C" {

int rusty_cuda_matmul_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* a, const rusty_cuda_buf* b, rusty_cuda_buf* out,
                          uint32_t M, uint32_t K, uint32_t N) {
    RUSTY_REQUIRE_CTX(ctx);
    return matmul_entry<false>(ctx, "matmul", a, b, out, M, K, N);
}

int rusty_cuda_matmul_bt_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* a, const rusty_cuda_buf* b,
                             rusty_cuda_buf* out, uint32_t M, uint32_t K, uint32_t N) {
    RUSTY_REQUIRE_CTX(ctx);
    return matmul_entry<true>(ctx, "matmul_bt", a, b, out, M, K, N);
}

int rusty_cuda_linear_lora_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* x, const rusty_cuda_buf* weight, const rusty_cuda_qlinear* ql,
                               const rusty_cuda_buf* lora_a, const rusty_cuda_buf* lora_b, rusty_cuda_buf* y, uint32_t M, uint32_t K,
                               uint32_t N, uint32_t rank) {
    RUSTY_REQUIRE_CTX(ctx);
    const char* op = "linear_lora";
    if ((weight == nullptr) == (ql == nullptr))
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: one of the f32 weight and the quantised linear is required", op);
    if (ql && (ql->K != K || ql->N != N || ql->act))
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: the quantised linear is [%u,%u]%s, not [%u,%u]", op, ql->N, ql->K,
                    ql->act ? " with an activation" : "", N, K);
    int rc;
    if ((rc = need(ctx, op, "x", x, (size_t)M * K * 4))) return rc;
    if (weight && (rc = need(ctx, op, "weight", weight, (size_t)K * N * 4))) return rc;
    if ((rc = need(ctx, op, "lora_a", lora_a, (size_t)K * rank * 4))) return rc;
    if ((rc = need(ctx, op, "lora_b", lora_b, (size_t)rank * N * 4))) return rc;
    if ((rc = need(ctx, op, "y", y, (size_t)M * N * 4))) return rc;
    if (M == 0 || N == 0) return RUSTY_CUDA_OK;
    if (too_many_rows(M)) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: M=%u too large", op, M);
    if (rank == 0)
        return weight ? rusty_cuda_matmul_f32(ctx, x, weight, y, M, K, N) : rusty_cuda_qlinear_forward(ctx, ql, x, RUSTY_CUDA_F32, M, y, RUSTY_CUDA_F32);
    // t = x . A lives in a pool buffer: later calls on this stream may take it over as soon as its reader is enqueued
    const uint32_t r4 = (rank + 3u) & ~3u, t_rows = M < PASS_ROWS ? M : PASS_ROWS;
    rusty_cuda_buf* t = nullptr;
    if ((rc = rusty_cuda_buf_alloc(ctx, (size_t)t_rows * r4 * 4, 1, &t))) return rc;
    DeviceGuard g(ctx->device);
    if (ql) rc = qlinear_forward_cols(ctx, ql, x, RUSTY_CUDA_F32, M, y, RUSTY_CUDA_F32, N, 0);
    // The kernel with K cut where rows and columns can be read four at a time and it is the faster one.  Below 2^20 weights the tiles
    // are (one chain of 512 k, 512 columns, against a cluster's meeting: 16 rows 5.3 / 7.6 us; 1024 x 1024: 8.0 / 7.6).  Up to four
    // rows they read W faster and only their chain of K is slow: us, tiles / cut, K x N at one row: 8192 x 512 40.5 / 14.2, 4096 x
    // 1024 21.9 / 17.2, 2048 x 2048 12.6 / 9.7, 4096 x 4096 22.4 / 22.0, 2048 x 8192 16.1 / 21.2, 8192 x 8192 48.6 / 63.1.
    const uint64_t weights = (uint64_t)K * N;
    const bool cut = weight && K % 4 == 0 && N % 4 == 0 && weights >= (1u << 20) && (M > 4 || (N <= K && weights < (1u << 24))) &&
                     ((reinterpret_cast<uintptr_t>(x->ptr) | reinterpret_cast<uintptr_t>(weight->ptr) | reinterpret_cast<uintptr_t>(lora_b->ptr) |
                       reinterpret_cast<uintptr_t>(y->ptr)) & 15) == 0;
    for (uint32_t m0 = 0; m0 < M && !rc; m0 += PASS_ROWS) {
        const uint32_t m = M - m0 < PASS_ROWS ? M - m0 : PASS_ROWS;
        const float* xp = (const float*)x->ptr + (size_t)m0 * K;
        float* yp = (float*)y->ptr + (size_t)m0 * N;
        const LoraTail tail{(const float*)t->ptr, (const float*)lora_b->ptr, (int)rank, (int)r4};
        rc = launch_lora_down(ctx, xp, (const float*)lora_a->ptr, (float*)t->ptr, m, K, rank, r4);
        if (rc) break;
        if (cut) {
            const float* w = (const float*)weight->ptr;
            rc = m <= 8    ? launch_splitk<1>(ctx, xp, w, yp, m, K, N, tail)
                 : m <= 16 ? launch_splitk<2>(ctx, xp, w, yp, m, K, N, tail)
                           : launch_splitk<4>(ctx, xp, w, yp, m, K, N, tail);
        } else if (weight) {
            rc = launch_matmul<false>(ctx, xp, (const float*)weight->ptr, yp, m, K, N, tail);
        } else {
            const unsigned gx = (N + LU_THREADS - 1) / LU_THREADS;
            unsigned rows = (unsigned)(((uint64_t)m * gx + 4ull * ctx->sm_count - 1) / (4ull * ctx->sm_count));   // four blocks an SM
            if (rows < (m + 65534u) / 65535u) rows = (m + 65534u) / 65535u;
            cudaError_t e = launch_pdl(lora_up_add_kernel, dim3(gx, (m + rows - 1) / rows), dim3(LU_THREADS), 0, ctx->stream, (const float*)t->ptr,
                                       (const float*)lora_b->ptr, yp, m, N, (int)rank, r4, rows);
            rc = e != cudaSuccess ? check_cuda(ctx, e, "lora_up_add") : after_launch(ctx, "lora_up_add");
        }
    }
    rusty_cuda_buf_release(t);
    return rc;
}

}  // extern "C"
