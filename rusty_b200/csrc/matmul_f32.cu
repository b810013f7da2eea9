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
// A global load as volatile asm, for the same reason.
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
// y[M, N] = [x | t] . [W ; B], f32 throughout: every product enters by a fused multiply-add, so that infinities, subnormals and single
// products are what f32 makes them.  No shader gives the order of this sum (the reference adds two products), so K is cut: a warp owns 64
// columns x TM rows x a range of K in units of sixteen links, its halves take the even and the odd ones, a lane four neighbouring columns
// (pairs of rows share an FMA instruction).  Each warp has a ring of its own: W as it is, by cp.async, and x as [link][row], so that four
// rows are one read: from 16 rows on by way of registers, a unit ahead (a copy of four bytes a lane takes the copy pipe some 15 cycles; 32 x 912
// x 7172 19.6 -> 17.8 us), below that by such copies.  The ranges of a CTA's warps are summed in shared memory, those of a cluster's
// CTAs in distributed shared memory, in a fixed order that depends on K, N and the rank, and beyond 32 rows on their number: up to there a
// row's bits do not depend on the rows beside it.  Against float64, 2-norm, K = 4096: 2.1e-7 where one f32 chain is off by 1.1e-6; K =
// 8192 x 8192: 3.4e-7 and 1.3e-6.
//
// What bounds it: up to eight rows W (96 KB in flight an SM) and the fixed part of two launches, beyond sixteen the FMAs: the pipe is busy 65 %
// of a CTA's time at 256 rows.  4096 x 4096, rank 8, whole call in a graph, one chain of K on the matmul's tiles / this, us: one row 21.6
// / 13.2, 8 rows 31.2 / 13.9, 16 rows 37.8 / 19.8, 64 rows 79.5 / 52.7, 256 rows 248 / 197; 8192 x 512: 8 rows 39.3 / 9.0, 64 rows 60.0 / 20.3;
// 8192 x 8192, rank 64: one row 47.2 / 40.2, 64 rows 495 / 203.
// Tried: two tf32 an f32 on the tensor cores (the products lose up to 2^-21 of themselves; 8 rows 21.7, 16 rows 25.6, 64 rows 57.4, 256 rows
// 213); W through registers instead of a ring (8 rows 23, 16 rows 28, 64 rows 72); 256 columns a CTA (clusters of eight, of which 15 fit: 47).
constexpr int SP_BN = 64, SP_WARPS = 8, SP_THREADS = 32 * SP_WARPS, SP_STAGES = 4;
template <int TM>
struct Sp {
    static constexpr int LDX = TM + 4;                                          // floats between links of x in shared memory
    static constexpr int STAGE = 16 * (SP_BN + LDX);                            // floats of a unit: W, then x
    static constexpr int PIECE = TM < 16 ? TM : 16;                             // rows read ahead of their FMAs
    static constexpr bool X_REGS = TM >= 16;                                    // x goes to shared memory by way of registers
    static constexpr int XV = X_REGS ? TM / 8 : 1;
    static constexpr int RING = SP_WARPS * SP_STAGES * STAGE, PART = SP_WARPS * TM * SP_BN;
    static constexpr size_t SMEM = (size_t)(RING > PART ? RING : PART) * 4;
};

__device__ __forceinline__ ulonglong2 lds_2xf32x2(uint32_t addr) {
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
    return v;
}

__device__ __forceinline__ void sts_f1(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

template <int TM>
__global__ void __launch_bounds__(SP_THREADS, 1) linear_splitk_f32_kernel(const float* x, const float* W, float* y, uint32_t M, uint32_t K, uint32_t N,
                                                                          const LoraTail lora, int ways, uint32_t row_tiles) {
    using C = Sp<TM>;
    constexpr int PIECE = C::PIECE, ST = SP_STAGES;
    extern __shared__ __align__(16) float sp_smem[];
    const int warp = warp_id(), lane = threadIdx.x & 31, half = lane >> 4;
    const uint32_t way = blockIdx.x % (uint32_t)ways, tile = blockIdx.x / (uint32_t)ways;
    const uint32_t m0 = (tile % row_tiles) * TM, n0 = (tile / row_tiles) * SP_BN;
    const uint32_t c0 = n0 + 4 * (lane & 15);                  // this lane's four columns (N % 4 == 0: there or not)
    const bool there = c0 < N;
    const uint32_t ring = smem_u32(sp_smem) + (uint32_t)(warp * ST * C::STAGE) * 4;
    unsigned long long acc[TM / 2][4];                         // [two rows][column]
#pragma unroll
    for (int i = 0; i < TM / 2; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0ull;

    // the K + r links in units of sixteen, the same number for every warp; the last ones hold t . B
    const uint32_t units_k = (K + 15) / 16, units = units_k + ((uint32_t)lora.r + 15) / 16;
    const uint32_t parts = (uint32_t)(ways * SP_WARPS), mine = way * SP_WARPS + warp;
    const uint32_t u0 = (uint32_t)((uint64_t)units * mine / parts), u1 = (uint32_t)((uint64_t)units * (mine + 1) / parts);
    // The kernel in front of this one only computes t, and it lets this one start after its own griddepcontrol.wait
    // (lora_down_kernel): x, W and y are free by then, only t has to be waited for.
    bool t_ready = false;
    auto fetch = [&](uint32_t u, int slot) {
        if (u < u1) {
            const bool tail = u >= units_k;
            if (tail && !t_ready) {
                pdl_wait();
                t_ready = true;
            }
            const uint32_t k0 = (tail ? u - units_k : u) * 16, len = tail ? (uint32_t)lora.r : K, lda = tail ? (uint32_t)lora.r4 : K;
            const uint32_t to = ring + (uint32_t)(slot * C::STAGE) * 4;
            // W: links 2 i + half, the lane's own four columns; x: link lane % 16 of rows lane / 16 + 2 i
            const uint32_t to_w = to + (uint32_t)(half * SP_BN + 4 * (lane & 15)) * 4, to_x = to + (uint32_t)(16 * SP_BN + (lane & 15) * C::LDX + half) * 4;
            const float* p = (tail ? lora.b : W) + (size_t)(k0 + half) * N + c0;
            const uint32_t k = k0 + (lane & 15);
            const float* a = (tail ? lora.t : x) + (size_t)m0 * lda + k;
            // Rows and columns that do not exist are not copied: whatever lies there goes into sums that are not stored.  (Copies of the last
            // ones in their place: a rolled loop over rows took 79.6 us for 40 x 4096 x 4096, now 52.1, and lanes that copied one address
            // 139.8 us for 194 x 3152 x 3980, now 123.)
            const int rows = (int)min((uint32_t)TM, M - m0) - half;
            a += (size_t)half * lda;
            if (k0 + 16 <= len) {
                if (there)
#pragma unroll
                    for (int i = 0; i < 8; ++i, p += 2 * (size_t)N) cp_async<true>(to_w + (uint32_t)(2 * i * SP_BN) * 4, p, 16u);
                if constexpr (!C::X_REGS)
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i, a += 2 * (size_t)lda)
                        if (2 * i < rows) cp_async<false>(to_x + (uint32_t)(2 * i) * 4, a, 4u);
            } else {   // links that do not exist are zeros (t's rows are padded with them to r4)
                const int left = (int)(len - k0) - half;
                const uint32_t bytes = k < lda ? 4u : 0u;
                if (there)
#pragma unroll 1
                    for (int i = 0; i < 8; ++i, p += 2 * (size_t)N) cp_async<true>(to_w + (uint32_t)(2 * i * SP_BN) * 4, 2 * i < left ? p : W, 2 * i < left ? 16u : 0u);
                if constexpr (!C::X_REGS)
#pragma unroll 1
                    for (int i = 0; 2 * i < rows; ++i, a += 2 * (size_t)lda) cp_async<false>(to_x + (uint32_t)(2 * i) * 4, bytes ? a : x, bytes);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // X_REGS: a lane takes four links of rows lane / 4 + 8 i, a unit ahead of their stores
    float4 xn[C::XV];
    auto load_x = [&](float4 (&v)[C::XV], uint32_t u) {
        if (u >= u1) return;
        const bool tail = u >= units_k;
        if (tail && !t_ready) {
            pdl_wait();
            t_ready = true;
        }
        const uint32_t lda = tail ? (uint32_t)lora.r4 : K, k = (tail ? u - units_k : u) * 16 + 4 * (lane & 3), row = m0 + (lane >> 2);
        const float* a = (tail ? lora.t : x) + (size_t)row * lda + k;
#pragma unroll
        for (int i = 0; i < C::XV; ++i, a += 8 * (size_t)lda)
            v[i] = k < lda && row + 8 * i < M ? ldg_f4(a) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto store_x = [&](const float4 (&v)[C::XV], int slot) {
        const int at = (lane >> 2) + 8 * ((lane >> 1) & 1);
        const uint32_t to = ring + (uint32_t)(slot * C::STAGE + 16 * SP_BN + 4 * (lane & 3) * C::LDX) * 4;
#pragma unroll
        for (int i = 0; i < C::XV; ++i) {
            const uint32_t d = to + (uint32_t)((at + 8 * i) & (TM - 1)) * 4;
            sts_f1(d, v[i].x);
            sts_f1(d + C::LDX * 4, v[i].y);
            sts_f1(d + 2 * C::LDX * 4, v[i].z);
            sts_f1(d + 3 * C::LDX * 4, v[i].w);
        }
    };
#pragma unroll 1
    for (int d = 0; d < ST - 1; ++d) fetch(u0 + d, d);
    if constexpr (C::X_REGS) {
        float4 first[C::XV];
        load_x(first, u0);
        load_x(xn, u0 + 1);
        store_x(first, 0);
    }
    int slot = 0;
#pragma unroll 1
    for (uint32_t u = u0; u < u1; ++u) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncwarp();                                          // unit u is there for all lanes, and the one before has been read by all
        fetch(u + ST - 1, slot == 0 ? ST - 1 : slot - 1);
        if constexpr (C::X_REGS) {
            store_x(xn, slot == ST - 1 ? 0 : slot + 1);
            load_x(xn, u + 2);
        }
        const uint32_t from_w = ring + (uint32_t)(slot * C::STAGE + half * SP_BN + 4 * (lane & 15)) * 4;
        const uint32_t from_x = ring + (uint32_t)(slot * C::STAGE + 16 * SP_BN + half * C::LDX) * 4;
        constexpr int PER = TM / PIECE, PIECES = 8 * PER;
        ulonglong2 xv[2][PIECE / 4];
        uint4 wv[2];
        auto read = [&](int p) {
            if (p % PER == 0) wv[(p / PER) & 1] = lds128(from_w + (uint32_t)((p / PER) * 2 * SP_BN) * 4);
#pragma unroll
            for (int q = 0; q < PIECE / 4; ++q) {
                const int row = ((p % PER) * PIECE + 4 * q + (C::X_REGS ? 8 * ((p / PER) >> 2) : 0)) & (TM - 1);
                xv[p & 1][q] = lds_2xf32x2(from_x + (uint32_t)((p / PER) * 2 * C::LDX + row) * 4);
            }
        };
        read(0);
#pragma unroll
        for (int p = 0; p < PIECES; ++p) {
            if (p + 1 < PIECES) read(p + 1);
            const uint4& w = wv[(p / PER) & 1];
            unsigned long long wd[4];
            asm("mov.b64 %0, {%1, %1};" : "=l"(wd[0]) : "r"(w.x));
            asm("mov.b64 %0, {%1, %1};" : "=l"(wd[1]) : "r"(w.y));
            asm("mov.b64 %0, {%1, %1};" : "=l"(wd[2]) : "r"(w.z));
            asm("mov.b64 %0, {%1, %1};" : "=l"(wd[3]) : "r"(w.w));
#pragma unroll
            for (int q = 0; q < PIECE / 4; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[(p % PER) * (PIECE / 2) + 2 * q][c]) : "l"(xv[p & 1][q].x), "l"(wd[c]));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[(p % PER) * (PIECE / 2) + 2 * q + 1][c]) : "l"(xv[p & 1][q].y), "l"(wd[c]));
                }
        }
        if (++slot == ST) slot = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                           // the sums go where the rings were
    float* part = sp_smem;                                     // [warp][TM][64]
    // ---- the halves' sums, then the warps': [warp][TM][64], then this CTA's in the first warp's place ----
#pragma unroll
    for (int i = 0; i < TM / 4; ++i) {                          // a half keeps its half of the rows
        float lo[4], hi[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const unsigned long long keep = half ? acc[i + TM / 4][c] : acc[i][c], give = half ? acc[i][c] : acc[i + TM / 4][c];
            const unsigned long long got = __shfl_xor_sync(0xffffffffu, give, 16);
            lo[c] = __uint_as_float((uint32_t)keep) + __uint_as_float((uint32_t)got);
            hi[c] = __uint_as_float((uint32_t)(keep >> 32)) + __uint_as_float((uint32_t)(got >> 32));
        }
        float* to = part + ((size_t)warp * TM + half * (TM / 2) + 2 * i) * SP_BN + 4 * (lane & 15);
        *reinterpret_cast<float4*>(to) = make_float4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<float4*>(to + SP_BN) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    }
    __syncthreads();
    constexpr int ITEMS = TM * SP_BN / 4;      // four columns of a row each
    float4* p4 = reinterpret_cast<float4*>(part);
    cg::cluster_group cl = cg::this_cluster();
    auto put = [&](int i, const float4& s) {
        const uint32_t m = m0 + (uint32_t)(i / (SP_BN / 4)), c = n0 + (uint32_t)(i % (SP_BN / 4)) * 4;
        if (m < M && c < N) *reinterpret_cast<float4*>(y + (size_t)m * N + c) = s;
    };
    for (int i = threadIdx.x; i < ITEMS; i += SP_THREADS) {
        float4 s = p4[i];
#pragma unroll
        for (int v = 1; v < SP_WARPS; ++v) {
            const float4 f = p4[v * ITEMS + i];
            s.x += f.x; s.y += f.y; s.z += f.z; s.w += f.w;
        }
        if (ways == 1) put(i, s);
        else p4[i] = s;                        // (an item is one thread's)
    }
    if (ways == 1) return;
    cl.sync();
    for (int i = (int)way * SP_THREADS + threadIdx.x; i < ITEMS; i += ways * SP_THREADS) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int v = 0; v < ways; ++v) {
            const float4 f = cl.map_shared_rank(p4, v)[i];
            s.x += f.x; s.y += f.y; s.z += f.z; s.w += f.w;
        }
        put(i, s);
    }
    cl.sync();                                 // the others have read this CTA's sums
}

// K ranges (CTAs of a cluster) for so many tiles: what fills the SMs with one CTA each, of a unit a warp at least.  Clusters lie in one
// GPC: of more than two CTAs not as many fit as there are SMs (of 148: 132 in clusters of four, 120 of eight), so beyond two an
// eighth of them is left out, and of eight only as many CTAs are taken as fit (4096 x 1024 at 16 rows: 16 clusters of eight 16.5 us, of four 12.1).
uint64_t splitk_ways(uint64_t tiles, uint32_t K, uint64_t sms) {
    uint64_t ways = sms / tiles >= 3 ? sms * 7 / 8 / tiles : sms / tiles;
    const uint64_t most = K / (16 * SP_WARPS);
    if (ways > most) ways = most;
    return ways < 1 ? 1 : ways <= 4 ? ways : ways < 8 || tiles * 8 > sms * 13 / 16 ? 4 : 8;
}

template <int TM>
int launch_splitk(rusty_cuda_ctx* ctx, const float* x, const float* W, float* y, uint32_t M, uint32_t K, uint32_t N, const LoraTail& lora) {
    const uint32_t groups = (N + SP_BN - 1) / SP_BN, row_tiles = (M + TM - 1) / TM;
    const uint64_t tiles = (uint64_t)groups * row_tiles, sms = (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    const uint64_t ways = splitk_ways(tiles, K, sms);
    auto kern = linear_splitk_f32_kernel<TM>;
    cudaError_t e = ensure_dynamic_smem((const void*)kern, ctx->device, Sp<TM>::SMEM);
    if (e == cudaSuccess)
        e = launch_pdl_cluster(kern, dim3((unsigned)(tiles * ways)), dim3(SP_THREADS), (unsigned)ways, Sp<TM>::SMEM, ctx->stream, x, W, y, M, K, N, lora,
                               (int)ways, row_tiles);
    if (e != cudaSuccess) return check_cuda(ctx, e, "linear_splitk_f32");
    return after_launch(ctx, "linear_splitk_f32");
}

// Rows a tile.  Up to 32 rows one tile holds them, and a row's sum is cut the same way whatever the tile.  Beyond, tiles of 32 or of 16: a unit takes
// a CTA 1.1 or 0.6 us, its start and end 4 or 3 and one more in a cluster; the tiles of 16 win where they fill the waves better.
// All of 32 / of 16, us: 38 x 912 x 2992 16.1 / 10.6, 99 x 4592 x 1244 58.1 / 36.2, 200 x 1552 x 684 25.6 / 17.6, 256 x 4096 x 4096 199.7 / 197.3; 64 x
// 4096 x 4096 52.8 / 58.5, 83 x 880 x 5996 29.6 / 36.2.  Of 125 shapes beyond 32 rows the rule takes the slower one for six, 4 % slower at most.
int launch_splitk_rows(rusty_cuda_ctx* ctx, const float* x, const float* W, float* y, uint32_t M, uint32_t K, uint32_t N, const LoraTail& lora) {
    if (M <= 4) return launch_splitk<4>(ctx, x, W, y, M, K, N, lora);
    if (M <= 8) return launch_splitk<8>(ctx, x, W, y, M, K, N, lora);
    if (M <= 16) return launch_splitk<16>(ctx, x, W, y, M, K, N, lora);
    if (M <= 32) return launch_splitk<32>(ctx, x, W, y, M, K, N, lora);
    const uint64_t sms = (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    auto us = [&](uint32_t tm, double unit, double ends) {
        const uint64_t tiles = (uint64_t)((N + SP_BN - 1) / SP_BN) * ((M + tm - 1) / tm), ways = splitk_ways(tiles, K, sms);
        const double units = (double)((K + 15) / 16 + (lora.r + 15) / 16) / (double)(SP_WARPS * ways);
        return (double)((tiles * ways + sms - 1) / sms) * (units * unit + ends + (ways > 1 ? 1.0 : 0.0));
    };
    return us(16, 0.6, 3.0) < us(32, 1.1, 4.0) ? launch_splitk<16>(ctx, x, W, y, M, K, N, lora) : launch_splitk<32>(ctx, x, W, y, M, K, N, lora);
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
    // The kernel with K cut where columns can be read four at a time and it is the faster one (tiles / cut, us).  Not below 2^20 weights (16 rows of
    // 512 x 512 4.7 / 5.8; 512 x 2048 at 16 / 32 / 64 rows 6.2 / 6.0, 7.3 / 7.7, 10.3 / 7.3; 512 x 8192 at 16 / 64 11.6 / 8.7 and 35.5 / 20.8;
    // 1024 x 1024 at 1 / 16 / 256 7.1 / 4.3, 7.8 / 6.5, 22.6 / 17.4).  Not beyond 512 rows for many outputs of few links each, where the tiles of
    // 64 x 64 fill the chip with whole CTAs: 512 x 4096 at 512 / 1024 rows 80.2 / 67.0 and 108 / 134, 1024 x 4096 153 / 106 and 206 / 214, 2048 x
    // 8192 390 / 365 and 675 / 734, 8192 x 8192 1530 / 1308 and 2656 / 2651, 4096 x 4096 588 / 345 and 795 / 705.
    const uint64_t weights = (uint64_t)K * N, outputs = (uint64_t)M * N;
    const bool cut = weight && K % 4 == 0 && N % 4 == 0 && weights >= (1u << 20) && (M <= 512 || outputs < 4096ull * K) &&
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
            rc = launch_splitk_rows(ctx, xp, (const float*)weight->ptr, yp, m, K, N, tail);
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
