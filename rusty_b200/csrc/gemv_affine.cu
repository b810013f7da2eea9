// Affine weights in [out,in] storage (u8, one f32 scale and bias per 64 consecutive k of a row: w[n,k] = u[n,k] * s[n,k/64] +
// b[n,k/64], rusty-loader/src/lib.rs:155-218 for a weight whose rows run along the contraction) for a batch of activation
// rows, on the warp-level integer tensor cores.
//
// Arithmetic.  Scales change every 64 k along the contraction, so the integer sums are taken per 64 k: the activations of such a
// chunk become four balanced signed bytes below a power-of-two scale of THEIR row and chunk (30 bits below the chunk's
// largest), two mma.sync.m16n8k32 (u8 x s8) give the exact dot products of 16 weight rows with the four digit planes of two
// activation rows, and the chunk's share of an output is dot * s + sum(x) * b in f32, rounded before it joins the sum: for weights
// around zero both terms are larger than their sum, and are never gathered apart.  sum(x) is exact, its upper part with the
// upper planes, the rest with the lower ones; ranges, and runs of RUN chunks, are added up in double.  A lane
// holds two neighbouring planes of a sum (columns 4m + 2h, 4m + 2h + 1): they fit one int32, the other two planes are the
// neighbour lane's, and the two halves meet after the last chunk.
//
// Data movement.  affine_prepare_kernel writes the digits in the order the MMA's B operand wants them: a lane's 16 bytes for
// both MMAs of a chunk are one load, a warp's 512 bytes consecutive; the warps of a CTA that walk the same chunks at the same
// time share them in L1.  Weights go from global memory straight into the A operand's registers (a lane's 16 bytes of a row
// are 16 neighbouring k; digits follow the same order, so nothing is permuted), two chunks ahead, the first ones before
// griddepcontrol.wait.  A warp owns 32 weight rows, all activation rows of the pass and a range of chunks; a CTA is wr row
// groups x 8/wr ranges, a cluster adds ranges.  Ranges are summed in shared memory (distributed, for a cluster) in a fixed order.
//
// What bounds it: up to about eight rows the weight stream and the two launches; beyond, waiting for the digits from L2 and the
// fold of a chunk (77 instructions per 32 x 2 outputs; at 24 rows 42 % of the issue slots and 19 % of the integer tensor pipe are
// used, with two warps per scheduler).  4096 x 4096, per call in a graph: 1 row 7.3 us, 8 rows 9.8, 16 rows 14.3, 24 rows 18.7, 64
// rows 49.5 (on CUDA cores, eight rows per walk over the weights, 9.9, 26, 52 and 207 us for 1, 8, 16 and 64); 3000 x 14336: 1 row
// 17.1 us (25.7).  Two digit tiles are fetched ahead (four where the tiles of a chunk are many): fetched where they are used, 64
// rows took 90 us.  Tiles of a pass beyond the rows there are, up to the next of 1, 2, 4, 8 or 12, are computed and dropped: 13
// rows take as long as 16, 14.3 us; with a row guard around a tile's arithmetic the compiler does not overlap neighbours.
#include <cooperative_groups.h>

#include <climits>
#include <type_traits>

#include "tc_common.cuh"

using namespace rusty_tc;
namespace cg = cooperative_groups;

namespace {

constexpr int AG = 64;             // k per scale
constexpr int AF_WARPS = 8;
constexpr int AF_THREADS = 32 * AF_WARPS;
constexpr int AF_ROWS = 32;        // weight rows of a warp: two MMA tiles
constexpr int RUN = 16;            // chunks of an f32 sum (a power of two)

struct AfParams {
    const uint8_t* W;
    const float* scales;     // [N][K/64]
    const float* biases;
    const uint4* digits;     // [K/64][tiles][32 lanes] x 16 bytes
    const float2* aux;       // [K/64][tiles][4]: (unit of the two planes, upper or lower part of the sum of x)
    void* y;
    int M, N, K;
    int tiles, tpp;          // pairs of activation rows: all, and per pass (blockIdx.y)
    int wr, ways;            // row groups per CTA; CTAs per cluster
    int ldy, y_col0, y_bf16;
};

__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Loads that stay where they are written, ahead of their use (plain ones were moved down to it).  Not through the read-only
// path: the pre-pass may still be writing when this kernel starts.
__device__ __forceinline__ uint4 ld_ahead(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_ahead(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// Digits of x: a half warp takes 64 k of a row.  Rows M .. 2 tiles are zeros.
template <typename XT>
__global__ void __launch_bounds__(256) affine_prepare_kernel(const XT* x, uint32_t* digits, float2* aux, int M, int K, int tiles) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, m = blockIdx.y;
    const int k = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 128 + lane * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (k < K && m < M) {
        const XT* src = x + (size_t)m * K + k;
        if constexpr (sizeof(XT) == 4) {
            const float4 f = *reinterpret_cast<const float4*>(src);
            v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
        } else {
            const uint2 raw = *reinterpret_cast<const uint2*>(src);
            v[0] = __uint_as_float(raw.x << 16), v[1] = __uint_as_float(raw.x & 0xffff0000u);
            v[2] = __uint_as_float(raw.y << 16), v[3] = __uint_as_float(raw.y & 0xffff0000u);
        }
    }
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) top = max(top, __float_as_uint(v[i]) & 0x7fffffffu);
    double sum = ((double)v[0] + (double)v[1]) + ((double)v[2] + (double)v[3]);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
    }
    if (k >= K) return;
    // |x| < 2^e, e >= -119 so that the units below are numbers, denormal ones below 2^-126
    const int e = max((int)(top >> 23) - 126, -119);
    const float up = __uint_as_float((uint32_t)(133 - e) << 23);      // 2^(6 - e)
    uint32_t q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = digits_of<4>(v[i] * up);
    const uint32_t t0 = __byte_perm(q[0], q[1], 0x5140), t1 = __byte_perm(q[2], q[3], 0x5140), t2 = __byte_perm(q[0], q[1], 0x7362),
                   t3 = __byte_perm(q[2], q[3], 0x7362);
    const uint32_t plane[4] = {__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632), __byte_perm(t2, t3, 0x5410), __byte_perm(t2, t3, 0x7632)};
    const int kk = k % AG;
    const size_t at = (size_t)(k / AG) * tiles + (m >> 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) digits[(at * 32 + ((m & 1) * 4 + i) * 4 + kk / 16) * 4 + (kk % 16) / 4] = plane[i];
    if (kk == 0) {
        const bool finite = top < 0x7f800000u;
        const float unit = finite ? __uint_as_float(e > -97 ? (uint32_t)(97 + e) << 23 : 1u << (119 + e)) : __uint_as_float(0x7fc00000u);   // 2^(e - 30)
        const float upper = (float)sum;   // (may be infinite where the largest x is not far from it: no rest then)
        *reinterpret_cast<float4*>(aux + at * 4 + (m & 1) * 2) =
            make_float4(unit, fabsf(upper) < 3.0e38f ? (float)(sum - (double)upper) : 0.0f, unit * 65536.0f, upper);
    }
}

// LONG: ranges of more than RUN chunks, whose f32 sums move on to doubles every RUN chunks: a longer chain rounds at the size of
// what it has gathered.  (In one kernel for both, 16 rows x 4096 x 4096, four chunks a range, took 15.7 us instead of 14.3.)
template <int NT, bool LONG>
__global__ void __launch_bounds__(AF_THREADS, NT <= 8 ? 2 : 1) gemv_affine_kernel(const AfParams p) {
    using Sum = std::conditional_t<LONG, double, float>;
    __shared__ Sum red[AF_WARPS * 2 * NT * AF_ROWS];      // [warp][activation row][weight row]
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    const int rank = blockIdx.x % p.ways, block = blockIdx.x / p.ways, wks = AF_WARPS / p.wr;
    const int wr = warp % p.wr, wk = warp / p.wr;
    const int groups = p.K / AG, slice = rank * wks + wk, slices = p.ways * wks;
    const int g0 = (int)((long long)groups * slice / slices), g1 = (int)((long long)groups * (slice + 1) / slices);
    const int tile0 = blockIdx.y * p.tpp, nt = min(p.tpp, p.tiles - tile0);

    uint32_t first[4];   // a row's first chunk: its place among the scales and biases, and 64 times that among the weights
#pragma unroll
    for (int i = 0; i < 4; ++i)
        first[i] = (uint32_t)min((block * p.wr + wr) * AF_ROWS + gid + 8 * i, p.N - 1) * (uint32_t)groups;   // (rows beyond N: read twice, not stored)
    struct Chunk {
        uint4 w[4];
        float s[4], b[4];
    };
    auto load = [&](int g, Chunk& c) {
        if (g < g1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) c.w[i] = ldg_stream(p.W + (size_t)(first[i] + g) * AG + tig * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) c.s[i] = __ldg(p.scales + (first[i] + g)), c.b[i] = __ldg(p.biases + (first[i] + g));
        }
    };
    float acc[NT][4];
    Sum* mine = red + (warp * 2 * NT + (tig >> 1)) * AF_ROWS + gid;   // (the even lane of a pair holds the pair's sums)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[t][i] = 0.0f;
            if (LONG && (tig & 1) == 0) mine[2 * t * AF_ROWS + 8 * i] = 0.0;
        }
    // digits of the next PF tiles, across the chunks: from L2 they take as long as several tiles' arithmetic
    constexpr int PF = NT < 2 ? 1 : NT <= 8 ? 2 : 4;
    static_assert(NT % PF == 0, "a tile's digits lie in the same registers in every chunk");
    uint4 q[PF];
    float2 u[PF];
    auto fetch = [&](int g, int t, int slot) {
        if (g < g1) {
            const size_t at = (size_t)g * p.tiles + tile0 + min(t, nt - 1);
            q[slot] = ld_ahead(p.digits + at * 32 + lane);
            u[slot] = ld_ahead(p.aux + at * 4 + tig);
        }
    };
    auto add = [&](int g, const Chunk& c) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const uint4 d = q[t % PF];
            const float2 a = u[t % PF];
            fetch(t + PF < NT ? g : g + 1, t + PF < NT ? t + PF : t + PF - NT, t % PF);
            int lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
            mma_u8s8(lo, c.w[0].x, c.w[1].x, c.w[0].y, c.w[1].y, d.x, d.y);
            mma_u8s8(hi, c.w[2].x, c.w[3].x, c.w[2].y, c.w[3].y, d.x, d.y);
            mma_u8s8(lo, c.w[0].z, c.w[1].z, c.w[0].w, c.w[1].w, d.z, d.w);
            mma_u8s8(hi, c.w[2].z, c.w[3].z, c.w[2].w, c.w[3].w, d.z, d.w);
            // |sum| <= 64 * 255 * 128 per plane: both planes together stay below 2^30
            acc[t][0] += fmaf((float)(lo[1] * 256 + lo[0]) * a.x, c.s[0], a.y * c.b[0]);
            acc[t][1] += fmaf((float)(lo[3] * 256 + lo[2]) * a.x, c.s[1], a.y * c.b[1]);
            acc[t][2] += fmaf((float)(hi[1] * 256 + hi[0]) * a.x, c.s[2], a.y * c.b[2]);
            acc[t][3] += fmaf((float)(hi[3] * 256 + hi[2]) * a.x, c.s[3], a.y * c.b[3]);
        }
    };
    Chunk c0, c1;
    load(g0, c0);
    load(g0 + 1, c1);
    pdl_wait();
#pragma unroll
    for (int t = 0; t < PF; ++t) fetch(g0, t, t);
    auto move_on = [&] {
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float v = acc[t][i] + __shfl_xor_sync(0xffffffffu, acc[t][i], 1);
                acc[t][i] = 0.0f;
                if ((tig & 1) == 0) mine[2 * t * AF_ROWS + 8 * i] = (LONG ? mine[2 * t * AF_ROWS + 8 * i] : (Sum)0) + (Sum)v;
            }
    };
    for (int g = g0; g < g1; g += 2) {
        add(g, c0);
        load(g + 2, c0);
        if (g + 1 < g1) add(g + 1, c1);
        load(g + 3, c1);
        if (LONG && ((g - g0) & (RUN - 1)) == RUN - 2) move_on();
    }
    move_on();
    cg::cluster_group cl = cg::this_cluster();
    if (p.ways > 1)
        cl.sync();
    else
        __syncthreads();
    const int rows = AF_ROWS * p.wr;
    for (int i = rank * AF_THREADS + threadIdx.x; i < rows * 2 * nt; i += p.ways * AF_THREADS) {
        const int r = i % rows, m = i / rows, n = block * rows + r, mg = 2 * tile0 + m;
        if (n >= p.N || mg >= p.M) continue;
        double sum = 0.0;   // of up to 64 ranges
        for (int c = 0; c < p.ways; ++c) {
            const Sum* src = p.ways > 1 ? cl.map_shared_rank(red, c) : red;
            for (int k = 0; k < wks; ++k) sum += (double)src[((k * p.wr + r / AF_ROWS) * 2 * NT + m) * AF_ROWS + r % AF_ROWS];
        }
        const float v = (float)sum;
        const size_t at = (size_t)mg * p.ldy + p.y_col0 + n;
        if (p.y_bf16)
            reinterpret_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16_rn(v);
        else
            reinterpret_cast<float*>(p.y)[at] = v;
    }
    if (p.ways > 1) cl.sync();   // the others have read this CTA's sums
}

}  // namespace

namespace rusty {

int launch_gemv_affine(rusty_cuda_ctx* ctx, const QLinearArgs& a) {
    AfParams p{};
    p.W = a.w;
    p.scales = a.scales;
    p.biases = a.biases;
    p.N = (int)a.N;
    p.K = (int)a.K;
    p.ldy = (int)a.ldy;
    p.y_col0 = (int)a.y_col0;
    p.y_bf16 = a.y_dtype == RUSTY_CUDA_BF16;
    const int groups = p.K / AG;
    const size_t xs = a.x_dtype == RUSTY_CUDA_BF16 ? 2 : 4, ys = p.y_bf16 ? 2 : 4;
    const size_t per_tile = (size_t)groups * (512 + 32);   // workspace bytes of two activation rows
    uint32_t most = (uint32_t)(tc_workspace_xq_bytes() / per_tile) * 2;
    if (most > 32768u) most = 32768u;
    if (most < 2) return fail(ctx, RUSTY_CUDA_ERR_UNSUPPORTED, "gemv_affine: the digit planes of K=%u do not fit the workspace", a.K);
    for (uint32_t m0 = 0; m0 < a.M; m0 += most) {
        p.M = (int)(a.M - m0 < most ? a.M - m0 : most);
        p.y = (char*)a.y + (size_t)m0 * a.ldy * ys;
        p.tiles = (p.M + 1) / 2;
        // Up to 24 activation rows share a pass over the weights (32 leave too few registers: 12288 x 2112 at 32 rows 60 us in
        // one pass, 47 in two); passes of equal width.
        const int passes = (p.tiles + 11) / 12;
        p.tpp = (p.tiles + passes - 1) / passes;
        uint32_t* digits = (uint32_t*)ctx->tc_ws;
        float2* aux = (float2*)((char*)ctx->tc_ws + (size_t)groups * p.tiles * 512);
        p.digits = (const uint4*)digits;
        p.aux = aux;
        const void* x = (const char*)a.x + (size_t)m0 * a.K * xs;
        const dim3 pg((unsigned)(p.K + 1023) / 1024, (unsigned)p.tiles * 2);
        cudaError_t e = xs == 2 ? launch_pdl(affine_prepare_kernel<__nv_bfloat16>, pg, dim3(256), 0, ctx->stream, (const __nv_bfloat16*)x, digits, aux, p.M, p.K, p.tiles)
                                : launch_pdl(affine_prepare_kernel<float>, pg, dim3(256), 0, ctx->stream, (const float*)x, digits, aux, p.M, p.K, p.tiles);
        if (e != cudaSuccess) return check_cuda(ctx, e, "affine_prepare");
        int rc = after_launch(ctx, "affine_prepare");
        if (rc) return rc;
        // Ranges of chunks a row group is cut into: the number for which waves x (chunks of a range + start and end, about two
        // chunks; a cluster, above eight ranges, about three more) is least.  4096 x 4096 at two rows: 16 ranges 7.1 us, 8 ranges
        // 9.5 us, 32 ranges (two waves) 10.9 us.
        const int row_groups = (p.N + AF_ROWS - 1) / AF_ROWS;
        const long long slots = (long long)ctx->sm_count * (p.tpp <= 8 ? 2 : 1);
        int slices = 1;
        long long least = LLONG_MAX;
        for (int s = 1; s <= 64 && s <= groups; s *= 2) {
            const long long ctas = ((long long)row_groups * s + AF_WARPS - 1) / AF_WARPS * passes;
            const long long cost = (ctas + slots - 1) / slots * ((groups + s - 1) / s + 2 + (s > AF_WARPS ? 3 : 0));
            if (cost < least) least = cost, slices = s;
        }
        const int wks = slices < AF_WARPS ? slices : AF_WARPS;
        p.wr = AF_WARPS / wks;
        p.ways = slices / wks;
        const dim3 grid((unsigned)((row_groups + p.wr - 1) / p.wr * p.ways), (unsigned)passes);
        const bool run_on = (groups + slices - 1) / slices > RUN;
        auto of = [&](auto nt) {
            constexpr int NT = decltype(nt)::value;
            return run_on ? gemv_affine_kernel<NT, true> : gemv_affine_kernel<NT, false>;
        };
        auto kern = p.tpp <= 1   ? of(std::integral_constant<int, 1>{})
                    : p.tpp <= 2 ? of(std::integral_constant<int, 2>{})
                    : p.tpp <= 4 ? of(std::integral_constant<int, 4>{})
                    : p.tpp <= 8 ? of(std::integral_constant<int, 8>{})
                                 : of(std::integral_constant<int, 12>{});
        e = launch_pdl_cluster(kern, grid, dim3(AF_THREADS), (unsigned)p.ways, 0, ctx->stream, p);
        if (e != cudaSuccess) return check_cuda(ctx, e, "gemv_affine");
        rc = after_launch(ctx, "gemv_affine");
        if (rc) return rc;
    }
    return RUSTY_CUDA_OK;
}

}  // namespace rusty
