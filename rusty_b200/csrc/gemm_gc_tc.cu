// Linear on the reference's own quantised format with f32 (or a few rows of bf16) activations, on the 5th-generation tensor
// cores (tcgen05 kind::i8, accumulators in tensor memory).
//
// Format (rusty-loader/src/lib.rs:155-218 for a weight stored [in,out]): u8 bytes, one f32 scale and bias per 64 consecutive
// OUTPUT features of an input row, w[k,n] = u[k,n] * s[k, n/64] + b[k, n/64]; re-laid-out once at create to bytes [out,in],
// scales and biases [N/64][K].  For the 64 output features of group g
//     y[m,n] = sum_k (x[m,k] * s_g[k]) * u[n,k]  +  sum_k x[m,k] * b_g[k],
// so the scales move over to the activations and the weight bytes enter the tensor core untouched.  A group's activations
// a = x (.) s_g exist nowhere in memory: a CTA owns one group (64 output features), up to 64 activation rows and a range of K,
// and its converter warps make them from x and s_g stage by stage.
//
// Arithmetic.  q = round(a * 2^e) with |q| < 2^31, e chosen per (row, group) so that the largest |a| of the WHOLE row times 2^e
// lies in [2^30, 2^31) (partial sums of different K ranges are then integers of one unit, and their order does not matter).
// q + 2^31 is four unsigned bytes: four planes of the A operand, no digit carries to work out; sum_k (q + 2^31) u is exact in
// int32 per plane (255 * 255 * K < 2^31 for K <= 32768) and int64 together, and 2^31 * sum_k u[n,k], a property of the weight
// row, is taken off once at the end.  The largest |a| has to be the true one: max|x| max|s| over a stretch of k is far above it
// where an outlier of x meets a small scale, and every factor of two of that is a bit of all other activations (an outlier of
// 10^6 on a scale of 10^-6 cost 1e-3 of the result).  Up to eight rows the CTAs multiply x and s_g once more for it.  Larger
// batches know the largest |x| of a stage (128 k), its place and the second largest: the product at that place is one of the
// row's, and second largest times the stage's largest |s| bounds the others; all products of a stage are taken only where
// that bound has a larger exponent than the largest product so far (hardly ever for weights and activations of one scale).
// The bias term is as large as the integer part and of the other sign for weights around zero, so it is summed as exactly: with
// b = r s it is sum_k a[m,k] r[k], and r, at create, becomes 32 bits below the group's largest |r|, four more "weight rows" of
// unsigned bytes per group (and a row of ones, for the sum of q that takes the offset off again).  An output is then
// sum_k a (u + r) with nothing rounded but a.  (Summed in f32 beside the conversion, 16 terms at a time and those in double, the
// bias alone cost 1.0e-7 of an output and everything else 0.6e-7; in double, 24 % of the time of a 512-row layer.)  A group with
// a b of more than 4096 scales has no such r: its bias term is summed in double after the last stage.
//
// Roles: warp 0 brings weights, bytes of r and scales by TMA into a ring of stages (128 k each), starting before
// griddepcontrol.wait; warp 1 issues the MMAs (M = 128: 32 rows x 4 planes, row 4m + p; N = 64 output features, 5 columns for the
// bias and 11 nobody reads; K = 32); eight converter warps take rows cw, cw + 8, ..., 128 k of a row at a time (a lane's four
// neighbours: one 16-byte load of x, one 4-byte store per plane, no bank conflicts under the 128-byte swizzle), and are the
// epilogue in the end.  Two CTAs fit an SM.
// A K range per CTA of a cluster (1, 2 or 4) where there are too few groups; their int64 sums meet in distributed shared memory.
//
// What bounds it: few rows, the weight stream and the fixed part of a launch; 4096 x 4096, per call in a graph: 1 row 8.2 us, 4 rows
// 10.5, 8 rows 12.8, 13 rows 12.4, 32 rows 16.3 (a GEMV kernel with a pair of rows per CTA: 4 rows 13.2, 32 rows 58.6);
// 12288 x 2112, whose last stage is half empty (rows padded at create), 1 row 11.1 us (on CUDA cores 15.5).
// Beyond 32 rows see the kernel for them, below.
#include <cooperative_groups.h>

#include <climits>
#include <cstdlib>

#include "tc_common.cuh"

using namespace rusty_tc;
namespace cg = cooperative_groups;

namespace {

constexpr int GN = 64;                         // output features per CTA = one group
constexpr int SK = 128;                        // k per stage
constexpr int CW = 8;                          // converter / epilogue warps
constexpr int GC_THREADS = 32 * (2 + CW);
constexpr int NC = 80;                         // columns of the MMA: GN, RD of r's bytes, one of ones (a multiple of 16)
constexpr int RD = 4;
constexpr int W_BYTES = GN * SK;               // weight bytes of a stage
// + eight rows for r and ones (9 KiB: every stage starts on 1 KiB; what lies behind a stage multiplies into columns nobody reads)
constexpr int STAGE_BYTES = W_BYTES + 8 * SK;
constexpr int S_BYTES = SK * 4;                // scales of a stage, in a ring of their own behind it
constexpr int TX_BYTES = W_BYTES + RD * SK + S_BYTES;
constexpr int R_MAX = 4096;                    // largest |b / s| that goes to the tensor core
constexpr int BSUM = 4;                        // K ranges start at multiples of this many stages
constexpr int MAX_STAGES = 8;
// The A operand of a stage, 128 rows of 128 bytes per row block.  A CTA of few rows fills the first 32 RPW rows only, and its
// buffers lie that close together: the MMA then multiplies what follows (other buffers, the ring) into rows nobody reads.
constexpr int A_BYTES = 32 * 1024;
template <int RPW>
constexpr int A_PITCH = RPW * 4096;
template <int RPW>
constexpr int A_BUFS = 8 / RPW;

struct GcParams {
    const float* scales;         // [N/64][K]
    const float* biases;         // [N/64][K]
    const uint8_t* rbytes;       // [N/64][K/128][RD * 128]: r's rows of a stage, swizzled as they lie in shared memory
    const int* rinfo;            // [N/64][8]: byte sums of r's four rows; r's unit is 2^-rinfo[4] (INT_MIN: a group without r)
    const float* smax;           // [N/64][K/128]: largest |scale| of a stage
    const int* rowsum;           // [N]: sum of a weight row's bytes
    const void* x;               // the caller's rows; RPW > 1: gc_prepare_kernel's copy [K/128][Mp][128]
    size_t xstep;                // elements from a stage to the next: 128, or 128 Mp
    const uint2* xtop;           // RPW > 1: [M][K/128], a stage's largest |x|s, made by gc_prepare_kernel
    void* y;
    const void* residual;        // null, or added to every output
    int M, N, K;
    int nst;                     // stages along K
    int ways;                    // K ranges = cluster size
    int stages;                  // ring depth
    int ldy, y_col0, y_bf16;
    rusty_cuda_dev_status* status;
    int n_peers;                          // other ranks whose copy of y also receives every output (peer.cu); 0: none
    long long peer_delta[PEER_MAX_RANKS];
};

// Magnitudes are compared as bits: a NaN or an infinity is above every number.
__device__ __forceinline__ uint32_t abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t abs_max(const float4& v) { return max(max(abs_bits(v.x), abs_bits(v.y)), max(abs_bits(v.z), abs_bits(v.w))); }
// Largest of top and the magnitudes of four products, rounded as the converters round them.  Two three-operand maxima that take the
// magnitudes by themselves: every CTA walks all rows x K of them (as integers, four more instructions).  A NaN stays one.
__device__ __forceinline__ float top_of(float top, const float4& x, const float4& s) {
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(__fmul_rn(x.x, s.x)), "f"(__fmul_rn(x.y, s.y)));
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(__fmul_rn(x.z, s.z)), "f"(__fmul_rn(x.w, s.w)));
    return top;
}

__device__ __forceinline__ float4 ldg_x4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }   // of the weight's own tables
// Activations: not through the read-only path, which wants data nobody writes while the kernel runs; this kernel is there while the
// ones in front of it still write x, its copy and xtop (at the same addresses on every call).
template <typename XT>
__device__ __forceinline__ float4 ld_x4(const XT* p) {
    if constexpr (sizeof(XT) == 4) {
        return *reinterpret_cast<const float4*>(p);
    } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                           __uint_as_float(raw.y & 0xffff0000u));
    }
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// Largest |a| (as float bits) -> exponent e of the row's unit 2^-e: |a| * 2^e in [2^30, 2^31).  Very small ones stop at 2^127.
__device__ __forceinline__ int unit_exponent(uint32_t bits) {
    return min(157 - (int)(bits >> 23), 127);
}

// What the outputs of a row and group share: its unit 2^-e (NaN: poisoned) and what r adds to the sums, from the sums with r's bytes and
// ones.
__device__ __forceinline__ double2 row_terms(const long long (&ext)[RD + 1], const int4& rsum, int runit, int e, int K) {
    // sum_k q r: the offsets off the planes, then r's own 2^31 off its top byte
    const long long sq = ext[RD] - ((long long)K << 31);
    const double top = (double)(ext[0] - ((long long)rsum.x << 31) - 128 * sq);
    const double rest = (double)(ext[1] - ((long long)rsum.y << 31)) * 65536.0 + (double)(ext[2] - ((long long)rsum.z << 31)) * 256.0 +
                        (double)(ext[3] - ((long long)rsum.w << 31));
    const double r_unit = runit == INT_MIN ? 0.0 : __longlong_as_double((long long)(1023 - runit) << 52);
    // 2^-e as a double from its exponent field; the sum is exact up to here
    return make_double2((top * 16777216.0 + rest) * r_unit, e == INT_MIN ? (double)__int_as_float(0x7fc00000) : __longlong_as_double((long long)(1023 - e) << 52));
}
__device__ __forceinline__ void store_output(const GcParams& p, float f, size_t at) {
    auto put = [&](auto* y0, auto value) {
        auto* dst = y0 + at;
        *dst = value;
#pragma unroll
        for (int r = 0; r < PEER_MAX_RANKS - 1; ++r)   // the same element of every other rank's y, over NVLink
            if (r < p.n_peers) *reinterpret_cast<decltype(dst)>(reinterpret_cast<char*>(dst) + p.peer_delta[r]) = value;
    };
    if (p.y_bf16) {
        if (p.residual) f += __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.residual)[at]);
        put(reinterpret_cast<__nv_bfloat16*>(p.y), __float2bfloat16_rn(f));
    } else {
        if (p.residual) f = __fadd_rn(reinterpret_cast<const float*>(p.residual)[at], f);
        put(reinterpret_cast<float*>(p.y), f);
    }
}

// Up to 32 rows.  XT: type of the caller's x (RPW = 1 reads it as it is).  RPW: rows per converter warp (1, 2 or 4).  MEET (RPW = 1): the cluster's CTAs share the look for the largest products (an instance of its own: the code of
// both in one cost calls that do not meet 0.3 us in instruction fetches).
template <typename XT, int RPW, bool MEET = false>
__global__ void __launch_bounds__(GC_THREADS, 2) qlinear_gc_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ GcParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int PITCH = A_PITCH<RPW>, BUFS = A_BUFS<RPW>, TCOLS = 128;
    uint8_t* sA = smem;                                              // [BUFS] x PITCH
    uint8_t* sIn = smem + A_BYTES;                                   // [stages][STAGE_BYTES]
    uint8_t* sSc = sIn + (size_t)p.stages * STAGE_BYTES;             // [stages][S_BYTES]
    uint64_t* in_full = reinterpret_cast<uint64_t*>(sSc + (size_t)p.stages * S_BYTES);
    uint64_t* in_empty = in_full + MAX_STAGES;
    uint64_t* a_full = in_empty + MAX_STAGES;
    uint64_t* a_empty = a_full + MAX_STAGES;
    uint64_t* d_full = a_empty + MAX_STAGES;
    double2* s_bias = reinterpret_cast<double2*>(d_full + 2);        // [32]: a group without r: this K range's bias term, in two parts
    int* s_exp = reinterpret_cast<int*>(s_bias + 32);           // [32]: e of a row, or INT_MIN: poisoned
    uint32_t* s_top = reinterpret_cast<uint32_t*>(s_exp + 32);  // [32]: largest |a| of a row (bits, its exponent at least)
    float* s_smax = reinterpret_cast<float*>(s_top + 32);       // [K / 128]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_smax + p.nst);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_id(), lane = threadIdx.x & 31;
    const int g = blockIdx.y;
    const int way = (int)blockIdx.x % p.ways, m0 = ((int)blockIdx.x / p.ways) * (32);
    const int rows = min(32, p.M - m0);
    // K ranges start at multiples of BSUM stages: the f32 pieces of the bias sum do not depend on how K is cut
    const int nb = (p.nst + BSUM - 1) / BSUM;
    const int st0 = nb * way / p.ways * BSUM, st1 = min(p.nst, nb * (way + 1) / p.ways * BSUM);
    const int active = min(CW, rows);          // converter warps that arrive on a stage
    pdl_launch_dependents();
    // The scales are needed before the first weights are: asked for ahead of the ring's 70 KB.  Up to eight rows the first
    // ones into registers, and where the cluster meets a CTA looks for the largest products of its own K range only.
    constexpr int AHEAD = 4;          // stages whose scales a converter warp holds while the rows go by (RPW = 1)
    const int top0 = MEET ? st0 : 0, top1 = MEET ? st1 : p.nst;
    const float* gs = p.scales + (size_t)g * p.K + lane * 4;
    float4 sv[AHEAD];
    auto fetch_scales = [&](int st) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (st + u * CW < top1) sv[u] = ldg_x4(gs + (st + u * CW) * SK);
    };
    if (warp >= 2) {
        if constexpr (RPW == 1) fetch_scales(top0 + warp - 2);
        for (int k = (top0 + (RPW == 1 ? AHEAD * CW : 0)) * SK + ((int)threadIdx.x - 64) * 32; k < top1 * SK; k += 32 * CW * 32)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.scales + (size_t)g * p.K + k));
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&in_full[s], 1);
            mbar_init(&in_empty[s], 1);
        }
        for (int s = 0; s < BUFS; ++s) {
            mbar_init(&a_full[s], (uint32_t)active);
            mbar_init(&a_empty[s], 1);
        }
        mbar_init(d_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + 32) {
        s_top[threadIdx.x - 64] = 0u;
        s_bias[threadIdx.x - 64] = make_double2(0.0, 0.0);
    }
    if (warp == 1) {
        // the rows of ones (by a warp without loads in flight: the fence would wait for them)
        for (int s = 0; s < p.stages; ++s) sts32(smem_u32(sIn + (size_t)s * STAGE_BYTES + W_BYTES + RD * SK) + lane * 4, 0x01010101u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tmem_alloc(tmem_slot, TCOLS);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // (both for the very end)
    const int4 rsum = warp >= 2 ? __ldg(reinterpret_cast<const int4*>(p.rinfo) + 2 * g) : make_int4(0, 0, 0, 0);
    const int runit = warp >= 2 ? __ldg(p.rinfo + 8 * g + 4) : 0;
    const int rowsum_n = warp >= 2 ? __ldg(p.rowsum + g * GN + ((threadIdx.x - 64) & (GN - 1))) : 0;

    if (MEET && warp < 2) cluster_arrive();   // for the converters' meeting; waited for at the end
    if (warp == 0) {
        // ------------------------------ producer ------------------------------
        // several row tiles read the weights again (from L2); one tile: a single pass
        const uint64_t pol = p.M > 32 ? policy_evict_last() : policy_evict_first();
        int s = 0, issued = 0;
        uint32_t ph = 0;
        for (int st = st0; st < st1; ++st, ++issued) {
            if (!mbar_wait(&in_empty[s], ph ^ 1u, abort_flag, p.status, 41)) break;
            uint8_t* dst = sIn + (size_t)s * STAGE_BYTES;
            if (elect_one()) {
                mbar_expect_tx(&in_full[s], (uint32_t)TX_BYTES);
                tma_load_2d(dst, &map_w, st * SK, g * GN, &in_full[s], pol);
                bulk_load(dst + W_BYTES, p.rbytes + ((size_t)g * p.nst + st) * (RD * SK), RD * SK, &in_full[s]);
                bulk_load(sSc + (size_t)s * S_BYTES, p.scales + (size_t)g * p.K + st * SK, S_BYTES, &in_full[s]);
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        // whatever happened to the other roles: no copy is in flight when this CTA's shared memory is used for other things
        for (int j = max(0, issued - p.stages); j < issued; ++j) {
            const long long t0 = clock64();
            while (!mbar_try_wait(&in_full[j % p.stages], (uint32_t)(j / p.stages) & 1u) && clock64() - t0 < 4000000ll) {}
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ----------------------------
        // u8 x u8 -> s32, both K-major: c_format = S32 (2) @4, a_format = b_format = U8 (0), N >> 3 @17, M >> 4 @24
        constexpr uint32_t idesc = (2u << 4) | ((uint32_t)(NC >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        int s = 0, ab = 0;
        uint32_t ph = 0, aph = 0;
        for (int st = st0; st < st1; ++st) {
            if (!mbar_wait(&in_full[s], ph, abort_flag, p.status, 42) || !mbar_wait(&a_full[ab], aph, abort_flag, p.status, 43)) break;
            tc_fence_after();
            const uint64_t da = make_smem_desc(smem_u32(sA + (size_t)ab * PITCH)), db = make_smem_desc(smem_u32(sIn + (size_t)s * STAGE_BYTES));
            if (elect_one()) {
#pragma unroll
                for (int k4 = 0; k4 < SK / 32; ++k4)
                    umma_i8(tmem_base, da + (uint64_t)(2 * k4), db + (uint64_t)(2 * k4), idesc, (st > st0 || k4 > 0) ? 1u : 0u);
                umma_commit(&in_empty[s]);
                umma_commit(&a_empty[ab]);
                if (st == st1 - 1) umma_commit(d_full);
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; ph ^= 1u; }
            if (++ab == BUFS) { ab = 0; aph ^= 1u; }
        }
    } else {
        // ------------------------------ converters ----------------------------
        const int cw = warp - 2, ct = threadIdx.x - 64;
        if constexpr (RPW > 1)      // the weight's own: before the wait
            for (int st = ct; st < p.nst; st += 32 * CW) s_smax[st] = __ldg(p.smax + (size_t)g * p.nst + st);
        pdl_wait();   // x (and xtop) may come from the previous kernel
        if constexpr (RPW > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * CW) : "memory");
        // Up to four rows: two warps a row, every other BSUM stages each (a ring of 8 stages and 8 A buffers: a warp meets the
        // same slots again and again, one phase further each time).
        const bool shared_rows = RPW == 1 && rows <= 4;
        const int row_w = shared_rows ? cw & 3 : cw;                    // this warp's first row; further ones 8 apart
        const int sub = shared_rows ? cw >> 2 : 0;
        const int nr = row_w < rows ? (rows - row_w + 7) / 8 : 0;       // rows of this warp
        if constexpr (RPW == 1) {
            // every warp takes an eighth of the range of every row
            const XT* xr = reinterpret_cast<const XT*>(p.x) + (size_t)m0 * p.K + lane * 4;
            for (int kb = top0 + cw; kb < top1; kb += AHEAD * CW) {
                if (kb != top0 + cw) fetch_scales(kb);
                for (int m = 0; m < rows; ++m) {
                    float4 v[AHEAD];
#pragma unroll
                    for (int u = 0; u < AHEAD; ++u)
                        if (kb + u * CW < top1) v[u] = ld_x4<XT>(xr + (size_t)m * p.K + (kb + u * CW) * SK);
                    float most = 0.0f;
#pragma unroll
                    for (int u = 0; u < AHEAD; ++u)
                        if (kb + u * CW < top1) most = top_of(most, v[u], sv[u]);
                    const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
                    if (lane == 0) atomicMax(s_top + m, top);
                }
            }
            if constexpr (MEET) {
                cluster_arrive();
                cluster_wait();
            } else {
                asm volatile("bar.sync 1, %0;" ::"n"(32 * CW) : "memory");
            }
        } else {
            // (the unit depends on the exponent alone, and that is the true one here as well: a row has the same in any batch)
            const uint2* xt = p.xtop + (size_t)(m0 + row_w) * p.nst;
            const float* xr = reinterpret_cast<const float*>(p.x) + (size_t)(m0 + row_w) * SK + lane * 4;
            auto rest_bound = [&](uint2 v, int st) { return abs_bits(__fmul_rn(__uint_as_float(v.y & 0xffff0000u), s_smax[st])); };
            uint32_t top[RPW], rest[RPW];
#pragma unroll
            for (int i = 0; i < RPW; ++i) top[i] = rest[i] = 0u;
            for (int st = lane; st < p.nst; st += 32) {
                uint2 v[RPW];
                float s1[RPW];
#pragma unroll
                for (int i = 0; i < RPW; ++i)
                    if (i < nr) v[i] = xt[(size_t)(8 * i) * p.nst + st];
#pragma unroll
                for (int i = 0; i < RPW; ++i)
                    if (i < nr) s1[i] = __ldg(p.scales + (size_t)g * p.K + st * SK + (v[i].y & 0xffffu));
#pragma unroll
                for (int i = 0; i < RPW; ++i)
                    if (i < nr) {
                        top[i] = max(top[i], abs_bits(__fmul_rn(__uint_as_float(v[i].x), s1[i])));
                        rest[i] = max(rest[i], rest_bound(v[i], st));
                    }
            }
#pragma unroll
            for (int i = 0; i < RPW; ++i)
                if (i < nr) {
                    top[i] = __reduce_max_sync(0xffffffffu, top[i]);
                    if (__any_sync(0xffffffffu, rest[i] >> 23 > top[i] >> 23)) {
                        for (int base = 0; base < p.nst; base += 32) {
                            const int st = base + lane;
                            const uint32_t b = st < p.nst ? rest_bound(xt[(size_t)(8 * i) * p.nst + st], st) >> 23 : 0u;
                            uint32_t todo = __ballot_sync(0xffffffffu, b > top[i] >> 23);
                            auto stage_max = [&](int s) { return __float_as_uint(top_of(0.0f, ld_x4(xr + (size_t)s * p.xstep + i * (8 * SK)), ldg_x4(gs + s * SK))); };
                            while (todo) {     // two stages at a time
                                const int sa = base + __ffs(todo) - 1;
                                todo &= todo - 1;
                                const int sb = todo ? base + __ffs(todo) - 1 : sa;
                                todo &= todo - 1;
                                top[i] = max(top[i], __reduce_max_sync(0xffffffffu, max(stage_max(sa), stage_max(sb))));
                                todo &= __ballot_sync(0xffffffffu, b > top[i] >> 23);
                            }
                        }
                    }
                    if (lane == 0) s_top[row_w + 8 * i] = top[i];
                }
            __syncwarp();
        }
        float scale[RPW];
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
            scale[i] = 0.0f;
            if (i < nr) {
                uint32_t top = s_top[row_w + 8 * i];
                if constexpr (MEET)
                    for (int w = 1; w < p.ways; ++w) top = max(top, cg::this_cluster().map_shared_rank(s_top, (way + w) % p.ways)[row_w]);
                const bool finite = top < 0x7f800000u;
                const int e = unit_exponent(top);
                // 2^e: between 2^-97 (products near the largest float) and 2^127, always a normal number
                scale[i] = finite ? __uint_as_float((uint32_t)(127 + e) << 23) : 0.0f;
                if (lane == 0) s_exp[row_w + 8 * i] = finite ? e : INT_MIN;
            }
        }
        if (nr > 0) {
            // Work items (row, stage) in groups of four: 4 stages of one row, 2 of two, one of four.  The x
            // values of a group are loaded while the group before it is converted.
            constexpr int GS = 4 / RPW;                         // stages of a group
            const int step = shared_rows ? 2 * BSUM : GS;       // from one group's first stage to the next one's
            // where this lane's four bytes of plane pl go: row 4m + pl of the tile, 16-byte chunk lane / 4 under the 128-byte
            // swizzle; m's parity is the first row's
            uint32_t off[4];
#pragma unroll
            for (int pl = 0; pl < 4; ++pl)
                off[pl] = smem_u32(sA) + (uint32_t)(row_w * 512 + pl * 128 + ((((lane >> 2) ^ pl) << 4) ^ ((row_w & 1) << 6)) + (lane & 3) * 4);
            const uint32_t sv0 = smem_u32(sSc) + lane * 16;
            bool ok = true;
            // (RPW > 1: the copy's rows are 512 bytes, and there are rows enough for the whole tile: no checks, constant offsets)
            const XT* xw = reinterpret_cast<const XT*>(p.x) + (RPW == 1 ? (size_t)(m0 + row_w) * p.K : (size_t)(m0 + row_w) * SK) + lane * 4 + st0 * p.xstep;
            auto fetch = [&](float4 (&v)[4], const XT* q, int st) {
#pragma unroll
                for (int h = 0; h < GS; ++h)
                    if (st + h < st1)
#pragma unroll
                        for (int i = 0; i < RPW; ++i) v[i * GS + h] = ld_x4<XT>(q + h * p.xstep + i * (8 * SK));
            };
            uint4 sq;
            int ab = 0;
            uint32_t at[4];
            // waits for stage idx's scales and biases and for its A buffer
            auto enter = [&](int idx) {
                // eight stages and a power of two of buffers
                const int slot = idx & (MAX_STAGES - 1);
                const uint32_t ph = ((uint32_t)idx / MAX_STAGES) & 1u, aph = ((uint32_t)idx / BUFS) & 1u;
                ab = idx & (BUFS - 1);
                if (!mbar_wait(&in_full[slot], ph, abort_flag, p.status, 44)) return false;
                sq = lds128(sv0 + (uint32_t)slot * S_BYTES);
                if (!mbar_wait(&a_empty[ab], aph ^ 1u, abort_flag, p.status, 45)) return false;
#pragma unroll
                for (int pl = 0; pl < 4; ++pl) at[pl] = off[pl] + (uint32_t)ab * PITCH;
                return true;
            };
            auto item = [&](const float4& x4, int r) {
                const int q0 = __float2int_rn(__fmul_rn(x4.x, __uint_as_float(sq.x)) * scale[r]);
                const int q1 = __float2int_rn(__fmul_rn(x4.y, __uint_as_float(sq.y)) * scale[r]);
                const int q2 = __float2int_rn(__fmul_rn(x4.z, __uint_as_float(sq.z)) * scale[r]);
                const int q3 = __float2int_rn(__fmul_rn(x4.w, __uint_as_float(sq.w)) * scale[r]);
                // 4 integers x 4 bytes -> 4 planes x 4 k; plane 0 is the top byte, its sign bit flipped: q + 2^31
                const uint32_t t0 = __byte_perm(q0, q1, 0x5140), t1 = __byte_perm(q2, q3, 0x5140);
                const uint32_t t2 = __byte_perm(q0, q1, 0x7362), t3 = __byte_perm(q2, q3, 0x7362);
                sts32(at[0] + (uint32_t)(r * 4096), __byte_perm(t2, t3, 0x7632) ^ 0x80808080u);
                sts32(at[1] + (uint32_t)(r * 4096), __byte_perm(t2, t3, 0x5410));
                sts32(at[2] + (uint32_t)(r * 4096), __byte_perm(t0, t1, 0x7632));
                sts32(at[3] + (uint32_t)(r * 4096), __byte_perm(t0, t1, 0x5410));
            };
            // hands the stage's rows to the MMA
            auto leave = [&] {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[ab]);
            };
            float4 xa[4], xb[4];
            auto convert = [&](const float4 (&v)[4], int st) {
#pragma unroll
                for (int h = 0; h < GS; ++h) {
                    if (!ok || st + h >= st1) return;
                    if (!enter(st + h - st0)) { ok = false; return; }
#pragma unroll
                    for (int i = 0; i < RPW; ++i) item(v[i * GS + h], i);
                    leave();
                }
            };
            int st = st0 + sub * BSUM;
            xw += (size_t)(sub * BSUM) * p.xstep;
            const size_t stride = (size_t)step * p.xstep;
            fetch(xa, xw, st);
            for (; ok && st < st1; st += 2 * step) {
                fetch(xb, xw + stride, st + step);
                convert(xa, st);
                xw += 2 * stride;
                fetch(xa, xw, st + 2 * step);
                convert(xb, st + step);
            }
            if (runit == INT_MIN && sub == 0) {
                // A group without r: x . b in double.  Upper 24 bits and the rest of every four terms are added up apart: exact
                // sums, whatever the K ranges.
                const XT* xb = reinterpret_cast<const XT*>(p.x) + (RPW == 1 ? (size_t)(m0 + row_w) * p.K : (size_t)(m0 + row_w) * SK) + lane * 4;
                const float* gb = p.biases + (size_t)g * p.K + lane * 4;
                for (int i = 0; i < nr; ++i) {
                    double hi = 0.0, lo = 0.0;
                    for (int st = st0; st < st1; ++st) {
                        const float4 x4 = ld_x4<XT>(xb + (size_t)st * p.xstep + i * (RPW == 1 ? 8 * p.K : 8 * SK)), b4 = ldg_x4(gb + st * SK);
                        const double d = fma((double)x4.x, (double)b4.x, fma((double)x4.y, (double)b4.y, fma((double)x4.z, (double)b4.z, (double)x4.w * (double)b4.w)));
                        const double u = __hiloint2double(__double2hiint(d), __double2loint(d) & (int)0xe0000000);
                        hi += u;
                        lo += d - u;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        hi += __shfl_xor_sync(0xffffffffu, hi, o);
                        lo += __shfl_xor_sync(0xffffffffu, lo, o);
                    }
                    if (lane == 0) s_bias[row_w + 8 * i] = make_double2(hi, lo);
                }
            }
        }
        // ------------------------------ epilogue, first half ------------------
        // accumulators -> shared memory as [warp][row 4m + p][column], in the memory of the A tiles: every MMA has read them once
        // d_full is reached
        if (st1 > st0) mbar_wait(d_full, 0, abort_flag, p.status, 46);
    }
    // All K ranges of a tile: bytes -> int64 sums per output, exact, parked in shared memory; then each CTA of the cluster adds
    // up and writes its share of the rows.
    // (a wait that gave up leaves the loops above in every role; the barriers below are reached all the same)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    constexpr int LDW = 37;                                            // words between rows of a warp's corner: no bank conflicts
    uint32_t* s_raw = reinterpret_cast<uint32_t*>(smem);               // [CW][32][LDW]
    long long* s_sum = reinterpret_cast<long long*>(smem + 40 * 1024); // [32][GN]
    long long* s_ext = s_sum + 32 * GN;                           // [32][RD + 1]: the bias columns
    const bool failed = *abort_flag != 0;
    if (warp >= 2 && !failed) {
        const int cw = warp - 2, q = warp & 3, half = cw >> 2;         // lane quarter of tensor memory, half of the columns
        uint32_t* mine = s_raw + (size_t)cw * 32 * LDW;
        const int row0 = q * 8;
        if (row0 < rows) {
            const uint32_t from = tmem_base + ((uint32_t)(q * 32) << 16);
            uint32_t v[2][16], ext[16];
#pragma unroll
            for (int c = 0; c < 2; ++c) tmem_ld16(from + half * 32 + c * 16, v[c]);
            if (half == 1) tmem_ld16(from + GN, ext);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int e = 0; e < 16; ++e) mine[lane * LDW + c * 16 + e] = v[c][e];
            if (half == 1)
#pragma unroll
                for (int e = 0; e <= RD; ++e) mine[lane * LDW + 32 + e] = ext[e];
            __syncwarp();
            auto sum_at = [&](int m, int c) {
                const uint32_t* r = mine + (4 * m) * LDW + c;
                return ((((long long)r[0] * 256 + r[LDW]) * 256 + r[2 * LDW]) * 256) + r[3 * LDW];
            };
            // a loop over the rows there are and not its copies: code that runs once waits for its instructions
#pragma unroll 1
            for (int m = 0; m < min(8, rows - row0); ++m) {
                s_sum[(size_t)(row0 + m) * GN + half * 32 + lane] = sum_at(m, lane);
                if (half == 1 && lane <= RD) s_ext[(size_t)(row0 + m) * (RD + 1) + lane] = sum_at(m, 32 + lane);
            }
        }
        tc_fence_before();
    }
    cg::cluster_group cl = cg::this_cluster();
    if (MEET && warp < 2) cluster_wait();
    if (p.ways > 1) cl.sync();
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TCOLS);
    }
    if (warp >= 2 && !failed) {
        const int t = threadIdx.x - 64, n = t & (GN - 1);              // 256 threads: 64 columns, every fourth row
        const int col = g * GN + n;
        const long long rs = (long long)rowsum_n << 31;
        for (int j = (t >> 6) + 4 * way; j < rows; j += 4 * p.ways) {
            long long sum = 0, ext[RD + 1] = {0, 0, 0, 0, 0};
            for (int w = 0; w < p.ways; ++w) {
                sum += p.ways > 1 ? cl.map_shared_rank(s_sum, w)[(size_t)j * GN + n] : s_sum[(size_t)j * GN + n];
                const long long* se = (p.ways > 1 ? cl.map_shared_rank(s_ext, w) : s_ext) + (size_t)j * (RD + 1);
#pragma unroll
                for (int i = 0; i <= RD; ++i) ext[i] += se[i];
            }
            double bhi = 0.0, blo = 0.0;
            if (runit == INT_MIN)
                for (int w = 0; w < p.ways; ++w) {
                    const double2 b = p.ways > 1 ? cl.map_shared_rank(s_bias, w)[j] : s_bias[j];
                    bhi += b.x;
                    blo += b.y;
                }
            const double2 terms = row_terms(ext, rsum, runit, s_exp[j], p.K);
            store_output(p, __double2float_rn(((double)(sum - rs) + terms.x) * terms.y + (bhi + blo)), (size_t)(m0 + j) * p.ldy + p.y_col0 + col);
        }
    }
    if (p.ways > 1) cl.sync();   // the others have read this CTA's sums
}

// ---- more than 32 rows ------------------------------------------------------------------------------------------------------
// The same arithmetic, tables and meeting of K ranges on tiles of 64 rows x TWO groups, one CTA an SM with sixteen converter warps:
// four rows of x in a warp's registers are multiplied by the scales of both groups before the next four are needed, and x crosses
// L2 -> SM half as often.  512 x 4096 x 4096 takes 92 us; one group a CTA of eight converter warps, two CTAs an SM: 112.  What bounds it: a
// stage takes 2000 cycles, of which the conversions to integers need 1130 (16 an SM a clock), the MMAs 640 and the shared-memory pipe
// 1300; the converters meet at two buffers of A, and 256 CTAs are 1.7 waves of 148.
constexpr int WG = 2, WCW = 16, WROWS = 64, WR = WROWS / WCW;      // groups, converter warps, rows of a tile, rows a warp
constexpr int W_THREADS = 32 * (2 + WCW);
constexpr int W_ABUF = 32 * 1024;              // A operand of a stage and group: 64 rows x 4 planes x 128 bytes
constexpr int W_IN = WG * STAGE_BYTES, W_SC = WG * S_BYTES;
constexpr int W_LDW = 33;                      // words between rows of a warp's corner in the epilogue: no bank conflicts
constexpr size_t W_SUM_AT = (size_t)WCW * 32 * W_LDW * 4 + 512;    // the sums' place behind the corners (16-byte aligned)

// a * s, two at a time, each half rounded like __fmul_rn
__device__ __forceinline__ void mul2(float& r0, float& r1, float a0, float a1, float s0, float s1) {
    asm("{\n\t.reg .b64 a, s;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 s, {%4, %5};\n\tmul.rn.f32x2 a, a, s;\n\tmov.b64 {%0, %1}, a;\n\t}"
        : "=f"(r0), "=f"(r1)
        : "f"(a0), "f"(a1), "f"(s0), "f"(s1));
}

__global__ void __launch_bounds__(W_THREADS, 1) qlinear_gc_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ GcParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = smem;                                              // [2][WG] x W_ABUF
    uint8_t* sIn = smem + 2 * WG * W_ABUF;                           // [stages][WG] x STAGE_BYTES
    uint8_t* sSc = sIn + (size_t)p.stages * W_IN;                    // [stages][WG] x S_BYTES
    uint64_t* in_full = reinterpret_cast<uint64_t*>(sSc + (size_t)p.stages * W_SC);
    uint64_t* in_empty = in_full + MAX_STAGES;
    uint64_t* a_full = in_empty + MAX_STAGES;                        // [2]
    uint64_t* a_empty = a_full + 2;
    uint64_t* d_full = a_empty + 2;
    double2* s_bias = reinterpret_cast<double2*>(d_full + 2);        // [WG][64]: a group without r: this K range's bias term, in two parts
    int* s_exp = reinterpret_cast<int*>(s_bias + WG * WROWS);        // [WG][64]: e of a row, or INT_MIN: poisoned
    float* s_smax = reinterpret_cast<float*>(s_exp + WG * WROWS);    // [WG][K / 128]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_smax + WG * p.nst);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_id(), lane = threadIdx.x & 31;
    const int groups = p.N / GN;
    // an odd last group is computed twice and stored once
    auto group_of = [&](int q) { return min((int)blockIdx.y * WG + q, groups - 1); };
    const int way = (int)blockIdx.x % p.ways, m0 = ((int)blockIdx.x / p.ways) * WROWS;
    const int rows = min(WROWS, p.M - m0);
    const int nb = (p.nst + BSUM - 1) / BSUM;
    const int st0 = nb * way / p.ways * BSUM, st1 = min(p.nst, nb * (way + 1) / p.ways * BSUM);
    const int active = min(WCW, rows);         // converter warps that arrive on a stage
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&in_full[s], 1);
            mbar_init(&in_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&a_full[s], (uint32_t)active);
            mbar_init(&a_empty[s], 1);
        }
        mbar_init(d_full, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + WG * WROWS) s_bias[threadIdx.x - 64] = make_double2(0.0, 0.0);
    if (warp == 1) {
        for (int s = 0; s < p.stages * WG; ++s) sts32(smem_u32(sIn + (size_t)s * STAGE_BYTES + W_BYTES + RD * SK) + lane * 4, 0x01010101u);   // ones
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tmem_alloc(tmem_slot, 512);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------ producer ------------------------------
        const uint64_t pol = p.M > WROWS ? policy_evict_last() : policy_evict_first();
        int s = 0, issued = 0;
        uint32_t ph = 0;
        for (int st = st0; st < st1; ++st, ++issued) {
            if (!mbar_wait(&in_empty[s], ph ^ 1u, abort_flag, p.status, 41)) break;
            if (elect_one()) {
                mbar_expect_tx(&in_full[s], (uint32_t)(WG * TX_BYTES));
#pragma unroll
                for (int q = 0; q < WG; ++q) {
                    const int g = group_of(q);
                    uint8_t* dst = sIn + (size_t)s * W_IN + q * STAGE_BYTES;
                    tma_load_2d(dst, &map_w, st * SK, g * GN, &in_full[s], pol);
                    bulk_load(dst + W_BYTES, p.rbytes + ((size_t)g * p.nst + st) * (RD * SK), RD * SK, &in_full[s]);
                    bulk_load(sSc + (size_t)s * W_SC + q * S_BYTES, p.scales + (size_t)g * p.K + st * SK, S_BYTES, &in_full[s]);
                }
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        // whatever happened to the other roles: no copy is in flight when this CTA's shared memory is used for other things
        for (int j = max(0, issued - p.stages); j < issued; ++j) {
            const long long t0 = clock64();
            while (!mbar_try_wait(&in_full[j % p.stages], (uint32_t)(j / p.stages) & 1u) && clock64() - t0 < 4000000ll) {}
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ----------------------------
        constexpr uint32_t idesc = (2u << 4) | ((uint32_t)(NC >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        int s = 0, ab = 0;
        uint32_t ph = 0, aph = 0;
        for (int st = st0; st < st1; ++st) {
            if (!mbar_wait(&in_full[s], ph, abort_flag, p.status, 42) || !mbar_wait(&a_full[ab], aph, abort_flag, p.status, 43)) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int q = 0; q < WG; ++q) {
                    const uint64_t db = make_smem_desc(smem_u32(sIn + (size_t)s * W_IN + q * STAGE_BYTES));
#pragma unroll
                    for (int rb = 0; rb < 2; ++rb) {
                        const uint64_t da = make_smem_desc(smem_u32(sA + (size_t)(ab * WG + q) * W_ABUF + (size_t)rb * 16384));
#pragma unroll
                        for (int k4 = 0; k4 < SK / 32; ++k4)
                            umma_i8(tmem_base + (uint32_t)((q * 2 + rb) * NC), da + (uint64_t)(2 * k4), db + (uint64_t)(2 * k4), idesc, (st > st0 || k4 > 0) ? 1u : 0u);
                    }
                }
                umma_commit(&a_empty[ab]);
                umma_commit(&in_empty[s]);
                if (st == st1 - 1) umma_commit(d_full);
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; ph ^= 1u; }
            ab ^= 1;
            if (ab == 0) aph ^= 1u;
        }
    } else {
        // ------------------------------ converters ----------------------------
        const int cw = warp - 2, ct = threadIdx.x - 64;
        for (int i = ct; i < WG * p.nst; i += 32 * WCW) s_smax[i] = __ldg(p.smax + (size_t)group_of(i / p.nst) * p.nst + i % p.nst);   // the weight's own: before the wait
        pdl_wait();   // x and xtop come from the previous kernel
        asm volatile("bar.sync 1, %0;" ::"n"(32 * WCW) : "memory");
        const int nr = cw < rows ? (rows - cw + WCW - 1) / WCW : 0;     // rows of this warp: cw, cw + 16, ...
        // The largest product of every row and group, as in the kernel above: the places of the stages' largest |x| first, all
        // products of a stage where the bound of the others has a larger exponent.
        const uint2* xt = p.xtop + (size_t)(m0 + cw) * p.nst;
        const float* xr = reinterpret_cast<const float*>(p.x) + (size_t)(m0 + cw) * SK + lane * 4;
        const float* gs[WG] = {p.scales + (size_t)group_of(0) * p.K, p.scales + (size_t)group_of(1) * p.K};
        auto rest_bound = [&](uint2 v, int q, int st) { return abs_bits(__fmul_rn(__uint_as_float(v.y & 0xffff0000u), s_smax[q * p.nst + st])); };
        float scale[WG][WR];
        {
            uint32_t top[WG][WR], rest[WG][WR];
#pragma unroll
            for (int i = 0; i < WR; ++i) top[0][i] = top[1][i] = rest[0][i] = rest[1][i] = 0u;
            for (int st = lane; st < p.nst; st += 32) {
                uint2 v[WR];
                float s1[WG][WR];
#pragma unroll
                for (int i = 0; i < WR; ++i)
                    if (i < nr) v[i] = xt[(size_t)(WCW * i) * p.nst + st];
#pragma unroll
                for (int i = 0; i < WR; ++i)
                    if (i < nr)
#pragma unroll
                        for (int q = 0; q < WG; ++q) s1[q][i] = __ldg(gs[q] + st * SK + (v[i].y & 0xffffu));
#pragma unroll
                for (int i = 0; i < WR; ++i)
                    if (i < nr)
#pragma unroll
                        for (int q = 0; q < WG; ++q) {
                            top[q][i] = max(top[q][i], abs_bits(__fmul_rn(__uint_as_float(v[i].x), s1[q][i])));
                            rest[q][i] = max(rest[q][i], rest_bound(v[i], q, st));
                        }
            }
#pragma unroll
            for (int q = 0; q < WG; ++q)
#pragma unroll
                for (int i = 0; i < WR; ++i) {
                    scale[q][i] = 0.0f;
                    if (i >= nr) continue;
                    uint32_t t = __reduce_max_sync(0xffffffffu, top[q][i]);
                    if (__any_sync(0xffffffffu, rest[q][i] >> 23 > t >> 23)) {
#pragma unroll 1
                        for (int base = 0; base < p.nst; base += 32) {
                            const int st = base + lane;
                            const uint32_t b = st < p.nst ? rest_bound(xt[(size_t)(WCW * i) * p.nst + st], q, st) >> 23 : 0u;
                            uint32_t todo = __ballot_sync(0xffffffffu, b > t >> 23);
                            while (todo) {
                                const int sa = base + __ffs(todo) - 1;
                                todo &= todo - 1;
                                t = max(t, __reduce_max_sync(0xffffffffu, __float_as_uint(top_of(0.0f, ld_x4(xr + (size_t)sa * p.xstep + i * (WCW * SK)), ldg_x4(gs[q] + sa * SK + lane * 4)))));
                                todo &= __ballot_sync(0xffffffffu, b > t >> 23);
                            }
                        }
                    }
                    const bool finite = t < 0x7f800000u;
                    const int e = unit_exponent(t);
                    scale[q][i] = finite ? __uint_as_float((uint32_t)(127 + e) << 23) : 0.0f;   // 2^e, a normal number
                    if (lane == 0) s_exp[q * WROWS + cw + WCW * i] = finite ? e : INT_MIN;
                }
        }
        if (nr > 0) {
            // where this lane's four bytes of plane pl go: row 4m + pl of the tile, 16-byte chunk lane / 4 under the 128-byte swizzle;
            // m's parity is the first row's
            uint32_t off[4];
#pragma unroll
            for (int pl = 0; pl < 4; ++pl)
                off[pl] = smem_u32(sA) + (uint32_t)(cw * 512 + pl * 128 + ((((lane >> 2) ^ pl) << 4) ^ ((cw & 1) << 6)) + (lane & 3) * 4);
            const uint32_t sv0 = smem_u32(sSc) + lane * 16;
            const float* xw = xr + (size_t)st0 * p.xstep;
            int slot = 0, ab = 0;
            uint32_t ph = 0, aph = 0;
            auto fetch = [&](float4 (&v)[WR], int st) {
                if (st < st1)
#pragma unroll
                    for (int i = 0; i < WR; ++i) v[i] = ld_x4(xw + i * (WCW * SK));     // (the copy has rows enough for the whole tile)
                xw += p.xstep;
            };
            auto convert = [&](const float4 (&v)[WR]) {
                if (!mbar_wait(&in_full[slot], ph, abort_flag, p.status, 44)) return false;
                uint4 sq[WG];
#pragma unroll
                for (int q = 0; q < WG; ++q) sq[q] = lds128(sv0 + (uint32_t)(slot * W_SC + q * S_BYTES));
                const uint32_t buf = (uint32_t)(ab * WG * W_ABUF);
                auto item = [&](const float4& x4, int q, int i) {
                    float a0, a1, a2, a3;
                    mul2(a0, a1, x4.x, x4.y, __uint_as_float(sq[q].x), __uint_as_float(sq[q].y));
                    mul2(a2, a3, x4.z, x4.w, __uint_as_float(sq[q].z), __uint_as_float(sq[q].w));
                    mul2(a0, a1, a0, a1, scale[q][i], scale[q][i]);
                    mul2(a2, a3, a2, a3, scale[q][i], scale[q][i]);
                    const int q0 = __float2int_rn(a0), q1 = __float2int_rn(a1), q2 = __float2int_rn(a2), q3 = __float2int_rn(a3);
                    // 4 integers x 4 bytes -> 4 planes x 4 k; plane 0 is the top byte, its sign bit flipped: q + 2^31
                    const uint32_t t0 = __byte_perm(q0, q1, 0x5140), t1 = __byte_perm(q2, q3, 0x5140);
                    const uint32_t t2 = __byte_perm(q0, q1, 0x7362), t3 = __byte_perm(q2, q3, 0x7362);
                    const uint32_t at = buf + (uint32_t)(q * W_ABUF + i * (WCW * 512));
                    sts32(off[0] + at, __byte_perm(t2, t3, 0x7632) ^ 0x80808080u);
                    sts32(off[1] + at, __byte_perm(t2, t3, 0x5410));
                    sts32(off[2] + at, __byte_perm(t0, t1, 0x7632));
                    sts32(off[3] + at, __byte_perm(t0, t1, 0x5410));
                };
                if (!mbar_wait(&a_empty[ab], aph ^ 1u, abort_flag, p.status, 45)) return false;
#pragma unroll
                for (int q = 0; q < WG; ++q)
#pragma unroll
                    for (int i = 0; i < WR; ++i) item(v[i], q, i);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[ab]);    // (group by group, four buffers: 512 rows 92 -> 97 us)
                if (++slot == p.stages) { slot = 0; ph ^= 1u; }
                ab ^= 1;
                if (ab == 0) aph ^= 1u;
                return true;
            };
            float4 xa[WR], xb[WR];
            fetch(xa, st0);
            for (int st = st0; st < st1; st += 2) {
                fetch(xb, st + 1);
                if (!convert(xa) || st + 1 >= st1) break;
                fetch(xa, st + 2);
                if (!convert(xb)) break;
            }
#pragma unroll 1
            for (int q = 0; q < WG; ++q) {
                if (__ldg(p.rinfo + 8 * group_of(q) + 4) != INT_MIN) continue;
                // a group without r: x . b in double, upper 24 bits and the rest of every four terms apart: exact sums
                const float* xb0 = reinterpret_cast<const float*>(p.x) + (size_t)(m0 + cw) * SK + lane * 4;
                const float* gb = p.biases + (size_t)group_of(q) * p.K + lane * 4;
                for (int i = 0; i < nr; ++i) {
                    double hi = 0.0, lo = 0.0;
                    for (int st = st0; st < st1; ++st) {
                        const float4 x4 = ld_x4(xb0 + (size_t)st * p.xstep + i * (WCW * SK)), b4 = ldg_x4(gb + st * SK);
                        const double d = fma((double)x4.x, (double)b4.x, fma((double)x4.y, (double)b4.y, fma((double)x4.z, (double)b4.z, (double)x4.w * (double)b4.w)));
                        const double u = __hiloint2double(__double2hiint(d), __double2loint(d) & (int)0xe0000000);
                        hi += u;
                        lo += d - u;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        hi += __shfl_xor_sync(0xffffffffu, hi, o);
                        lo += __shfl_xor_sync(0xffffffffu, lo, o);
                    }
                    if (lane == 0) s_bias[q * WROWS + cw + WCW * i] = make_double2(hi, lo);
                }
            }
        }
        if (st1 > st0) mbar_wait(d_full, 0, abort_flag, p.status, 46);
    }
    // bytes -> int64 sums per output, exact, parked where A and the ring were; then each CTA of the cluster adds up and writes its
    // share of the rows (a wait that gave up leaves the loops above in every role; the barriers below are reached all the same)
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    long long* s_sum = reinterpret_cast<long long*>(smem + W_SUM_AT);  // [WG][64][GN]
    long long* s_ext = s_sum + WG * WROWS * GN;                        // [WG][64][RD + 1]: the bias columns
    const bool failed = *abort_flag != 0;
    if (warp >= 2 && !failed) {
        const int cw = warp - 2, quarter = warp & 3, half = (cw >> 2) & 1, q = cw >> 3;   // lanes of tensor memory, columns, group
        uint32_t* mine = reinterpret_cast<uint32_t*>(smem) + (size_t)cw * 32 * W_LDW;
#pragma unroll 1
        for (int rb = 0; rb < 2; ++rb) {
            const int row0 = rb * 32 + quarter * 8;
            if (row0 >= rows) continue;
            const uint32_t from = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((q * 2 + rb) * NC);
            uint32_t v[2][16], ext[16];
#pragma unroll
            for (int c = 0; c < 2; ++c) tmem_ld16(from + half * 32 + c * 16, v[c]);
            tmem_ld16(from + GN, ext);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int e = 0; e < 16; ++e) mine[lane * W_LDW + c * 16 + e] = v[c][e];
            __syncwarp();
            auto sum_at = [&](int m, int c) {
                const uint32_t* w = mine + (4 * m) * W_LDW + c;
                return ((((long long)w[0] * 256 + w[W_LDW]) * 256 + w[2 * W_LDW]) * 256) + w[3 * W_LDW];
            };
#pragma unroll
            for (int m = 0; m < 8; ++m) s_sum[(size_t)(q * WROWS + row0 + m) * GN + half * 32 + lane] = sum_at(m, lane);
            __syncwarp();
            if (half == 1) {
#pragma unroll
                for (int e = 0; e <= RD; ++e) mine[lane * W_LDW + e] = ext[e];
                __syncwarp();
                for (int i = lane; i < 8 * (RD + 1); i += 32) s_ext[(size_t)(q * WROWS + row0) * (RD + 1) + i] = sum_at(i / (RD + 1), i % (RD + 1));
            }
            __syncwarp();
        }
        tc_fence_before();
    }
    cg::cluster_group cl = cg::this_cluster();
    if (p.ways > 1) cl.sync();
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
    if (warp >= 2 && !failed) {
        const int t = threadIdx.x - 64, n = t & (GN - 1), q = (t >> 6) & 1;      // 512 threads: both groups' 64 columns, every fourth row
        const int g = (int)blockIdx.y * WG + q;
        double2* s_terms = reinterpret_cast<double2*>(smem);           // [WG][64], where the corners were
        double* s_plus = reinterpret_cast<double*>(s_terms + WG * WROWS);
        if (t < WG * WROWS && (t & (WROWS - 1)) < rows) {
            const int tg = group_of(t / WROWS), runit = __ldg(p.rinfo + 8 * tg + 4);
            const int4 rsum = __ldg(reinterpret_cast<const int4*>(p.rinfo) + 2 * tg);
            long long ext[RD + 1] = {0, 0, 0, 0, 0};
            double bhi = 0.0, blo = 0.0;
            for (int w = 0; w < p.ways; ++w) {
                const long long* se = (p.ways > 1 ? cl.map_shared_rank(s_ext, w) : s_ext) + (size_t)t * (RD + 1);
#pragma unroll
                for (int i = 0; i <= RD; ++i) ext[i] += se[i];
                if (runit == INT_MIN) {
                    const double2 b = (p.ways > 1 ? cl.map_shared_rank(s_bias, w) : s_bias)[t];
                    bhi += b.x;
                    blo += b.y;
                }
            }
            s_terms[t] = row_terms(ext, rsum, runit, s_exp[t], p.K);
            s_plus[t] = bhi + blo;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * WCW) : "memory");
        if (g < groups) {
            const long long rs = (long long)__ldg(p.rowsum + g * GN + n) << 31;
            // four rows at a time: one by one the way from a sum to its f32 is a chain of 300 cycles
            for (int j0 = (t >> 7) + 4 * way; j0 < rows; j0 += 16 * p.ways) {
                long long sum[4] = {0, 0, 0, 0};
                for (int w = 0; w < p.ways; ++w) {
                    const long long* from = (p.ways > 1 ? cl.map_shared_rank(s_sum, w) : s_sum) + (size_t)(q * WROWS) * GN + n;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j0 + u * 4 * p.ways < rows) sum[u] += from[(size_t)(j0 + u * 4 * p.ways) * GN];
                }
                float f[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int at_row = q * WROWS + min(j0 + u * 4 * p.ways, rows - 1);
                    f[u] = __double2float_rn(((double)(sum[u] - rs) + s_terms[at_row].x) * s_terms[at_row].y + s_plus[at_row]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j0 + u * 4 * p.ways < rows) store_output(p, f[u], (size_t)(m0 + j0 + u * 4 * p.ways) * p.ldy + p.y_col0 + g * GN + n);
            }
        }
    }
    if (p.ways > 1) cl.sync();   // the others have read this CTA's sums
}

// For batches of more than 8 rows, once instead of in every CTA: xtop[m][st] = (largest |x| of 128 k; the next largest, rounded
// up to 16 bits, above the place of the largest), as bits: a NaN is above every number; and x as f32 in the order the
// converters read it, [K/128][Mp][128]: a warp's rows of a stage then lie at constant offsets, and rows M .. Mp and k beyond K
// (zeros) need no checks.  A block takes 1024 k of a row.  K % 4 == 0.
template <typename XT>
__global__ void __launch_bounds__(256) gc_prepare_kernel(const XT* x, float* xs, uint2* xtop, int M, int Mp,
                                                         int K) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, m = blockIdx.x;
    const XT* row = x + (size_t)m * K;
    const int Kp = (K + SK - 1) / SK * SK;
    const int k = (blockIdx.y * 256 + threadIdx.x) * 4;
    if (k < Kp) {                                        // (a warp is inside or outside)
        const float4 v = m < M && k < K ? ld_x4<XT>(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(xs + ((size_t)(k / SK) * Mp + m) * SK + (k & (SK - 1))) = v;
        const uint32_t c[4] = {abs_bits(v.x), abs_bits(v.y), abs_bits(v.z), abs_bits(v.w)};
        uint32_t best = c[0], next = 0u, at = 0u;
#pragma unroll
        for (uint32_t i = 1; i < 4; ++i) {
            const bool more = c[i] > best;
            next = max(next, more ? best : c[i]);
            if (more) best = c[i], at = i;
        }
        const uint32_t top = __reduce_max_sync(0xffffffffu, best);
        const int who = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
        next = __reduce_max_sync(0xffffffffu, lane == who ? next : best);
        next = min((next >> 16) + ((next & 0xffffu) != 0u), 0x7fffu);
        if (lane == who && m < M) xtop[(size_t)m * (Kp / SK) + k / SK] = make_uint2(top, next << 16 | (lane * 4 + at));
    }
}

// The weight's own tables, once at create: largest |scale| of every 128 k of a group (a NaN or infinite scale shows as such),
// and the byte sum of every row.
__global__ void __launch_bounds__(256) gc_smax_kernel(const float* __restrict__ s, float* __restrict__ smax, size_t entries) {
    for (size_t c = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); c < entries; c += (size_t)gridDim.x * 8) {
        const int lane = threadIdx.x & 31;
        const uint32_t b = __reduce_max_sync(0xffffffffu, abs_max(ldg_x4(s + c * SK + lane * 4)));
        if (lane == 0) smax[c] = __uint_as_float(b);
    }
}
__global__ void __launch_bounds__(256) gc_rowsum_kernel(const uint8_t* __restrict__ w, int* __restrict__ rowsum, int N, int K) {
    const int n = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (n >= N) return;
    const uint4* p = reinterpret_cast<const uint4*>(w + (size_t)n * K);
    unsigned sum = 0;
    for (int i = lane; i < K / 16; i += 32) {
        const uint4 v = __ldg(p + i);
        sum = __dp4a(v.x, 0x01010101u, sum);
        sum = __dp4a(v.y, 0x01010101u, sum);
        sum = __dp4a(v.z, 0x01010101u, sum);
        sum = __dp4a(v.w, 0x01010101u, sum);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) rowsum[n] = (int)sum;
}

// r = b / s of a group (one block each) as 32-bit integers below its largest |r|: four rows of bytes, offset 2^31, top byte first, in
// the order of the 128-byte swizzle (16-byte chunk c of row i at c ^ i).
__global__ void __launch_bounds__(256) gc_ratio_kernel(const float* __restrict__ scales, const float* __restrict__ biases, uint8_t* __restrict__ rows,
                                                       int* __restrict__ info, int K) {
    __shared__ double s_max[8];
    __shared__ int s_sum[RD];
    const int g = blockIdx.x, lane = threadIdx.x & 31;
    const float *s = scales + (size_t)g * K, *b = biases + (size_t)g * K;
    auto ratio = [&](int k) { return b[k] == 0.0f ? 0.0 : (double)b[k] / (double)s[k]; };
    double most = 0.0;
    for (int k = threadIdx.x; k < K; k += 256) {
        const double r = fabs(ratio(k));
        most = r <= (double)R_MAX ? fmax(most, r) : 2.0 * R_MAX;   // (a NaN lands there as well)
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = fmax(most, __shfl_xor_sync(0xffffffffu, most, o));
    if (lane == 0) s_max[threadIdx.x >> 5] = most;
    if (threadIdx.x < RD) s_sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) most = fmax(most, s_max[w]);
    const bool fits = most <= (double)R_MAX;
    const int unit = fits ? (most > 0x1p-30 ? 30 - ilogb(most) : 60) : INT_MIN;
    int sum[RD] = {0, 0, 0, 0};
    for (int k = threadIdx.x; k < K; k += 256) {
        const long long q = fits ? llrint(ldexp(ratio(k), unit)) : 0;
        const uint32_t v = (uint32_t)((q > 0x7fffffffll ? 0x7fffffffll : q < -0x80000000ll ? -0x80000000ll : q) + 0x80000000ll);
#pragma unroll
        for (int i = 0; i < RD; ++i) {
            const uint32_t byte = v >> (24 - 8 * i) & 255u;
            rows[((size_t)g * (K / SK) + k / SK) * (RD * SK) + i * SK + ((k % SK) ^ (i << 4))] = (uint8_t)byte;
            sum[i] += (int)byte;
        }
    }
#pragma unroll
    for (int i = 0; i < RD; ++i) {
        sum[i] = __reduce_add_sync(0xffffffffu, sum[i]);
        if (lane == 0) atomicAdd(&s_sum[i], sum[i]);
    }
    __syncthreads();
    if (threadIdx.x < 8) info[8 * g + threadIdx.x] = threadIdx.x < RD ? s_sum[threadIdx.x] : threadIdx.x == 4 ? unit : 0;
}

template <typename XT, int RPW, bool MEET = false>
cudaError_t launch_gc(rusty_cuda_ctx* ctx, const CUtensorMap& map_w, const GcParams& p, dim3 grid, size_t smem) {
    auto kern = qlinear_gc_tc_kernel<XT, RPW, MEET>;
    cudaError_t e = rusty::ensure_dynamic_smem((const void*)kern, ctx->device, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl_cluster(kern, grid, dim3(GC_THREADS), (unsigned)p.ways, smem, ctx->stream, map_w, p);
}
}  // namespace

namespace rusty {

bool gc_tc_supported(const rusty_cuda_ctx* ctx, uint32_t N, uint32_t K) {
    return ctx->tc_ws && encode_tiled_fn() && K % 4 == 0 && K <= 32768u && N % GN == 0 && N / GN <= 65535u;
}
uint32_t gc_padded(uint32_t K) { return (K + SK - 1) / SK * SK; }
// r's rows (they start on 512 bytes) | r's sums and units | largest scales | byte sums
static size_t gc_r_bytes(uint32_t N, uint32_t Kp) { return (size_t)(N / GN) * RD * Kp; }
size_t gc_tables_bytes(uint32_t N, uint32_t K) {
    const uint32_t Kp = gc_padded(K);
    return gc_r_bytes(N, Kp) + (size_t)(N / GN) * (8 + Kp / SK) * 4 + (size_t)N * 4;
}
int launch_gc_tables(rusty_cuda_ctx* ctx, const uint8_t* w, const float* scales, const float* biases, void* tables, uint32_t N, uint32_t K) {
    K = gc_padded(K);
    const size_t entries = (size_t)(N / GN) * (K / SK);
    int* info = (int*)((char*)tables + gc_r_bytes(N, K));
    float* smax = (float*)(info + (size_t)(N / GN) * 8);
    const size_t blocks = (entries + 7) / 8, cap = (size_t)ctx->sm_count * 8;
    gc_ratio_kernel<<<N / GN, 256, 0, ctx->stream>>>(scales, biases, (uint8_t*)tables, info, (int)K);
    int rc = after_launch(ctx, "gc_ratio");
    if (rc) return rc;
    gc_smax_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, ctx->stream>>>(scales, smax, entries);
    rc = after_launch(ctx, "gc_smax");
    if (rc) return rc;
    gc_rowsum_kernel<<<(N + 7) / 8, 256, 0, ctx->stream>>>(w, (int*)(smax + entries), (int)N, (int)K);
    return after_launch(ctx, "gc_rowsum");
}

int launch_gc_tc(rusty_cuda_ctx* ctx, const QLinearArgs& a) {
    GcParams p{};
    p.scales = a.scales;
    p.biases = a.biases;
    p.N = (int)a.N;
    p.K = (int)gc_padded(a.K);   // the weight's rows, scales and biases are that long, zeros behind a.K
    p.rbytes = (const uint8_t*)a.gc_tables;
    p.rinfo = (const int*)((const char*)a.gc_tables + gc_r_bytes(a.N, (uint32_t)p.K));
    p.smax = (const float*)(p.rinfo + (size_t)(p.N / GN) * 8);
    p.rowsum = (const int*)(p.smax + (size_t)(p.N / GN) * (p.K / SK));
    p.nst = p.K / SK;
    p.ldy = (int)a.ldy;
    p.y_col0 = (int)a.y_col0;
    p.y_bf16 = a.y_dtype == RUSTY_CUDA_BF16;
    p.status = ctx->status_dev;
    if (a.push && a.push->nranks > 1)
        for (int r = 0; r < a.push->nranks && r < PEER_MAX_RANKS; ++r)
            if (r != a.push->rank) p.peer_delta[p.n_peers++] = a.push->delta[r];
    CUtensorMap map_w;
    if (!make_map_u8(&map_w, a.w, a.N, (uint32_t)p.K, GN)) return fail(ctx, RUSTY_CUDA_ERR_KERNEL_EXECUTION, "gc_tc: cuTensorMapEncodeTiled failed");
    const bool xb = a.x_dtype == RUSTY_CUDA_BF16;
    const size_t xs = xb ? 2 : 4, ys = p.y_bf16 ? 2 : 4;
    // the digit region of the workspace: x rearranged (Mp rows), then its largest values
    const size_t row_bytes = (size_t)p.K * 4 + (size_t)p.nst * 8;
    const uint32_t per_pass = (uint32_t)(tc_workspace_xq_bytes() / row_bytes) & ~63u;
    for (uint32_t m0 = 0; m0 < a.M; m0 += per_pass) {
        p.M = (int)(a.M - m0 < per_pass ? a.M - m0 : per_pass);
        p.x = (const char*)a.x + (size_t)m0 * a.K * xs;
        p.y = (char*)a.y + (size_t)m0 * a.ldy * ys;
        p.residual = a.residual ? (const char*)a.residual + (size_t)m0 * a.ldy * ys : nullptr;
        // K ranges: as many CTAs as the SMs hold (two an SM; the wide kernel one), four stages each at least.  More than two tiles of
        // rows (wide: one): none, the CTAs suffice, and the start and the end of a CTA cost as much as ten stages.
        const int groups = p.N / GN;
        auto ways_of = [&](int ctas, int slots, bool cut) {
            int w = 1;
            while (cut && w < 4 && ctas * w * 2 <= slots && p.nst / (w * 2) >= 4) w *= 2;
            return w;
        };
        // Beyond 32 rows: tiles of 32 on the narrow kernel or of 64 x two groups on the wide one, which does four times the work of a
        // CTA in 41 us where 2 an SM of the others take 27 (32 stages), but starts and ends in 14 instead of 8 us and fills whole
        // waves less well.  us, narrow / wide: 64 x 4096 x 4096 23.3 / 25.3, 64 x 4096 x 1024 13.1 / 23.7, 64 x 4096 x 11008 55.3 / 47.2, 96 x
        // 4096 x 4096 33.2 / 44.9, 200 x 4096 x 4096 62.9 / 47.7, 512 x 4096 x 4096 118 / 91.4, 512 x 4096 x 11008 295 / 224.
        bool wide = false;
        if (p.M > 32) {
            const int tn = (p.M + 31) / 32, tw = (p.M + WROWS - 1) / WROWS, un = groups * tn, uw = (groups + WG - 1) / WG * tw;
            const int wn = ways_of(un, 2 * ctx->sm_count, tn <= 2), ww = ways_of(uw, ctx->sm_count, tw == 1);
            auto us = [&](int ctas, int slots, int ways, double us32, double fixed) {
                return (double)((ctas * ways + slots - 1) / slots) * us32 * p.nst / 32.0 / ways + fixed;
            };
            wide = us(uw, ctx->sm_count, ww, 41.0, 6.0 + (p.M < WROWS ? p.M : WROWS) / 8) < us(un, 2 * ctx->sm_count, wn, 27.0, 8.0);
        }
        // rows per converter warp; up to 8 rows the converters read x as it is and find its maxima themselves (16 KB a row from
        // L2 at K = 4096, while the first weights arrive) if x has no partial stage: the copy pads it
        const int rpw = p.M <= 8 && p.K == (int)a.K ? 1 : p.M <= 16 ? 2 : 4;
        const int tile = wide ? WROWS : 8 * rpw, tiles = (p.M + tile - 1) / tile;
        const int units = wide ? (groups + WG - 1) / WG : groups;
        p.ways = ways_of(units * tiles, (wide ? 1 : 2) * ctx->sm_count, tiles <= (wide ? 1 : 2));
        p.xstep = SK;
        p.xtop = nullptr;
        if (wide || rpw > 1) {
            const int Mp = tiles * tile;
            float* xbuf = (float*)ctx->tc_ws;
            uint2* xtop = (uint2*)(xbuf + (size_t)Mp * p.K);
            const dim3 pg((unsigned)Mp, (unsigned)(p.K + 1023) / 1024);
            cudaError_t e = xb ? launch_pdl(gc_prepare_kernel<__nv_bfloat16>, pg, dim3(256), 0, ctx->stream, (const __nv_bfloat16*)p.x, xbuf, xtop, p.M, Mp, (int)a.K)
                               : launch_pdl(gc_prepare_kernel<float>, pg, dim3(256), 0, ctx->stream, (const float*)p.x, xbuf, xtop, p.M, Mp, (int)a.K);
            if (e != cudaSuccess) return check_cuda(ctx, e, "gc_prepare");
            int rc = after_launch(ctx, "gc_prepare");
            if (rc) return rc;
            p.x = xbuf;
            p.xtop = xtop;
            p.xstep = (size_t)Mp * SK;
        }
        // Meeting costs 1 to 2 us, walking x and the scales beyond what the registers hold more than that with rows x stages.  One
        // CTA alone / together, us: 4096 x 4096 at one / eight rows 8.2 / 10.0 and 12.8 / 13.4; 5120 x 4096 at three / four / six
        // 12.0 / 12.6, 13.1 / 13.2, 15.0 / 14.0; 8192 x 4096 at two / four 13.2 / 13.9, 15.5 / 15.0; 11008 x 4096 at one / two /
        // eight 15.4 / 15.8, 16.6 / 16.5, 24.9 / 19.6; 14336 x 3008 at one / eight 16.5 / 16.0, 28.3 / 20.3.
        const bool meet = rpw == 1 && p.ways > 1 && p.nst > 32 && (p.M * p.nst >= 160 || p.nst > 96);
        const size_t stage_bytes = wide ? W_IN + W_SC : STAGE_BYTES + S_BYTES;
        const size_t fixed = wide ? 1024 + (size_t)2 * WG * W_ABUF + (2 * MAX_STAGES + 6) * 8 + (size_t)WG * WROWS * 20 + (size_t)WG * p.nst * 4 + 64
                                  : 1024 + (size_t)A_BYTES + (4 * MAX_STAGES + 2) * 8 + (size_t)32 * 24 + (size_t)p.nst * 4 + 64;
        const size_t budget = wide ? ctx->smem_optin : (ctx->smem_optin + 1024) / 2 - 1024;   // an SM, or half of it less the 1 KiB every block pays
        int stages = budget > fixed ? (int)((budget - fixed) / stage_bytes) : 0;
        if (stages > MAX_STAGES) stages = MAX_STAGES;
        if (stages < (wide ? 3 : MAX_STAGES)) return fail(ctx, RUSTY_CUDA_ERR_UNSUPPORTED, "gc_tc: the ring does not fit shared memory");
        p.stages = stages;
        const size_t smem = fixed + (size_t)stages * stage_bytes;
        const dim3 grid((unsigned)(tiles * p.ways), (unsigned)units);
        cudaError_t e;
        if (wide) {
            e = rusty::ensure_dynamic_smem((const void*)qlinear_gc_wide_kernel, ctx->device, smem);
            if (e == cudaSuccess) e = launch_pdl_cluster(qlinear_gc_wide_kernel, grid, dim3(W_THREADS), (unsigned)p.ways, smem, ctx->stream, map_w, p);
        } else {
            e = rpw == 4   ? launch_gc<float, 4>(ctx, map_w, p, grid, smem)
                : rpw == 2 ? launch_gc<float, 2>(ctx, map_w, p, grid, smem)
                : xb       ? (meet ? launch_gc<__nv_bfloat16, 1, true>(ctx, map_w, p, grid, smem) : launch_gc<__nv_bfloat16, 1>(ctx, map_w, p, grid, smem))
                : meet     ? launch_gc<float, 1, true>(ctx, map_w, p, grid, smem)
                           : launch_gc<float, 1>(ctx, map_w, p, grid, smem);
        }
        if (e != cudaSuccess) return check_cuda(ctx, e, "qlinear_gc_tc");
        int rc = after_launch(ctx, "qlinear_gc_tc");
        if (rc) return rc;
    }
    return RUSTY_CUDA_OK;
}

}  // namespace rusty
