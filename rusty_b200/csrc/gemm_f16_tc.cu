// Prefill GEMM over int8 weights on tcgen05 / TMEM with bf16 operands.
//
// Replaces, for many activation rows at once, the reference's "dequantise once
// at load, f32 tiled matmul per forward" (rusty-loader/src/lib.rs:155-218,
// rusty-backend/src/kernels.wgsl:16-54, :234-242):
//     y[m,n] = scale[n] * sum_k x[m,k] * q[n,k]        x bf16, q int8, fp32 accumulation
//
// The weight rows are the M side of the MMA (128 rows per tile), the activation
// rows the N side (up to 256 per tile), so the accumulator tile is y^T.
//   * int8 weight tiles (128 rows x 128 k, 16 KB) arrive by TMA with the 128-byte
//     swizzle; eight converter warps (two threads per weight row) read their row
//     conflict-free, turn bytes into bf16 pairs (byte-permute into the mantissa of
//     2^23, subtract, packed convert: exact since |q| <= 128), and write them
//     straight into TENSOR MEMORY with tcgen05.st — the A operand never goes back
//     through shared memory;
//   * bf16 activation tiles (up to 256 rows x 64 k) arrive by TMA as the B operand;
//   * one elected thread issues tcgen05.mma kind::f16 (A bf16 from TMEM, B bf16
//     from shared memory, fp32 accumulators in TMEM); bf16 x bf16 products are
//     exact in the fp32 accumulate, so the only rounding is the summation;
//   * eight epilogue warps read the accumulators, apply the per-row weight scale and
//     store y (bf16 or f32) while the converters already work on the next tile;
//   * tiles beyond whole waves are cut along K: the pieces meet in f32 slots (digit
//     region of the workspace, which this path has no digits for), summed in piece order.
// Persistent CTAs, one per SM; every mbarrier wait is bounded.
#include <cstdlib>
#include <cstring>

#include "tc_common.cuh"

using namespace rusty_tc;

namespace {

constexpr int BM = 128;          // weight rows per tile (UMMA M)
constexpr int WK = 128;          // k per weight stage (bytes per row)
constexpr int XK = 64;           // k per activation stage (128 bytes of bf16 per row)
constexpr int A_BUFS = 3;        // converted-weight buffers in tensor memory, 64 columns each
constexpr int A_COLS = WK / 2;   // two 16-bit values per 32-bit column
constexpr int D_COLS = 256;      // accumulator columns reserved
constexpr int CONV_WARPS = 8;     // two per TMEM lane quarter, each takes half of a stage's k range
constexpr int EPI_WARPS = 8;      // two per TMEM lane quarter, each drains half of the accumulator's columns: the
                                  // accumulator is single-buffered, so the drain holds up the next tile's first MMA
constexpr int W_WARP = 2 + CONV_WARPS + EPI_WARPS;        // the weights' producer
constexpr int F16_THREADS = 32 * (W_WARP + 1);            // activation producer, MMA, converter, epilogue and weight producer warps
constexpr int W_STAGE_BYTES = BM * WK;

struct F16Params {
    const float* scales;  // SYM_ROW: [N], applied to the sums; AFFINE_G64: [N*K/64], applied to the weights as they are converted
    const float* biases;  // AFFINE_G64: [N*K/64]; null selects SYM_ROW
    void* y;
    int Mx, N, K;
    int BN;               // activation rows per tile (multiple of 16, <= 256)
    int tiles_w, tiles_n, nws;  // weight-row tiles, activation-row tiles, weight stages per tile
    int x_stages, w_stages;     // ring depths: activation stages (64 k), weight stages (128 k)
    // Schedule: units = tiles_w * tiles_n tiles of the output.  The last `sk_units` of them are cut along K, the other units are
    // taken whole, unit = cta, cta + grid, ...  sk_ways > 0: every cut unit has that many equal pieces, one per CTA; else the
    // units' sk_units*nws weight stages form one linear space dealt out in contiguous runs of `sk_per_cta` (at most a unit
    // long) to the first `sk_ctas` CTAs, so that a CTA holds pieces of at most two cut units.
    int dp_units, sk_units, sk_per_cta, sk_ctas, sk_ways;
    float* slots;             // [2 * cta + (0: the run starts in this unit, 1: it goes on into it)][BN/4][128] x float4
    unsigned int* counters;   // [sk_units] pieces stored, then [sk_units] pieces done with (zero between uses)
    int ldy, y_col0;
    int vec;                  // the outputs (and the residual) can be accessed 16 bytes at a time, and there are no peers
    int act;                  // RUSTY_CUDA_ACT_*: the pair epilogue writes N/2 columns
    const void* residual;     // null, or added to every output (same layout as y)
    PeerPush push;            // nranks > 1: every output is also stored into the other ranks' arenas (peer.cu)
    uint32_t idesc;
    rusty_cuda_dev_status* status;
};

template <typename T>
__device__ __forceinline__ void store_y(T* p, float v);
template <>
__device__ __forceinline__ void store_y<float>(float* p, float v) { *p = v; }
template <>
__device__ __forceinline__ void store_y<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

template <typename T>
__device__ __forceinline__ float load_y(const T* p);
template <>
__device__ __forceinline__ float load_y<float>(const float* p) { return *p; }
template <>
__device__ __forceinline__ float load_y<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// One output of activation row m and weight row n (this lane's), already scaled.  Every lane of the warp calls this
// together.  With the pair activation rows 2j / 2j+1 of the weight are gate_j / up_j (MLP::forward,
// rusty-graph/src/lib.rs:317-323): the even lane takes its neighbour's value and writes silu(gate) * up into column
// (y_col0 + n) / 2; silu as kernels.wgsl:104-113.
// The same element of every other rank's y, over NVLink (plain stores to peer addresses; the byte offsets of the other
// arenas sit in shared memory: indexing the kernel parameter with a run-time index would copy it to local memory).
struct PeerOut {
    int n;
    const long long* delta;
};
template <typename YT>
__device__ __forceinline__ void store_everywhere(YT* dst, float v, const PeerOut& po) {
    store_y<YT>(dst, v);
    for (int g = 0; g < po.n; ++g) store_y<YT>(reinterpret_cast<YT*>(reinterpret_cast<char*>(dst) + po.delta[g]), v);
}

template <typename YT>
__device__ __forceinline__ void store_out(const F16Params& p, YT* y, int m, int n, float v, bool row_ok, const PeerOut& po, float loaded, bool have = false) {
    if (p.act) {
        const float up = __shfl_down_sync(0xffffffffu, v, 1);
        v = __fdividef(v, 1.0f + __expf(-v)) * up;
        if (row_ok && m < p.Mx && !(n & 1)) store_everywhere<YT>(y + (size_t)m * p.ldy + ((p.y_col0 + n) >> 1), v, po);
    } else if (row_ok && m < p.Mx) {
        const size_t at = (size_t)m * p.ldy + p.y_col0 + n;
        if (p.residual) v += have ? loaded : load_y<YT>(reinterpret_cast<const YT*>(p.residual) + at);
        store_everywhere<YT>(y + at, v, po);
    }
}

// ---- vector epilogue --------------------------------------------------------
// A lane of the accumulator is a weight row, so a warp that stores its lanes' values one activation row at a time issues 2- and
// 4-byte accesses, and a residual is a trip to L2 per element: 4096 x 14336 at 2048 rows 190 us, with the residual 348.  Here
// eight activation rows of the warp's 32 columns are turned in shared memory, a lane then has eight neighbouring outputs of
// one row: one 16-byte access for each of residual and y (bf16), and silu(gate) * up without idle lanes.
constexpr int ST_PITCH = 36;                              // floats between rows of the staging tile: no bank conflicts
constexpr int ST_BYTES = EPI_WARPS * 8 * ST_PITCH * 4;    // 8 activation rows x 32 columns a warp
template <typename YT>
struct Octet {   // eight neighbouring elements
    uint4 q[sizeof(YT) / 2];
};
template <typename YT>
__device__ __forceinline__ void add_octet(float (&o)[8], const Octet<YT>& r) {
    if constexpr (sizeof(YT) == 2) {
        const uint32_t w[4] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o[2 * i] += __uint_as_float(w[i] << 16);
            o[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
        }
    } else {
        const uint32_t w[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += __uint_as_float(w[i]);
    }
}
template <typename YT, int COUNT>
__device__ __forceinline__ void store_run(YT* dst, const float (&o)[8]) {   // COUNT = 8, or 4 (pairs)
    if constexpr (sizeof(YT) == 2) {
        uint32_t w[COUNT / 2];
#pragma unroll
        for (int i = 0; i < COUNT / 2; ++i) {
            __nv_bfloat162 b = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&b);
        }
        if constexpr (COUNT == 8) *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        else *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int i = 0; i < COUNT; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
    }
}

// 16 int8 (one 128-bit word) -> 8 registers of packed bf16 pairs (low half = even k).
// A byte under the exponent of 128 (0x43) is two bf16 at once: its seven low bits make 128 + low, its sign bit 128 or 256, and the
// difference of the two is q, exactly (|q| <= 128 fits bf16's 8 significant bits): a permute, two masks and a subtraction for two
// weights.  (By way of f32, two permutes, two subtractions and a packing conversion: 300 x 14336 x 4096 43.8 us, so 40.7; 300 x 4096 x
// 6144 21.7 and 20.5; 2048 rows, under the power cap, 1 to 2 %.)
__device__ __forceinline__ void int8x16_to_bf16x2(const uint4& w, uint32_t* out) {
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t t = __byte_perm(words[i >> 1], 0x43434343u, i & 1 ? 0x4342 : 0x4140);
        const uint32_t low = t & 0xff7fff7fu, sign = t & 0xff80ff80u;
        const __nv_bfloat162 q = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&low), *reinterpret_cast<const __nv_bfloat162*>(&sign));
        out[i] = *reinterpret_cast<const uint32_t*>(&q);
    }
}

// The reference's affine layout (WGSL `affine_dequantize`, rusty-backend/src/kernels.wgsl:385-400): w = f32(u8) * scale +
// bias, one (scale, bias) per 64 consecutive elements.  The product is rounded to bf16 for the tensor core (2^-9
// relative per weight: inside the 1e-2 tolerance of the bf16 path, not the 1e-5 of the f32 paths).
// Two weights at a time: packed f32 additions and FMAs round each half like the single ones.
__device__ __forceinline__ uint32_t affine_pair(uint32_t word, uint32_t sel_lo, uint32_t sel_hi, float s0, float s1, float b0, float b1) {
    float f0 = __uint_as_float(__byte_perm(word, 0x4B000000u, sel_lo)), f1 = __uint_as_float(__byte_perm(word, 0x4B000000u, sel_hi));   // 2^23 + u
    asm("{\n\t.reg .b64 u, s, b, m;\n\tmov.b64 u, {%0, %1};\n\tmov.b64 s, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 m, {%6, %6};\n\t"
        "add.rn.f32x2 u, u, m;\n\tfma.rn.f32x2 u, u, s, b;\n\tmov.b64 {%0, %1}, u;\n\t}"
        : "+f"(f0), "+f"(f1)
        : "f"(s0), "f"(s1), "f"(b0), "f"(b1), "f"(-8388608.0f));
    const __nv_bfloat162 a = __floats2bfloat162_rn(f0, f1);
    return *reinterpret_cast<const uint32_t*>(&a);
}
__device__ __forceinline__ void u8x16_affine_to_bf16x2(const uint4& w, float sc, float bi, uint32_t* out) {
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        out[2 * i] = affine_pair(words[i], 0x7650, 0x7651, sc, sc, bi, bi);
        out[2 * i + 1] = affine_pair(words[i], 0x7652, 0x7653, sc, sc, bi, bi);
    }
}

// The same with one (scale, bias) per element: 16 consecutive k of one row whose scales and biases are 16 consecutive
// floats each (an [in,out] affine weight after its re-layout: groups run along the output dimension).
__device__ __forceinline__ void u8x16_affine_vec_to_bf16x2(const uint4& w, const float* sc, const float* bi, uint32_t* out) {
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 s4 = reinterpret_cast<const float4*>(sc)[i], b4 = reinterpret_cast<const float4*>(bi)[i];   // shared memory, broadcast
        out[2 * i] = affine_pair(words[i], 0x7650, 0x7651, s4.x, s4.y, b4.x, b4.y);
        out[2 * i + 1] = affine_pair(words[i], 0x7652, 0x7653, s4.z, s4.w, b4.z, b4.w);
    }
}

// One piece of work: weight stages [s0, s1) of output tile `u`.  nseg > 1: the tile is shared with the CTAs first ..
// first + nseg - 1, and lu is its number among the cut ones.
struct Piece {
    int u, s0, s1, nseg, lu, first;
};

// Every role of the CTA walks the same list of pieces: its share of the cut tiles first, whole tiles after it.
struct PieceSched {
    const F16Params& p;
    int g, g_end, dp_next;
    __device__ PieceSched(const F16Params& pp) : p(pp) {
        const int c = blockIdx.x;
        g = g_end = 0;
        if (c < p.sk_ctas) {
            if (p.sk_ways > 0) {
                const int lu = c / p.sk_ways, j = c - lu * p.sk_ways;
                g = lu * p.nws + j * p.nws / p.sk_ways;
                g_end = lu * p.nws + (j + 1) * p.nws / p.sk_ways;
            } else {
                g = c * p.sk_per_cta;
                g_end = min(p.sk_units * p.nws, g + p.sk_per_cta);
            }
        }
        dp_next = c;
    }
    __device__ bool next(Piece& q) {
        if (g < g_end) {
            q.lu = g / p.nws;
            q.u = p.dp_units + q.lu;
            q.s0 = g % p.nws;
            q.s1 = min(p.nws, q.s0 + (g_end - g));
            if (p.sk_ways > 0) {
                q.first = q.lu * p.sk_ways;
                q.nseg = p.sk_ways;
            } else {
                q.first = (q.lu * p.nws) / p.sk_per_cta;
                q.nseg = ((q.lu + 1) * p.nws - 1) / p.sk_per_cta - q.first + 1;
            }
            g += q.s1 - q.s0;
            return true;
        }
        if (dp_next < p.dp_units) {
            q.u = dp_next;
            q.lu = q.first = 0;
            q.s0 = 0;
            q.s1 = p.nws;
            q.nseg = 1;
            dp_next += gridDim.x;
            return true;
        }
        return false;
    }
};
// Where CTA c keeps its piece of cut unit lu.
__device__ __forceinline__ float4* piece_slot(const F16Params& p, int c, int lu) {
    const int tail = (p.sk_ways == 0 && c * p.sk_per_cta < lu * p.nws) ? 1 : 0;
    return reinterpret_cast<float4*>(p.slots) + (size_t)(2 * c + tail) * (p.BN / 4) * BM;
}

// QM: 0 = one scale per output row (applied to the sums); 1 = AFFINE_G64 with groups along K ([N][K/64] scales and biases);
// 2 = AFFINE_G64 of an [in,out] weight after its re-layout: one (scale, bias) per 64 consecutive OUTPUT rows and k,
// stored [N/64][K] (internal mode QMODE_AFFINE_GC)
template <typename YT, int QM>
__global__ void __launch_bounds__(F16_THREADS, 1)
qlinear_f16_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const F16Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;   // 1 KB aligned as declared
    const int x_stage_bytes = p.BN * XK * 2;
    uint8_t* sW = smem;
    uint8_t* sX = smem + (size_t)p.w_stages * W_STAGE_BYTES;
    float* sStage = reinterpret_cast<float*>(sX + (size_t)p.x_stages * x_stage_bytes);   // [EPI_WARPS][8][ST_PITCH]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStage) + ST_BYTES);
    uint64_t* w_full = bars;                   // [p.w_stages]
    uint64_t* w_empty = w_full + p.w_stages;     // [p.w_stages]
    uint64_t* a_full = w_empty + p.w_stages;     // [A_BUFS]
    uint64_t* a_empty = a_full + A_BUFS;       // [A_BUFS]
    uint64_t* d_full = a_empty + A_BUFS;       // [1]
    uint64_t* d_empty = d_full + 1;            // [1]
    uint64_t* x_full = d_empty + 1;            // [x_stages]
    uint64_t* x_empty = x_full + p.x_stages;   // [x_stages]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(x_empty + p.x_stages);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* last_flag = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = warp_id(), lane = threadIdx.x & 31;
    pdl_launch_dependents();
    __shared__ long long s_peer_delta[PEER_MAX_RANKS];
    // QM == 2: per converter warp two buffers of (64 scales, 64 biases): those of the stage being converted and of the next
    __shared__ __align__(16) float s_gc[QM == 2 ? CONV_WARPS * 256 : 4];
    if (threadIdx.x == 0) {
        int k = 0;  // the other ranks, compacted (own rank left out); static indices into the parameter
#pragma unroll
        for (int g = 0; g < PEER_MAX_RANKS; ++g)
            if (g < p.push.nranks && g != p.push.rank) s_peer_delta[k++] = p.push.delta[g];
    }
    const PeerOut po = {p.push.nranks > 1 ? p.push.nranks - 1 : 0, s_peer_delta};   // visible after the set-up barrier below

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.w_stages; ++s) {
            mbar_init(&w_full[s], 1);
            mbar_init(&w_empty[s], CONV_WARPS);
        }
        for (int s = 0; s < A_BUFS; ++s) {
            mbar_init(&a_full[s], CONV_WARPS);
            mbar_init(&a_empty[s], 1);
        }
        mbar_init(d_full, 1);
        mbar_init(d_empty, EPI_WARPS);
        for (int s = 0; s < p.x_stages; ++s) {
            mbar_init(&x_full[s], 1);
            mbar_init(&x_empty[s], 1);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a0 = tmem_base + D_COLS;

    if (warp == 0) {
        // ------------------------------ activation producer -----------------------
        const uint64_t pol_x = policy_evict_last();
        int xs = 0;
        uint32_t xph = 0;
        bool ok = true;
        PieceSched sched(p);
        Piece pc;
        pdl_wait();   // the activations may come from the previous kernel
        while (ok && sched.next(pc)) {
            const int j = pc.u / p.tiles_w;
            for (int s = 2 * pc.s0; s < 2 * pc.s1; ++s) {
                if (!mbar_wait(&x_empty[xs], xph ^ 1u, abort_flag, p.status, 12)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(&x_full[xs], (uint32_t)x_stage_bytes);
                    tma_load_2d(sX + (size_t)xs * x_stage_bytes, &map_x, s * XK, j * p.BN, &x_full[xs], pol_x);
                }
                __syncwarp();
                if (++xs == p.x_stages) { xs = 0; xph ^= 1u; }
            }
        }
    } else if (warp == W_WARP) {
        // ------------------------------ weight producer ---------------------------
        // a warp of its own: behind the activations it was held up by their ring, and the converters waited 900 cycles a stage
        // for weights that could have been there (the weights have their ring and the converted buffers to run ahead in).
        // The weights never depend on earlier kernels.
        const uint64_t pol_w = policy_evict_first();
        int ws = 0;
        uint32_t wph = 0;
        bool ok = true;
        PieceSched sched(p);
        Piece pc;
        while (ok && sched.next(pc)) {
            const int t = pc.u % p.tiles_w;
            for (int s = pc.s0; s < pc.s1; ++s) {
                if (!mbar_wait(&w_empty[ws], wph ^ 1u, abort_flag, p.status, 11)) { ok = false; break; }
                if (elect_one()) {
                    mbar_expect_tx(&w_full[ws], (uint32_t)W_STAGE_BYTES);
                    tma_load_2d(sW + (size_t)ws * W_STAGE_BYTES, &map_w, s * WK, t * BM, &w_full[ws], pol_w);
                }
                __syncwarp();
                if (++ws == p.w_stages) { ws = 0; wph ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------
        // the whole warp walks the pieces and waits; one elected lane issues
        int ab = 0, xs = 0;
        uint32_t aph = 0, xph = 0;
        bool ok = true;
        int i = 0;
        PieceSched sched(p);
        Piece pc;
        for (; ok && sched.next(pc); ++i) {
            if (!mbar_wait(d_empty, ((uint32_t)i & 1u) ^ 1u, abort_flag, p.status, 13)) { ok = false; break; }
            tc_fence_after();
            for (int s = pc.s0; s < pc.s1 && ok; ++s) {
                if (!mbar_wait(&a_full[ab], aph, abort_flag, p.status, 14)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_tmem = tmem_a0 + (uint32_t)(ab * A_COLS);
                for (int h = 0; h < WK / XK; ++h) {
                    if (!mbar_wait(&x_full[xs], xph, abort_flag, p.status, 15)) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t db = make_smem_desc(smem_u32(sX + (size_t)xs * x_stage_bytes));
                    if (elect_one()) {
#pragma unroll
                        for (int k16 = 0; k16 < XK / 16; ++k16)
                            umma_f16_ts(tmem_base, a_tmem + (uint32_t)((h * (XK / 16) + k16) * 8), db + (uint64_t)(2 * k16), p.idesc,
                                        (s > pc.s0 || h > 0 || k16 > 0) ? 1u : 0u);
                        umma_commit(&x_empty[xs]);
                        if (h == WK / XK - 1) {
                            umma_commit(&a_empty[ab]);
                            if (s == pc.s1 - 1) umma_commit(d_full);
                        }
                    }
                    __syncwarp();
                    if (++xs == p.x_stages) { xs = 0; xph ^= 1u; }
                }
                if (++ab == A_BUFS) { ab = 0; aph ^= 1u; }
            }
        }
    } else if (warp < 2 + CONV_WARPS) {
        // ------------------------------ converters --------------------------------
        // Warp pair (w, w+4) shares TMEM lane quarter q = w & 3; `half` picks k 0..63 or 64..127 of the stage.
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;
        const int r = q * 32 + lane;  // weight row inside the tile = TMEM lane
        int ws = 0, ab = 0;
        uint32_t wph = 0, aph = 0;
        bool ok = true;
        PieceSched sched(p);
        Piece pc;
        while (ok && sched.next(pc)) {
            const int n_row = (pc.u % p.tiles_w) * BM + r;   // this thread's weight row
            for (int s = pc.s0; s < pc.s1 && ok; ++s) {
                // affine: this thread's 64 k-elements of the stage are exactly one group of its row (K % 64 == 0)
                float g_sc = 0.0f, g_bi = 0.0f;
                // QM == 2: the warp's 32 rows lie in one 64-row group, so the stage's 64 scales and 64 biases are the same
                // for every lane: lane l copies four of them (cp.async, 16 bytes) into the warp's own corner of shared
                // memory, one stage ahead of the conversion that reads them back as broadcasts
                [[maybe_unused]] const float* gc = nullptr;
                if constexpr (QM == 2) {
                    float* mine = s_gc + (size_t)(warp - 2) * 256;
                    const bool rows_ok = n_row - lane < p.N;   // (N % 64 == 0: the group is inside the matrix or outside)
                    auto issue = [&](int st, int buf) {
                        const int k0 = st * WK + half * 64;
                        if (rows_ok && k0 < p.K) {
                            const float* src = (lane < 16 ? p.scales : p.biases) + (size_t)(n_row >> 6) * p.K + k0 + (lane & 15) * 4;
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(mine + buf * 128 + lane * 4)), "l"(src) : "memory");
                        }
                        asm volatile("cp.async.commit_group;" ::: "memory");
                    };
                    const int buf = (s - pc.s0) & 1;
                    if (s == pc.s0) issue(s, buf);
                    if (s + 1 < pc.s1) {
                        issue(s + 1, buf ^ 1);
                        asm volatile("cp.async.wait_group 1;" ::: "memory");
                    } else {
                        asm volatile("cp.async.wait_group 0;" ::: "memory");
                    }
                    __syncwarp();
                    if (rows_ok && s * WK + half * 64 < p.K) gc = mine + buf * 128;
                }
                if constexpr (QM == 1) {
                    const int k0 = s * WK + half * 64;
                    if (n_row < p.N && k0 < p.K) {
                        const size_t g = ((size_t)n_row * p.K + k0) >> 6;
                        g_sc = __ldg(p.scales + g);
                        g_bi = __ldg(p.biases + g);
                    }
                }
                if (!mbar_wait(&w_full[ws], wph, abort_flag, p.status, 16)) { ok = false; break; }
                // row r of the swizzled tile: logical 16-byte chunk c sits at physical chunk c ^ (r & 7)
                const uint32_t row = smem_u32(sW + (size_t)ws * W_STAGE_BYTES + (size_t)r * WK);
                uint4 raw[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) raw[c] = lds128(row + (uint32_t)(((half * 4 + c) ^ (r & 7)) << 4));
                __syncwarp();
                if (lane == 0) mbar_arrive_after(&w_empty[ws], raw, opaque_zero());  // this warp's share is in registers
                if (++ws == p.w_stages) { ws = 0; wph ^= 1u; }
                uint32_t cv[32];
                if constexpr (QM == 2) {
                    if (gc) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) u8x16_affine_vec_to_bf16x2(raw[c], gc + 16 * c, gc + 64 + 16 * c, cv + 8 * c);
                    } else {
#pragma unroll
                        for (int e = 0; e < 32; ++e) cv[e] = 0u;
                    }
                } else if constexpr (QM == 1) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) u8x16_affine_to_bf16x2(raw[c], g_sc, g_bi, cv + 8 * c);
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) int8x16_to_bf16x2(raw[c], cv + 8 * c);
                }
                if (!mbar_wait(&a_empty[ab], aph ^ 1u, abort_flag, p.status, 17)) { ok = false; break; }
                tc_fence_after();
                tmem_st32(tmem_a0 + ((uint32_t)(q * 32) << 16) + (uint32_t)(ab * A_COLS + half * 32), cv);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[ab]);
                if (++ab == A_BUFS) { ab = 0; aph ^= 1u; }
            }
        }
    } else {
        // ------------------------------ epilogue ----------------------------------
        const int q = warp & 3;
        const int r = q * 32 + lane;
        // this warp's share of the accumulator's columns (activation rows of the tile), in chunks of 16
        const int c_split = ((p.BN / 2 + 15) / 16) * 16;
        const int c_lo = (warp - (2 + CONV_WARPS)) >= 4 ? c_split : 0;
        const int c_hi = (warp - (2 + CONV_WARPS)) >= 4 ? p.BN : c_split;
        YT* y = reinterpret_cast<YT*>(p.y);
        float* stage = sStage + (size_t)(warp - (2 + CONV_WARPS)) * 8 * ST_PITCH;
        const int ev_row = lane >> 2, ev_col = (lane & 3) * 8;   // this lane's output row and columns of a turned tile
        pdl_wait();
        bool ok = true;
        int i = 0, n_cut = 0;
        PieceSched sched(p);
        Piece pc;
        Piece cut0, cut1;
        auto finish_cuts = [&]() {
            // Every CTA of the grid is resident (one an SM) and stores its pieces before it waits here: no wait depends on a CTA that
            // has not started.
            for (int e = 0; e < n_cut; ++e) {
                const Piece ct = e == 0 ? cut0 : cut1;
                if (threadIdx.x == 32 * (2 + CONV_WARPS)) {
                    const long long t0 = clock64();
                    while (ok && ld_acquire_gpu_u32(p.counters + ct.lu) < (unsigned)ct.nseg) {
                        if (*abort_flag || clock64() - t0 > WAIT_LIMIT_CYCLES) {
                            *abort_flag = 1;
                            if (atomicExch(&p.status->timeout_flag, 1u) == 0u) p.status->timeout_where = 19;
                            ok = false;
                        }
                    }
                    // the last of the tile's CTAs to get here leaves zeros for the next launch
                    if (ok && atomicAdd(p.counters + p.sk_units + ct.lu, 1u) == (unsigned)(ct.nseg - 1)) {
                        p.counters[ct.lu] = 0u;
                        p.counters[p.sk_units + ct.lu] = 0u;
                    }
                    *last_flag = ok ? 1 : 0;
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
                if (!*last_flag) { ok = false; break; }
                const int t = ct.u % p.tiles_w, j = ct.u / p.tiles_w;
                const int n = t * BM + r;
                const bool row_ok = n < p.N;
                const float sc = !row_ok ? 0.0f : QM != 0 ? 1.0f : __ldg(p.scales + n);
                const int quads = p.BN / 4, piece = (int)blockIdx.x - ct.first;
                const int q0 = piece * quads / ct.nseg, q1 = (piece + 1) * quads / ct.nseg;
                for (int qd = q0 + ((warp - (2 + CONV_WARPS)) >> 2); qd < q1; qd += 2) {
                    float res[4];   // on its way together with the pieces
                    if (p.residual) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int m = j * p.BN + qd * 4 + k;
                            res[k] = (row_ok && m < p.Mx) ? load_y<YT>(reinterpret_cast<const YT*>(p.residual) + (size_t)m * p.ldy + p.y_col0 + n) : 0.0f;
                        }
                    }
                    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int k0 = 0; k0 < ct.nseg; k0 += 4) {   // in a fixed order: the same bits on every run
                        float4 v[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k0 + k < ct.nseg) v[k] = __ldcg(piece_slot(p, ct.first + k0 + k, ct.lu) + (size_t)qd * BM + r);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k0 + k < ct.nseg) { f.x += v[k].x; f.y += v[k].y; f.z += v[k].z; f.w += v[k].w; }
                    }
                    const float vals[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) store_out<YT>(p, y, j * p.BN + qd * 4 + k, n, vals[k] * sc, row_ok, po, p.residual ? res[k] : 0.0f, true);
                }
                asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");   // last_flag is used again
            }
            n_cut = 0;
        };
        for (; ok && sched.next(pc); ++i) {
            // in front of a whole tile the exchange runs beside that tile's main loop
            if (n_cut > 0 && pc.nseg == 1) finish_cuts();
            if (!ok) break;
            const int t = pc.u % p.tiles_w, j = pc.u / p.tiles_w;
            const int n = t * BM + r;
            const bool row_ok = n < p.N;
            const float sc = !row_ok ? 0.0f : QM != 0 ? 1.0f : __ldg(p.scales + n);
            // the residual of the warp's first columns is on its way before the accumulator is there; two chunks ahead from then on
            const int n8 = t * BM + q * 32 + ev_col;
            const bool res = p.vec && p.residual && pc.nseg == 1;
            Octet<YT> r0[2], r1[2], r2[2];
            auto fetch_res = [&](Octet<YT> (&o)[2], int c0) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int m = j * p.BN + c0 + h * 8 + ev_row;
                    if (c0 < c_hi && m < p.Mx && n8 < p.N) {
                        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const YT*>(p.residual) + (size_t)m * p.ldy + p.y_col0 + n8);
#pragma unroll
                        for (int k = 0; k < (int)(sizeof(YT) / 2); ++k) o[h].q[k] = src[k];
                    }
                }
            };
            if (res) {
                fetch_res(r0, c_lo);
                fetch_res(r1, c_lo + 16);
            }
            if (!mbar_wait(d_full, (uint32_t)i & 1u, abort_flag, p.status, 18)) { ok = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
            if (pc.nseg == 1 && p.vec) {
                for (int c0 = c_lo; c0 < c_hi; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld16(taddr + (uint32_t)c0, v);
                    if (res) fetch_res(r2, c0 + 32);
                    tmem_ld_wait();
                    if (c0 + 16 >= c_hi) {   // the accumulator has been read
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(d_empty);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) stage[e * ST_PITCH + lane] = __uint_as_float(v[h * 8 + e]) * sc;
                        __syncwarp();
                        const float4 lo = *reinterpret_cast<const float4*>(stage + ev_row * ST_PITCH + ev_col);
                        const float4 hi = *reinterpret_cast<const float4*>(stage + ev_row * ST_PITCH + ev_col + 4);
                        __syncwarp();
                        float o[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                        const int m = j * p.BN + c0 + h * 8 + ev_row;
                        if (m < p.Mx && n8 < p.N) {
                            YT* dst = y + (size_t)m * p.ldy;
                            if (p.act) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) o[k] = __fdividef(o[2 * k], 1.0f + __expf(-o[2 * k])) * o[2 * k + 1];
                                store_run<YT, 4>(dst + ((p.y_col0 + n8) >> 1), o);
                            } else {
                                if (res) add_octet<YT>(o, r0[h]);
                                store_run<YT, 8>(dst + p.y_col0 + n8, o);
                            }
                        }
                    }
                    if (res) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            r0[h] = r1[h];
                            r1[h] = r2[h];
                        }
                    }
                }
                if (c_lo >= c_hi) {   // narrow tiles: nothing for this warp
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty);
                }
            } else if (pc.nseg == 1) {
                for (int c0 = c_lo; c0 < c_hi; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld16(taddr + (uint32_t)c0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; ++e) store_out<YT>(p, y, j * p.BN + c0 + e, n, __uint_as_float(v[e]) * sc, row_ok, po, 0.0f);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty);
            } else {
                // A K-slice of a shared tile goes into this CTA's slot; after its last piece the CTA adds up an equal share of the
                // tile's columns from all slots and writes it.  (Adding the slices into one tile with vector reductions and
                // letting the last arrival convert it cost 20 us at 256 rows: 128 KB of atomics a CTA, then one CTA alone.)
                float4* slot = piece_slot(p, (int)blockIdx.x, pc.lu);
                for (int c0 = c_lo; c0 < c_hi; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld16(taddr + (uint32_t)c0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        __stcg(slot + (size_t)((c0 + e) / 4) * BM + r, make_float4(__uint_as_float(v[e]), __uint_as_float(v[e + 1]),
                                                                                  __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3])));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty);
                __threadfence();
                asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
                if (threadIdx.x == 32 * (2 + CONV_WARPS)) atomicAdd(p.counters + pc.lu, 1u);
                if (n_cut == 0) cut0 = pc;
                else cut1 = pc;
                ++n_cut;
            }
        }
        finish_cuts();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace

namespace rusty {

bool f16tc_supported(const rusty_cuda_ctx*, const QLinearArgs& a) {
    if (!encode_tiled_fn()) return false;
    if (a.layout != RUSTY_CUDA_LAYOUT_NK) return false;
    if (a.qmode == RUSTY_CUDA_QMODE_AFFINE_G64 ? (a.K % 64 != 0 || a.act)
        : a.qmode == QMODE_AFFINE_GC          ? (a.K % 128 != 0 || a.N % 64 != 0 || a.act)
                                              : a.qmode != RUSTY_CUDA_QMODE_SYM_ROW)
        return false;
    if (a.x_dtype != RUSTY_CUDA_BF16) return false;
    if (a.K % 16 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(a.w) & 15) != 0 || (reinterpret_cast<uintptr_t>(a.x) & 15) != 0) return false;
    return true;
}

int launch_f16tc(rusty_cuda_ctx* ctx, const QLinearArgs& a) {
    F16Params p{};
    p.scales = a.scales;
    p.biases = (a.qmode == RUSTY_CUDA_QMODE_AFFINE_G64 || a.qmode == QMODE_AFFINE_GC) ? a.biases : nullptr;
    p.y = a.y;
    p.Mx = (int)a.M;
    p.N = (int)a.N;
    p.K = (int)a.K;
    // as few row tiles as 256 rows each allow, of equal width: 300 rows are 2 x 160, not 256 + 44 padded to 256
    p.tiles_n = (p.Mx + 255) / 256;
    p.BN = ((p.Mx + p.tiles_n - 1) / p.tiles_n + 15) / 16 * 16;
    p.tiles_w = (p.N + BM - 1) / BM;
    p.nws = (p.K + WK - 1) / WK;
    p.ldy = (int)a.ldy;
    p.y_col0 = (int)a.y_col0;
    p.act = a.act;
    p.residual = a.residual;
    {
        const size_t ysz = a.y_dtype == RUSTY_CUDA_BF16 ? 2 : 4, out_n = a.act ? a.N / 2 : a.N, col0 = a.act ? a.y_col0 / 2 : a.y_col0;
        const uint32_t run = (uint32_t)(a.act ? 4 : 8) * ysz >= 16 ? 16 : 8;   // bytes of a lane's access
        p.vec = !(a.push && a.push->nranks > 1) && a.N % 8 == 0 && (out_n * ysz) % run == 0 && (a.ldy * ysz) % run == 0 && (col0 * ysz) % run == 0 &&
                (reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.residual)) % run == 0;
    }
    if (a.push && a.push->nranks > 1) p.push = *a.push;
    p.status = ctx->status_dev;
    // bf16 A x bf16 B -> f32: c_format=F32(1)@4, a_format=BF16(1)@7, b_format=BF16(1)@10, N>>3 @17, M>>4 @24
    p.idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    // beside the rings: static shared memory (1 KB; 8 KB more in the group-column affine variant for its scales and biases), the
    // epilogue's staging, barriers.  The dynamic part starts on 1 KB as it is declared to: no slack for aligning it.
    const size_t reserve = (a.qmode == QMODE_AFFINE_GC ? 8192 : 0) + 1024 + ST_BYTES + 512;
    const size_t budget = ctx->smem_optin > reserve ? ctx->smem_optin - reserve : 0;
    const size_t x_stage = (size_t)p.BN * XK * 2;
    // Three weight stages and what is left in activation stages (five at 256 rows: 2.5 weight stages ahead); narrow tiles, whose
    // stages are short next to the trip to memory, take up to eight of each.
    int ws = 3;
    int xs = budget > (size_t)ws * W_STAGE_BYTES ? (int)((budget - (size_t)ws * W_STAGE_BYTES) / x_stage) : 0;
    if (xs > 16) xs = 16;
    if (xs < 2) return fail(ctx, RUSTY_CUDA_ERR_UNSUPPORTED, "f16 tensor-core path: tile does not fit shared memory");
    while (ws < 8 && xs >= 2 * (ws + 1) && (size_t)(ws + 1) * W_STAGE_BYTES + (size_t)(2 * (ws + 1)) * x_stage <= budget) ++ws;
    if (ws > 3) xs = 2 * ws;
    p.x_stages = xs;
    p.w_stages = ws;
    const size_t smem = (size_t)ws * W_STAGE_BYTES + (size_t)xs * x_stage + ST_BYTES + (size_t)(2 * ws + 2 * A_BUFS + 2 + 2 * xs) * 8 + 64;

    CUtensorMap map_w, map_x;
    if (!make_map_u8(&map_w, a.w, a.N, a.K, BM) || !make_map_bf16(&map_x, a.x, a.M, a.K, (uint32_t)p.BN))
        return fail(ctx, RUSTY_CUDA_ERR_KERNEL_EXECUTION, "f16 tensor-core path: cuTensorMapEncodeTiled failed");
    const int units = p.tiles_w * p.tiles_n;
    // Whole waves of tiles are taken tile-per-CTA.  The rest (all tiles, where there are fewer than SMs) is cut along K when that
    // saves more stages than exchanging the pieces costs: ten (~5 us) when every CTA has one piece and nothing else, more with
    // the tile's width when runs of stages leave a CTA with two pieces; in front of whole tiles only the storing of the pieces
    // shows.  (4096 x 14336 at 78 rows as 32 whole tiles: 102 us, 32 SMs busy; in four pieces each 29.)
    int grid = ctx->sm_count;
    const int rest = units % grid;
    p.sk_units = p.sk_per_cta = p.sk_ctas = p.sk_ways = 0;
    p.slots = nullptr;
    p.counters = nullptr;
    const int ways = rest > 0 ? (grid / rest < p.nws / 4 ? grid / rest : p.nws / 4) : 0;
    const int cut_stages = rest == 0 ? 0 : ways >= 2 ? (p.nws + ways - 1) / ways : (rest * p.nws + grid - 1) / grid;
    if (rest > 0 && cut_stages >= 2 && p.nws - cut_stages > (units >= grid ? 4 + p.BN / 32 : ways >= 2 ? 10 : 8 + p.BN / 12)) {
        size_t cnt_bytes = 0;
        unsigned int* counters = tc_workspace_counters(ctx, &cnt_bytes);
        // the pieces take the digit region, which this path has no digits for
        if (counters && (size_t)2 * grid * p.BN * BM * 4 <= tc_workspace_xq_bytes() && (size_t)2 * rest * 4 <= cnt_bytes) {
            p.sk_units = rest;
            p.sk_ways = ways >= 2 ? ways : 0;
            p.sk_per_cta = cut_stages;
            p.sk_ctas = ways >= 2 ? rest * ways : (rest * p.nws + cut_stages - 1) / cut_stages;
            p.slots = (float*)ctx->tc_ws;
            p.counters = counters;
        }
    }
    p.dp_units = units - p.sk_units;
    const int blocks = p.dp_units >= grid ? grid : p.dp_units > p.sk_ctas ? p.dp_units : p.sk_ctas;
    const bool yb = a.y_dtype == RUSTY_CUDA_BF16;
    const int qm = a.qmode == QMODE_AFFINE_GC ? 2 : p.biases != nullptr ? 1 : 0;
    auto kern = qm == 2   ? (yb ? qlinear_f16_tc_kernel<__nv_bfloat16, 2> : qlinear_f16_tc_kernel<float, 2>)
                : qm == 1 ? (yb ? qlinear_f16_tc_kernel<__nv_bfloat16, 1> : qlinear_f16_tc_kernel<float, 1>)
                          : (yb ? qlinear_f16_tc_kernel<__nv_bfloat16, 0> : qlinear_f16_tc_kernel<float, 0>);
    {
        cudaError_t e = ensure_dynamic_smem((const void*)kern, ctx->device, smem);
        if (e != cudaSuccess) return check_cuda(ctx, e, "qlinear_f16_tc: cudaFuncSetAttribute");
    }
    cudaError_t le = launch_pdl(kern, dim3(blocks), dim3(F16_THREADS), smem, ctx->stream, map_w, map_x, p);
    if (le != cudaSuccess) return check_cuda(ctx, le, "qlinear_f16_tc");
    return after_launch(ctx, "qlinear_f16_tc");
}

}  // namespace rusty
