// The step after the LM head, k > 1: the k largest logits of every row, on the device.
//
// WGSL `top_k` (rusty-backend/src/kernels.wgsl:168-188) is one thread running k rounds of "first index of the largest
// value not taken yet" (strict `>`, each round starting from max_v = -1e9 and max_idx = 0): the result is the k
// largest values in descending order, equal values in ascending index order; a value that is not > -1e9 (NaN
// included) is never taken, and a round that finds nothing reports index 0.  Same result here, computed per row by a
// cluster of blocks that bounds the k-th largest from below, collects what reaches the bound and orders it; the
// soft-max statistics of the row come from the same two walks.  With output-feature shards
// every rank selects from its own columns and only k (key, index) pairs per row and rank cross NVLink; every rank
// then merges the G x k candidates.  The reference's temperature / top-p Sampler (rusty-loader/src/tokenizer.rs:
// 149-204) needs exactly these k pairs when used with a top-k cut-off.
#include <cooperative_groups.h>

#include <cstring>

#include "internal.h"
#include "tc_common.cuh"

using namespace rusty;
using namespace rusty_tc;
namespace cg = cooperative_groups;

namespace {

constexpr int TK_THREADS = 1024;
constexpr int TK_MAX_K = 1024;
constexpr int TK_MAX_MERGE = 2048;      // sharded: G * k candidates per row

// Larger float <=> larger key; 0 = "not a candidate" (NaN, or not > -1e9 as in the shader).  -0.0 counts as +0.0.
__device__ __forceinline__ uint32_t key_of(float v) {
    if (!(v > -1e9f)) return 0u;
    uint32_t b = __float_as_uint(v);
    if (v == 0.0f) b = 0u;
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? (key ^ 0x80000000u) : ~key);
}
// sort item: key in the high word, inverted index in the low word: descending order of the 64-bit item is descending
// value, then ascending index.  0 = empty.
__device__ __forceinline__ unsigned long long item_of(uint32_t key, uint32_t idx) {
    return ((unsigned long long)key << 32) | (unsigned long long)(0xffffffffu - idx);
}

// descending bitonic sort of P (power of two, <= blockDim.x * per) items in shared memory
__device__ __forceinline__ void bitonic_desc(unsigned long long* a, int P) {
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int t = threadIdx.x; t < P / 2; t += blockDim.x) {
                const int lo = 2 * t - (t & (stride - 1));   // index with bit `stride` clear
                const int hi = lo + stride;
                const bool desc = (lo & size) == 0;
                const unsigned long long x = a[lo], y = a[hi];
                if ((x < y) == desc) {
                    a[lo] = y;
                    a[hi] = x;
                }
            }
        }
    }
    __syncthreads();
}

// The k winners of row[0, n) by ONE block, as items in descending order in cand[0, k) (zero-padded up to TK_MAX_K): an 8-bit
// radix select over the keys finds the k-th largest in four passes over the row, a fifth collects, a bitonic sort orders.
// Used by the sharded kernel, and by the cluster kernel below when too many logits tie with the k-th for its shortcut.
template <int T>
struct RadixScratch {
    unsigned int hist[T / 32][256];
    unsigned int prefix, need, kk, eq, cnt, run;
    unsigned int warp[T / 32];
};
template <int T>
__device__ void radix_topk(const float* row, int n, unsigned int col0, int k, unsigned long long* cand, RadixScratch<T>& s) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        s.prefix = 0u;
        s.need = (unsigned)k;
        s.kk = 0u;
    }
    uint32_t mask = 0u;
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < (T / 32) * 256; i += T) (&s.hist[0][0])[i] = 0u;
        __syncthreads();
        const uint32_t prefix = s.prefix;
        for (int j0 = 0; j0 < n; j0 += T) {
            const int j = j0 + tid;
            const uint32_t key = j < n ? key_of(row[j]) : 0u;
            const bool in = key != 0u && (key & mask) == prefix;
            const uint32_t d = (key >> shift) & 255u;
            // lanes of the warp that hit the same bin add once
            const unsigned peers = __match_any_sync(0xffffffffu, in ? d : 256u + (uint32_t)lane);
            if (in && (unsigned)lane == (unsigned)(__ffs(peers) - 1)) s.hist[warp][d] += (unsigned)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < 256) {
            unsigned sum = 0;
#pragma unroll 8
            for (int w = 0; w < T / 32; ++w) sum += s.hist[w][tid];
            s.hist[0][tid] = sum;
        }
        __syncthreads();
        if (tid == 0) {
            if (pass == 0) {
                unsigned total = 0;
                for (int d = 0; d < 256; ++d) total += s.hist[0][d];
                s.kk = total < (unsigned)k ? total : (unsigned)k;
                s.need = s.kk;
            }
            unsigned need = s.need, cum = 0;
            if (need > 0) {
                int d = 255;
                for (; d > 0; --d) {
                    if (cum + s.hist[0][d] >= need) break;
                    cum += s.hist[0][d];
                }
                s.need = need - cum;                 // how many of this bin are still wanted
                s.prefix = prefix | ((uint32_t)d << shift);
                s.eq = s.hist[0][d];                 // after the last pass: elements equal to the k-th key
            }
        }
        mask |= 0xffu << shift;
        __syncthreads();
    }
    const unsigned kk = s.kk, need_eq = s.need, count_eq = s.eq;
    const uint32_t Tk = s.prefix;
    for (int i = tid; i < TK_MAX_K; i += T) cand[i] = 0ull;
    if (tid == 0) {
        s.cnt = 0u;
        s.run = 0u;
    }
    __syncthreads();
    if (kk > 0) {
        // everything above the k-th key, and the equals when all of them are wanted
        const bool all_eq = count_eq == need_eq;
        for (int j = tid; j < n; j += T) {
            const uint32_t key = key_of(row[j]);
            if (key > Tk || (all_eq && key == Tk)) cand[atomicAdd(&s.cnt, 1u)] = item_of(key, col0 + (uint32_t)j);
        }
        __syncthreads();
        if (!all_eq) {
            // more equals than wanted: the first need_eq of them in index order (a block-wide ordered count per
            // chunk of T consecutive elements; stops once enough are found)
            for (int j0 = 0; j0 < n; j0 += T) {
                const int j = j0 + tid;
                const bool eq = j < n && key_of(row[j]) == Tk;
                const unsigned bal = __ballot_sync(0xffffffffu, eq);
                if (lane == 0) s.warp[warp] = (unsigned)__popc(bal);
                __syncthreads();
                unsigned before = s.run;
                for (int w = 0; w < warp; ++w) before += s.warp[w];
                const unsigned rank_eq = before + (unsigned)__popc(bal & ((1u << lane) - 1u));
                if (eq && rank_eq < need_eq) cand[kk - need_eq + rank_eq] = item_of(Tk, col0 + (uint32_t)j);
                __syncthreads();
                if (tid == 0) {
                    unsigned tot = 0;
                    for (int w = 0; w < T / 32; ++w) tot += s.warp[w];
                    s.run += tot;
                }
                __syncthreads();
                if (s.run >= need_eq) break;
            }
        }
        int P = 1;
        while (P < (int)kk) P <<= 1;
        bitonic_desc(cand, P);
    }
    __syncthreads();
}

// Sharded, first half.  One block per row (rows b, b + grid, ...): the row's k winners, sorted, as items into slot `rank` of
// every rank's candidate table ([G][M][k], zero-padded).
__global__ void __launch_bounds__(TK_THREADS) topk_rows_push_kernel(const float* x, int n, size_t ld, unsigned int col0, int k, int M,
                                                                    unsigned long long* __restrict__ table, const PeerPush pp) {
    __shared__ RadixScratch<TK_THREADS> scratch;
    __shared__ unsigned long long cand[TK_MAX_K];
    const int tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (tid < 32) peer_sync_block(pp, (int)blockIdx.x, 34);   // the table of the previous step has been merged everywhere
    __syncthreads();
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        radix_topk<TK_THREADS>(x + (size_t)m * ld, n, col0, k, cand, scratch);
        for (int i = tid; i < k; i += TK_THREADS) {
            const unsigned long long it = cand[i];
            unsigned long long* slot = table + ((size_t)pp.rank * M + m) * k + i;
            *slot = it;
            for (int g = 0; g < pp.nranks; ++g)
                if (g != pp.rank) *reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(slot) + pp.delta[g]) = it;
        }
        __syncthreads();
    }
}

// The k largest of every row and / or its soft-max statistics, one device.  A cluster of S blocks per row (row_cluster):
// each block walks its slice of the row (L2-resident after the LM head) at most twice.
//   Walk 1 keeps each thread's largest key; the maxima of groups of 2^g lanes are distinct elements of the row, so the k-th
//   largest of these (rank counting over the <= RC_GROUPS of all blocks) bounds the k-th largest logit from below.  g is the
//   largest group that leaves at least 2k maxima: then only ~1.4 k elements lie above the bound when the large logits are
//   spread over the row.
//   Walk 2 hands every element at or above the bound to block 0, which orders them by counting ranks (items are unique), and
//   adds up exp((x - max) / T) for the statistics.
// More than RC_CAP elements at the bound (masses of ties, or all large logits side by side): block 0 runs the radix select.
// Bound by latency: two walks, three cluster barriers.  32 rows x 128256, k = 64: the radix select with one block of 1024
// threads a row took 525 us, this takes 15; the statistics alone 26 -> 9.
constexpr int RC_THREADS = 512;
constexpr int RC_GROUPS = 4096;      // maxima of all blocks: 8 blocks x 512 threads at most
constexpr int RC_CAP = 2048;
struct RowShared {
    union {
        uint32_t gmax[RC_GROUPS];                        // every block: the group maxima of all blocks
        struct {
            unsigned long long sorted[TK_MAX_K];         // block 0, after the bound is known
            RadixScratch<RC_THREADS> radix;
        } s;
    } u;
    unsigned long long cand[RC_CAP];                     // block 0: elements at or above the bound
    uint32_t max_of[8];                                  // every block: the largest key of every block
    float sum_of[8];                                     // block 0: every block's part of the sum
    uint32_t bound, count, red_k[RC_THREADS / 32];
    float red_f[RC_THREADS / 32];
};
// keys of the statistics: every number but NaN counts, -inf included
__device__ __forceinline__ uint32_t stat_key_of(float v) {
    if (v != v) return 0u;
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// The draw of temperature / top-p sampling from the row's k winners (Sampler::sample, rusty-loader/src/tokenizer.rs:161-204): in f32 and in
// the reference's order of operations.  One token per row instead of k pairs: the walk over them on the host, in numpy, took 60 us
// for 32 rows.
constexpr uint32_t NO_TOKEN = 0xffffffffu;     // the winners' probabilities do not reach top_p: the row has to be drawn from as a whole
struct DrawArgs {
    const float* draws;    // [M] uniform numbers in [0, 1); null: no draw
    uint32_t* tokens;      // [M]
    float temperature, top_p;
};

__global__ void __launch_bounds__(RC_THREADS) logits_rows_kernel(const float* x, int n, size_t ld, int k, int glog,
                                                                 unsigned int* __restrict__ out_idx, float* __restrict__ out_val,
                                                                 float inv_t, float* __restrict__ out_max, float* __restrict__ out_sum, const DrawArgs draw) {
    extern __shared__ __align__(16) unsigned char row_smem[];
    RowShared& sh = *reinterpret_cast<RowShared*>(row_smem);
    cg::cluster_group cl = cg::this_cluster();
    const unsigned S = cl.num_blocks(), r = cl.block_rank(), m = blockIdx.x / S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool stats = out_sum != nullptr || draw.draws != nullptr;
    const float rnd = draw.draws && r == 0 && tid == 0 ? draw.draws[m] : 0.0f;     // (from host memory: asked for early)
    if (tid == 0) sh.count = 0u;
    pdl_launch_dependents();
    cl.barrier_arrive();          // the blocks of the cluster have started and cleared their counters (waited for below)
    pdl_wait();
    const float* row = x + (size_t)m * ld;
    uint32_t kmax = 0u, smax = 0u;
    walk_row_slice<RC_THREADS>(row, n, r, S, [&](float v, int) {
        if (k > 0) kmax = max(kmax, key_of(v));
        if (stats) smax = max(smax, stat_key_of(v));
    });
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, smax);
    if (lane == 0) sh.red_k[warp] = wmax;
    for (int off = 1; off < (1 << glog); off <<= 1) kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, off));
    __syncthreads();
    cl.barrier_wait();
    const int per = RC_THREADS >> glog, groups = per * (int)S;   // group maxima per block, in all
    if (k > 0 && (tid & ((1 << glog) - 1)) == 0)
        for (unsigned b = 0; b < S; ++b) cl.map_shared_rank(sh.u.gmax, b)[r * per + (tid >> glog)] = kmax;
    if (warp == 0 && stats) {
        const uint32_t bmax = __reduce_max_sync(0xffffffffu, lane < RC_THREADS / 32 ? sh.red_k[lane] : 0u);
        if (lane < (int)S) cl.map_shared_rank(sh.max_of, lane)[r] = bmax;
    }
    cl.sync();
    float mx = __int_as_float(0xff800000);
    if (stats) {
        uint32_t key = 0u;
        for (unsigned b = 0; b < S; ++b) key = max(key, sh.max_of[b]);
        if (key) mx = value_of(key);
    }
    uint32_t bound = 1u;          // key 0 is no candidate
    if (k > 0 && groups >= k) {
        // the maximum whose rank (larger ones, equal ones at lower positions) is k - 1 is the bound
        if (tid == 0) sh.bound = 1u;
        __syncthreads();
        for (int i = tid; i < groups; i += RC_THREADS) {
            const uint32_t mine = sh.u.gmax[i];
            int rank = 0;
            for (int j = 0; j < groups; j += 4) {   // groups is a multiple of 16
                const uint4 q = *reinterpret_cast<const uint4*>(sh.u.gmax + j);
                rank += (q.x > mine || (q.x == mine && j < i)) + (q.y > mine || (q.y == mine && j + 1 < i)) +
                        (q.z > mine || (q.z == mine && j + 2 < i)) + (q.w > mine || (q.w == mine && j + 3 < i));
            }
            if (rank == k - 1) sh.bound = max(mine, 1u);
        }
        __syncthreads();
        bound = sh.bound;
    }
    float sum = 0.0f;
    unsigned long long* cand0 = cl.map_shared_rank(sh.cand, 0);
    uint32_t* count0 = cl.map_shared_rank(&sh.count, 0);
    walk_row_slice<RC_THREADS>(row, n, r, S, [&](float v, int j) {
        if (k > 0) {
            const uint32_t key = key_of(v);
            if (key >= bound) {
                const uint32_t at = atomicAdd(count0, 1u);
                if (at < (uint32_t)RC_CAP) cand0[at] = item_of(key, (uint32_t)j);
            }
        }
        if (stats && v == v) sum += expf((v - mx) * inv_t);
    });
    if (stats) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) sh.red_f[warp] = sum;
        __syncthreads();
        if (warp == 0) {
            sum = lane < RC_THREADS / 32 ? sh.red_f[lane] : 0.0f;
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (lane == 0) cl.map_shared_rank(sh.sum_of, 0)[r] = sum;
        }
    }
    cl.sync();
    if (r != 0) return;
    float total = 0.0f;
    if (stats) {
        for (unsigned b = 0; b < S; ++b) total += sh.sum_of[b];
        if (tid == 0 && out_sum) {
            out_max[m] = mx;
            out_sum[m] = total;
        }
    }
    if (k == 0) return;
    unsigned int* oi = out_idx + (size_t)m * k;
    float* ov = out_val ? out_val + (size_t)m * k : nullptr;
    unsigned long long* sorted = sh.u.s.sorted;           // (draw: where the group maxima were)
    auto put = [&](int at, unsigned long long it) {
        if (draw.draws) {
            sorted[at] = it;
            return;
        }
        oi[at] = it ? 0xffffffffu - (uint32_t)(it & 0xffffffffull) : 0u;
        if (ov) ov[at] = it ? value_of((uint32_t)(it >> 32)) : __int_as_float(0xff800000);
    };
    const uint32_t C = sh.count;
    if (C <= (uint32_t)RC_THREADS) {
        if ((uint32_t)tid < C) {
            const unsigned long long mine = sh.cand[tid];
            int rank = 0;
            for (uint32_t j = 0; j < C; ++j) rank += sh.cand[j] > mine;
            if (rank < k) put(rank, mine);
        }
        for (int i = (int)C + tid; i < k; i += RC_THREADS) put(i, 0ull);
    } else if (C <= (uint32_t)RC_CAP) {
        int P = 1;
        while (P < (int)C) P <<= 1;
        for (int i = (int)C + tid; i < P; i += RC_THREADS) sh.cand[i] = 0ull;
        bitonic_desc(sh.cand, P);
        for (int i = tid; i < k; i += RC_THREADS) put(i, sh.cand[i]);
    } else {
        radix_topk<RC_THREADS>(row, n, 0u, k, sorted, sh.u.s.radix);
        if (!draw.draws)
            for (int i = tid; i < k; i += RC_THREADS) put(i, sorted[i]);
    }
    if (!draw.draws) return;
    __syncthreads();
    float* probs = reinterpret_cast<float*>(sh.cand);     // [k]
    uint32_t idx[TK_MAX_K / RC_THREADS];
    float prob[TK_MAX_K / RC_THREADS];
    const float top = __fdiv_rn(mx, draw.temperature);
#pragma unroll
    for (int u = 0; u < TK_MAX_K / RC_THREADS; ++u) {
        const int i = tid + u * RC_THREADS;
        const unsigned long long it = i < k ? sorted[i] : 0ull;
        idx[u] = it ? 0xffffffffu - (uint32_t)(it & 0xffffffffull) : 0u;
        const float v = it ? value_of((uint32_t)(it >> 32)) : __int_as_float(0xff800000);
        prob[u] = __fdiv_rn(expf(__fdiv_rn(v, draw.temperature) - top), total);
    }
    __syncthreads();                                       // (the candidates and the sorted items have been read)
    uint32_t* index = reinterpret_cast<uint32_t*>(sorted);
#pragma unroll
    for (int u = 0; u < TK_MAX_K / RC_THREADS; ++u) {
        const int i = tid + u * RC_THREADS;
        if (i < k) {
            probs[i] = prob[u];
            index[i] = idx[u];
        }
    }
    __syncthreads();
    if (tid == 0) {
        float cum = 0.0f;
        int last = -1;
        for (int i = 0; i < k && last < 0; ++i) {
            cum = __fadd_rn(cum, probs[i]);
            if (cum >= draw.top_p) last = i;
        }
        uint32_t token = NO_TOKEN;
        if (last >= 0) {
            token = index[0];
            float c = 0.0f;
            for (int i = 0; i <= last; ++i) {
                c = __fadd_rn(c, __fdiv_rn(probs[i], cum));
                if (rnd < c) {
                    token = index[i];
                    break;
                }
            }
        }
        draw.tokens[m] = token;
    }
}

// k == 0: no top-k; out_sum == null: no statistics.
cudaError_t launch_logits_rows(rusty_cuda_ctx* ctx, const float* x, uint32_t M, uint32_t N, uint32_t k, unsigned int* out_idx, float* out_val,
                               float temperature, float* out_max, float* out_sum, const DrawArgs& draw = DrawArgs{}) {
    const unsigned S = row_cluster(M, N, ctx->sm_count);
    int glog = 5;
    while (glog > 0 && (uint64_t)S * (RC_THREADS >> glog) < 2ull * k) --glog;
    cudaError_t e = ensure_dynamic_smem((const void*)logits_rows_kernel, ctx->device, sizeof(RowShared));
    if (e != cudaSuccess) return e;
    return launch_pdl_cluster(logits_rows_kernel, dim3(M * S), dim3(RC_THREADS), S, sizeof(RowShared), ctx->stream, x, (int)N, (size_t)N, (int)k,
                              glog, out_idx, out_val, out_sum || draw.draws ? 1.0f / temperature : 0.0f, out_max, out_sum, draw);
}

// Sharded, second half: once every rank's candidates have landed, the best k of the G x k items of each row.
__global__ void __launch_bounds__(TK_THREADS) topk_merge_kernel(const unsigned long long* __restrict__ table, int M, int G, int k,
                                                                unsigned int* __restrict__ out_idx, float* __restrict__ out_val,
                                                                const PeerPush pp) {
    __shared__ unsigned long long items[TK_MAX_MERGE];
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x < 32) peer_sync_block(pp, (int)blockIdx.x, 35);
    __syncthreads();
    const int total = G * k;
    int P = 1;
    while (P < total) P <<= 1;
    for (int m = blockIdx.x; m < M; m += gridDim.x) {
        for (int i = threadIdx.x; i < P; i += blockDim.x) {
            unsigned long long it = 0ull;
            if (i < total) {
                const int g = i / k, j = i - g * k;
                it = __ldcg(table + ((size_t)g * M + m) * k + j);
            }
            items[i] = it;
        }
        bitonic_desc(items, P);
        for (int i = threadIdx.x; i < k; i += blockDim.x) {
            const unsigned long long it = items[i];
            out_idx[(size_t)m * k + i] = it ? 0xffffffffu - (uint32_t)(it & 0xffffffffull) : 0u;
            if (out_val) out_val[(size_t)m * k + i] = it ? value_of((uint32_t)(it >> 32)) : __int_as_float(0xff800000);
        }
        __syncthreads();
    }
    // like the arg-max table: the next table write of any rank waits until every rank has merged this one
}

}  // namespace

namespace rusty {
const PeerPush* arena_push_state(const rusty_cuda_arena* arena);
bool arena_holds(const rusty_cuda_arena* arena, const void* ptr, size_t bytes);
rusty_cuda_ctx* arena_ctx(const rusty_cuda_arena* arena);
}  // namespace rusty

extern "C" {

int rusty_cuda_top_k_rows_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* logits, uint32_t M, uint32_t N, uint32_t k, rusty_cuda_buf* out_idx,
                              rusty_cuda_buf* out_val) {
    RUSTY_REQUIRE_CTX(ctx);
    if (!logits || !out_idx) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "top_k_rows: null buffer");
    if (k == 0 || k > (uint32_t)TK_MAX_K) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows: k=%u must lie in 1..%d", k, TK_MAX_K);
    if (N > 0x7fffffffu) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows: N=%u too large", N);
    if (logits->bytes < (size_t)M * N * 4 || out_idx->bytes < (size_t)M * k * 4 || (out_val && out_val->bytes < (size_t)M * k * 4))
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows: [%u,%u] logits need %zu bytes, [%u,%u] indices (and values) %zu", M, N,
                    (size_t)M * N * 4, M, k, (size_t)M * k * 4);
    if (M == 0) return RUSTY_CUDA_OK;
    DeviceGuard g(ctx->device);
    cudaError_t e = launch_logits_rows(ctx, (const float*)logits->ptr, M, N, k, (unsigned int*)out_idx->ptr,
                                       out_val ? (float*)out_val->ptr : nullptr, 1.0f, nullptr, nullptr);
    if (e != cudaSuccess) return check_cuda(ctx, e, "top_k_rows");
    return after_launch(ctx, "top_k_rows");
}

int rusty_cuda_softmax_stats_rows_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* logits, uint32_t M, uint32_t N, float temperature,
                                      rusty_cuda_buf* out_max, rusty_cuda_buf* out_sum) {
    RUSTY_REQUIRE_CTX(ctx);
    if (!logits || !out_max || !out_sum) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "softmax_stats_rows: null buffer");
    if (!(temperature > 0.0f)) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "softmax_stats_rows: temperature must be > 0 (greedy choice is argmax_rows)");
    if (N > 0x7fffffffu) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "softmax_stats_rows: N=%u too large", N);
    if (logits->bytes < (size_t)M * N * 4 || out_max->bytes < (size_t)M * 4 || out_sum->bytes < (size_t)M * 4)
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "softmax_stats_rows: [%u,%u] logits need %zu bytes, the outputs %zu each", M, N,
                    (size_t)M * N * 4, (size_t)M * 4);
    if (M == 0) return RUSTY_CUDA_OK;
    DeviceGuard g(ctx->device);
    cudaError_t e = launch_logits_rows(ctx, (const float*)logits->ptr, M, N, 0u, nullptr, nullptr, temperature, (float*)out_max->ptr,
                                       (float*)out_sum->ptr);
    if (e != cudaSuccess) return check_cuda(ctx, e, "softmax_stats_rows");
    return after_launch(ctx, "softmax_stats_rows");
}

// What both calls for a sampling host check.
static int sampler_check(rusty_cuda_ctx* ctx, const char* op, const rusty_cuda_buf* logits, uint32_t M, uint32_t N, uint32_t k, float temperature) {
    if (ctx->capturing) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: not allowed while a graph capture is open", op);
    if (!(temperature > 0.0f)) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: temperature must be > 0 (greedy choice is argmax_rows)", op);
    if (k == 0 || k > (uint32_t)TK_MAX_K) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: k=%u must lie in 1..%d", op, k, TK_MAX_K);
    if (N > 0x7fffffffu) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: N=%u too large", op, N);
    if (logits->bytes < (size_t)M * N * 4)
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "%s: [%u,%u] logits need %zu bytes", op, M, N, (size_t)M * N * 4);
    return RUSTY_CUDA_OK;
}
// The context's pinned staging memory, of `need` bytes at least, and its address on the device.
static int sampler_stage(rusty_cuda_ctx* ctx, const char* op, size_t need, void** dev) {
    if (ctx->host_stage_bytes < need) {
        if (ctx->host_stage) cudaFreeHost(ctx->host_stage);   // (nothing in flight uses it: every use ends with a wait)
        ctx->host_stage = nullptr;
        ctx->host_stage_bytes = 0;
        cudaError_t e = cudaHostAlloc(&ctx->host_stage, need, cudaHostAllocMapped);
        if (e != cudaSuccess) {
            cudaGetLastError();
            ctx->host_stage = nullptr;
            return fail(ctx, RUSTY_CUDA_ERR_MEMORY_ALLOCATION, "%s: pinned staging of %zu bytes", op, need);
        }
        ctx->host_stage_bytes = need;
    }
    return check_cuda(ctx, cudaHostGetDevicePointer(dev, ctx->host_stage, 0), "sampler: staging");
}

int rusty_cuda_sampler_candidates_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* logits, uint32_t M, uint32_t N, uint32_t k, float temperature,
                                      uint32_t* host_idx, float* host_val, float* host_max, float* host_sum) {
    RUSTY_REQUIRE_CTX(ctx);
    const char* op = "sampler_candidates";
    if (!logits || !host_idx || !host_val || !host_max || !host_sum) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: null argument", op);
    int rc = sampler_check(ctx, op, logits, M, N, k, temperature);
    if (rc || M == 0) return rc;
    DeviceGuard g(ctx->device);
    const size_t pairs = (size_t)M * k;
    void* dev = nullptr;
    if ((rc = sampler_stage(ctx, op, pairs * 8 + (size_t)M * 8, &dev))) return rc;
    // one kernel, whose last block per row stores the results into host memory: no copies behind it
    unsigned int* d_idx = (unsigned int*)dev;
    float *d_val = (float*)(d_idx + pairs), *d_max = d_val + pairs, *d_sum = d_max + M;
    cudaError_t e = launch_logits_rows(ctx, (const float*)logits->ptr, M, N, k, d_idx, d_val, temperature, d_max, d_sum);
    if (e != cudaSuccess) return check_cuda(ctx, e, "sampler_candidates");
    if ((rc = after_launch(ctx, "sampler_candidates"))) return rc;
    if ((rc = rusty_cuda_sync(ctx))) return rc;
    const char* h = (const char*)ctx->host_stage;
    memcpy(host_idx, h, pairs * 4);
    memcpy(host_val, h + pairs * 4, pairs * 4);
    memcpy(host_max, h + pairs * 8, (size_t)M * 4);
    memcpy(host_sum, h + pairs * 8 + (size_t)M * 4, (size_t)M * 4);
    return RUSTY_CUDA_OK;
}

int rusty_cuda_sample_top_p_f32(rusty_cuda_ctx* ctx, const rusty_cuda_buf* logits, uint32_t M, uint32_t N, uint32_t k, float temperature, float top_p,
                                const float* host_draws, uint32_t* host_tokens) {
    RUSTY_REQUIRE_CTX(ctx);
    const char* op = "sample_top_p";
    if (!logits || !host_draws || !host_tokens) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "%s: null argument", op);
    int rc = sampler_check(ctx, op, logits, M, N, k, temperature);
    if (rc || M == 0) return rc;
    DeviceGuard g(ctx->device);
    void* dev = nullptr;
    if ((rc = sampler_stage(ctx, op, (size_t)M * 8, &dev))) return rc;
    memcpy(ctx->host_stage, host_draws, (size_t)M * 4);
    uint32_t* tokens = (uint32_t*)dev + M;
    cudaError_t e = launch_logits_rows(ctx, (const float*)logits->ptr, M, N, k, nullptr, nullptr, temperature, nullptr, nullptr,
                                       DrawArgs{(const float*)dev, tokens, temperature, top_p});
    if (e != cudaSuccess) return check_cuda(ctx, e, op);
    if ((rc = after_launch(ctx, op))) return rc;
    if ((rc = rusty_cuda_sync(ctx))) return rc;
    memcpy(host_tokens, (const char*)ctx->host_stage + (size_t)M * 4, (size_t)M * 4);
    return RUSTY_CUDA_OK;
}

int rusty_cuda_top_k_rows_sharded(rusty_cuda_ctx* ctx, rusty_cuda_arena* arena, const rusty_cuda_buf* logits_shard, uint32_t M, uint32_t Nl,
                                  uint32_t k, rusty_cuda_buf* table, rusty_cuda_buf* out_idx, rusty_cuda_buf* out_val) {
    RUSTY_REQUIRE_CTX(ctx);
    if (!arena || !logits_shard || !table || !out_idx) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "top_k_rows_sharded: null argument");
    if (arena_ctx(arena) != ctx) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "top_k_rows_sharded: arena of another context");
    const PeerPush* pp = arena_push_state(arena);
    if (!pp) return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "top_k_rows_sharded: arena not attached");
    const int G = pp->nranks < 1 ? 1 : pp->nranks;
    if (k == 0 || (size_t)k * G > (size_t)TK_MAX_MERGE || k > (uint32_t)TK_MAX_K)
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows_sharded: k=%u x %d ranks must lie in 1..%d", k, G, TK_MAX_MERGE);
    if ((uint64_t)Nl * (uint64_t)G > 0x7fffffffull) return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows_sharded: N too large");
    if (logits_shard->bytes < (size_t)M * Nl * 4 || out_idx->bytes < (size_t)M * k * 4 || (out_val && out_val->bytes < (size_t)M * k * 4))
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_DIMENSIONS, "top_k_rows_sharded: buffers too small for [%u,%u], k=%u", M, Nl, k);
    const size_t table_b = (size_t)G * M * k * 8;
    if (table->bytes < table_b || !arena_holds(arena, table->ptr, table_b))
        return fail(ctx, RUSTY_CUDA_ERR_INVALID_OPERATION, "top_k_rows_sharded: the candidate table ([%d][%u][%u] x 8 bytes) must be a buffer of the arena", G, M, k);
    if (M == 0) return RUSTY_CUDA_OK;
    DeviceGuard g(ctx->device);
    const unsigned blocks = M < (uint32_t)PEER_SYNC_SLOTS ? M : (unsigned)PEER_SYNC_SLOTS;
    cudaError_t e = launch_pdl(topk_rows_push_kernel, dim3(blocks), dim3(TK_THREADS), 0, ctx->stream, (const float*)logits_shard->ptr, (int)Nl, (size_t)Nl,
                               (unsigned int)pp->rank * Nl, (int)k, (int)M, (unsigned long long*)table->ptr, *pp);
    if (e != cudaSuccess) return check_cuda(ctx, e, "top_k_rows_push");
    int rc = after_launch(ctx, "top_k_rows_push");
    if (rc) return rc;
    e = launch_pdl(topk_merge_kernel, dim3(blocks), dim3(TK_THREADS), 0, ctx->stream, (const unsigned long long*)table->ptr, (int)M, G, (int)k,
                   (unsigned int*)out_idx->ptr, out_val ? (float*)out_val->ptr : (float*)nullptr, *pp);
    if (e != cudaSuccess) return check_cuda(ctx, e, "top_k_merge");
    return after_launch(ctx, "top_k_merge");
}

}  // extern "C"
