// Causal grouped-query attention over the paged cache in float32 FMA arithmetic: the attention of the float32 path.  (Head sizes
// and layouts it does not take, and bfloat16 without tensor cores, go to attention_generic.cu.)
//
// THE ORDER OF A SUM is a function of the query's position alone (and of the window), so a token's result does not depend on how the
// tokens were cut into steps, on the batch, or on the pages: the keys are cut into chunks of 64 that start at multiples of 64, and
// the chunks into 8 stripes (chunk mod 8).  A stripe is an online softmax over its chunks in ascending order; the stripes are merged
// in order 0 .. 7.  A score is two chains of fused multiply-adds (even and odd elements), a chunk's probabilities are added by the
// butterfly of a warp, an output column is one chain over a chunk's keys.  Query head h reads KV head h / (nh / nkv); the query at
// position p sees keys max(0, p - window + 1) .. p.
//
// What bounds it: a few tokens, the latency of one block's walk over the keys, which is why there are stripes: the blocks of a
// cluster take one each and merge through distributed shared memory.  Many tokens, the FMA pipes: a block takes 32 rows (tokens x
// the query heads that share the KV head), each staged key serves all of them, and it walks the stripes itself, one after another.
// Keys and values come by cp.async, each into one buffer that is refilled as soon as its product is done.
// Measured (16 heads, 4 KV heads of 128; before: a block per token and head, a thread per key with scalar loads, all keys in one
// walk): 4 tokens over contexts of 350 to 700, 113 -> 17 us; 301 tokens of a prompt, 432 -> 56 us.
//
// Semantics follow the reference's float32 kernels: scale applied to the dot product, running maximum and sum in float32, one
// rounding at the store (src/kernels/attention.cu:51-110 decode, :126-219 prefill; causal offset kv_len - q_len + i,
// src/model/attention.rs:1038-1063).
#include "common.cuh"
#include <type_traits>
#include <limits.h>
#include <math.h>

namespace {

constexpr int AF_THREADS = 128;
constexpr int AF_KEYS = 64;                 // keys per chunk
constexpr int AF_STRIPES = 8;               // = blocks of a cluster (the portable limit)
constexpr int AF_SP = AF_KEYS + 4;          // pitch of the score rows: 8 rows' 16-byte reads meet 32 banks
constexpr int AF_TILE = 64;                 // tokens of an entry of the step's tile list

struct AttnF32Args {
    const float* q;              // [T, q_stride]; head h at column h*d
    const float* k_pool;         // [num_pages, nkv, page_size, d]
    const float* v_pool;
    float* out;                  // [T, nh*d]
    const int* positions;        // [T]
    const int* seq_slot;         // [B]
    const int* q_start;          // [B + 1]
    const int* block_table;      // [slots, max_pages]
    const int* tiles;            // (sequence, first token) of every AF_TILE tokens, or null: sequence x brings one token
    int* status;
    int nh, nkv, d, q_stride, page_size, max_pages, num_pages, window;
    int group, tokens;           // query heads of a KV head; tokens of a block's rows
    int stripes_apart;           // 1: the blocks of a cluster take a stripe each
    int overlap;                 // kernels behind may start before this one ends
    float scale;
};

__device__ __forceinline__ uint32_t af_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void af_cp16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(af_smem(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ float af_ld_cluster(const float* local, int rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(af_smem(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void af_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// What the states so far and the next stripe are multiplied with when the stripe (maximum m) joins them (maximum M, updated).
struct AfMerge {
    float before, stripe;
};
__device__ __forceinline__ AfMerge af_merge(float& M, float m) {
    const float top = fmaxf(M, m);
    AfMerge f{M == -INFINITY ? 0.f : expf(M - top), m == -INFINITY ? 0.f : expf(m - top)};
    M = top;
    return f;
}
// The inverse of a row's sum of exponentials.  A sum of nothing is 0 where the row's own key lies on a page the request does not hold
// (reported in status); where it was seen, every score was -inf, and the softmax of those is not a number.
__device__ __forceinline__ float af_inverse(const AttnF32Args& a, const int* table, int position, float sum) {
    if (sum > 0.f) return 1.0f / sum;
    const int page = table[position / a.page_size];
    return page >= 0 && page < a.num_pages ? NAN : 0.f;
}
__device__ __forceinline__ float af_join(float total, float part, const AfMerge& f) { return __fmaf_rn(part, f.stripe, __fmul_rn(total, f.before)); }

// Rows lane % 8 + 8 i (i < RT) a thread; CT x 4 output columns a thread (d <= 64 CT).
template <int RT, int CT>
__global__ void __launch_bounds__(AF_THREADS, 2) attention_f32_kernel(AttnF32Args a) {
    if (a.overlap) ce_pdl_launch_dependents();
    ce_pdl_wait();
    constexpr int ROWS = 8 * RT;
    extern __shared__ __align__(16) float af_mem[];
    const int d = a.d, pitch = d + 4, d4 = d >> 2;
    float* qs = af_mem;                               // [ROWS][pitch]
    float* ks = qs + ROWS * pitch;                    // [AF_KEYS][pitch]
    float* vs = ks + AF_KEYS * pitch;                 // [AF_KEYS][d]
    float* ss = vs + AF_KEYS * d;                     // [ROWS][AF_SP] scores, then probabilities
    __shared__ long long s_row[AF_KEYS];              // where a chunk's keys lie in the pools, or -1
    __shared__ int s_seen[AF_KEYS];                   // 0: the key's page is not one of the request's
    __shared__ float s_m[ROWS], s_l[ROWS], s_alpha[ROWS];
    __shared__ int s_lo[ROWS], s_hi[ROWS];            // first and last key a row sees (a row that does not exist sees none)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane & 7, ln = lane >> 3;
    const int kvh = blockIdx.y;
    int b = blockIdx.x, q0 = 0;
    if (a.tiles) {
        const int subs = (AF_TILE + a.tokens - 1) / a.tokens, i = blockIdx.x / subs;
        b = a.tiles[2 * i];
        const int off = (blockIdx.x % subs) * a.tokens;
        q0 = a.tiles[2 * i + 1] + off;
    }
    const int t_seq = a.q_start[b], n = a.q_start[b + 1] - t_seq;
    int n_tok = min(a.tokens, n - q0);
    if (a.tiles) n_tok = min(n_tok, AF_TILE - (q0 % AF_TILE));
    if (n_tok <= 0) return;                           // (the same in every block of a cluster)
    const int t0 = t_seq + q0, rows = n_tok * a.group;
    const int* table = a.block_table + (size_t)a.seq_slot[b] * a.max_pages;

    if (tid < ROWS) {
        const int p = tid < rows ? a.positions[t0 + tid / a.group] : -1;
        s_hi[tid] = p;
        s_lo[tid] = a.window > 0 ? max(0, p - a.window + 1) : 0;
        s_m[tid] = -INFINITY;
        s_l[tid] = 0.f;
    }
    for (int e = tid; e < ROWS * d4; e += AF_THREADS) {
        const int r = e / d4, c = (e % d4) * 4;
        const bool in = r < rows;
        af_cp16(qs + r * pitch + c, in ? a.q + (size_t)(t0 + r / a.group) * a.q_stride + (size_t)(kvh * a.group + r % a.group) * d + c : a.q, in);
    }
    __syncthreads();
    const int first = s_lo[0], last = s_hi[rows - 1];            // (a sequence's positions ascend)
    const int c_first = first / AF_KEYS, c_last = last / AF_KEYS;

    auto page_of = [&](int c) {                       // the page of a thread's key of chunk c (beyond the visible ones: none)
        const int key = c * AF_KEYS + tid;
        return c >= 0 && tid < AF_KEYS && key >= first && key <= last ? table[key / a.page_size] : INT_MIN;
    };
    auto set_row = [&](int c, int page) {
        if (tid >= AF_KEYS) return;
        const int key = c * AF_KEYS + tid;
        long long row = -1;
        if (page != INT_MIN) {
            if (page < 0 || page >= a.num_pages) atomicExch(a.status, 4);
            else row = (((long long)page * a.nkv + kvh) * a.page_size + key % a.page_size) * d;
        }
        s_row[tid] = row;
    };
    auto copy = [&](float* dst, int ld, const float* pool) {
        for (int e = tid; e < AF_KEYS * d4; e += AF_THREADS) {
            const int r = e / d4, c = (e % d4) * 4;
            const long long row = s_row[r];
            af_cp16(dst + r * ld + c, row >= 0 ? pool + row + c : pool, row >= 0);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float2 o[RT][2 * CT];                             // this stripe's outputs
    float M[RT], L[RT];                               // the stripes merged so far (walking them all)
    float2 total[RT][2 * CT];
    const int cg = warp * 4 + ln;                     // columns cg * 4 + 64 j
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        M[i] = -INFINITY;
        L[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 2 * CT; ++j) o[i][j] = total[i][j] = make_float2(0.f, 0.f);
    }
    // the chunks in the order of the walk: stripe after stripe, or this block's stripe alone
    auto first_of = [&](int s) { return c_first + ((s - c_first) & (AF_STRIPES - 1)); };
    int stripe = a.stripes_apart ? (int)blockIdx.z : 0;
    const int stripe_end = a.stripes_apart ? stripe + 1 : AF_STRIPES;
    while (stripe < stripe_end && first_of(stripe) > c_last) ++stripe;
    int c = stripe < stripe_end ? first_of(stripe) : -1;
    if (c >= 0) {
        set_row(c, page_of(c));
        __syncthreads();
        copy(ks, pitch, a.k_pool);
        copy(vs, d, a.v_pool);
    }
    while (c >= 0) {
        int next = c + AF_STRIPES, next_stripe = stripe;
        if (next > c_last) {
            ++next_stripe;
            while (next_stripe < stripe_end && first_of(next_stripe) > c_last) ++next_stripe;
            next = next_stripe < stripe_end ? first_of(next_stripe) : -1;
        }
        if (tid < AF_KEYS) s_seen[tid] = s_row[tid] >= 0;
        const int next_page = page_of(next);                       // on its way while the scores are taken
        asm volatile("cp.async.wait_group 1;" ::: "memory");       // the keys (and the queries) are here; the values may still travel
        __syncthreads();
        {   // scores: rows lm + 8 i, keys warp * 16 + ln + 4 j
            float2 s[RT][4];
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = make_float2(0.f, 0.f);
            const float* kp = ks + (warp * 16 + ln) * pitch;
            const float* qp = qs + lm * pitch;
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                float4 k[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(kp + 4 * j * pitch + e);
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const float4 x = *reinterpret_cast<const float4*>(qp + 8 * i * pitch + e);
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = __ffma2_rn(make_float2(x.x, x.y), make_float2(k[j].x, k[j].y), s[i][j]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = __ffma2_rn(make_float2(x.z, x.w), make_float2(k[j].z, k[j].w), s[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) ss[(lm + 8 * i) * AF_SP + warp * 16 + ln + 4 * j] = (s[i][j].x + s[i][j].y) * a.scale;
        }
        if (next >= 0) set_row(next, next_page);
        __syncthreads();
        // the keys' buffer is free; an empty group stands for the copy of a walk's end, so that the waits count alike
        if (next >= 0) copy(ks, pitch, a.k_pool);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        {   // softmax: a warp takes every fourth row, a lane keys lane and lane + 32; the rows' butterflies travel together
            float p0[2 * RT], p1[2 * RT], top[2 * RT], sum[2 * RT], was[2 * RT];
            const int key = c * AF_KEYS + lane;
            const bool seen0 = s_seen[lane], seen1 = s_seen[lane + 32];
#pragma unroll
            for (int i = 0; i < 2 * RT; ++i) {
                const int r = warp + 4 * i, lo = s_lo[r], hi = s_hi[r];
                p0[i] = key >= lo && key <= hi && seen0 ? ss[r * AF_SP + lane] : -INFINITY;
                p1[i] = key + 32 >= lo && key + 32 <= hi && seen1 ? ss[r * AF_SP + lane + 32] : -INFINITY;
                top[i] = fmaxf(p0[i], p1[i]);
                was[i] = s_m[r];
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < 2 * RT; ++i) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], w));
#pragma unroll
            for (int i = 0; i < 2 * RT; ++i) {
                const int r = warp + 4 * i;
                top[i] = fmaxf(was[i], top[i]);
                const float use = top[i] == -INFINITY ? 0.f : top[i];
                p0[i] = expf(p0[i] - use);
                p1[i] = expf(p1[i] - use);
                was[i] = expf(was[i] - use);
                sum[i] = p0[i] + p1[i];
                ss[r * AF_SP + lane] = p0[i];
                ss[r * AF_SP + lane + 32] = p1[i];
            }
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
#pragma unroll
                for (int i = 0; i < 2 * RT; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], w);
            if (lane == 0)
#pragma unroll
                for (int i = 0; i < 2 * RT; ++i) {
                    const int r = warp + 4 * i;
                    s_alpha[r] = was[i];
                    s_m[r] = top[i];
                    s_l[r] = __fmaf_rn(s_l[r], was[i], sum[i]);
                }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");       // the values are here
        __syncthreads();
        {   // outputs: rows lm + 8 i, columns cg * 4 + 64 j; a key a row does not see adds nothing, whatever its value row holds
            int lo[RT], hi[RT];
            bool whole = true;
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int r = lm + 8 * i;
                const float alpha = s_alpha[r];
                lo[i] = s_lo[r] - c * AF_KEYS;
                hi[i] = s_hi[r] - c * AF_KEYS;
                whole = whole && (r >= rows || (lo[i] <= 0 && hi[i] >= AF_KEYS - 1));
#pragma unroll
                for (int j = 0; j < 2 * CT; ++j) o[i][j] = __fmul2_rn(o[i][j], make_float2(alpha, alpha));
            }
            auto keys = [&](auto masked) {
#pragma unroll(RT == 1 ? 4 : 2)
                for (int kk = 0; kk < AF_KEYS; kk += 4) {
                    float4 p[RT];
#pragma unroll
                    for (int i = 0; i < RT; ++i) p[i] = *reinterpret_cast<const float4*>(ss + (lm + 8 * i) * AF_SP + kk);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float4 v[CT];
#pragma unroll
                        for (int j = 0; j < CT; ++j) {
                            const int col = cg * 4 + 64 * j;
                            v[j] = col < d ? *reinterpret_cast<const float4*>(vs + (kk + u) * d + col) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
#pragma unroll
                        for (int i = 0; i < RT; ++i) {
                            const float pu = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                            if (!decltype(masked)::value || (kk + u >= lo[i] && kk + u <= hi[i])) {
#pragma unroll
                                for (int j = 0; j < CT; ++j) {
                                    o[i][2 * j] = __ffma2_rn(make_float2(pu, pu), make_float2(v[j].x, v[j].y), o[i][2 * j]);
                                    o[i][2 * j + 1] = __ffma2_rn(make_float2(pu, pu), make_float2(v[j].z, v[j].w), o[i][2 * j + 1]);
                                }
                            }
                        }
                    }
                }
            };
            if (__all_sync(0xffffffffu, whole)) keys(std::false_type{});
            else keys(std::true_type{});
        }
        __syncthreads();
        if (next >= 0) copy(vs, d, a.v_pool);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        if (!a.stripes_apart && next_stripe != stripe) {            // the stripe joins the ones before it
            __syncthreads();                                       // (s_m and s_l are read below and set back by other threads)
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const int r = lm + 8 * i;
                const AfMerge f = af_merge(M[i], s_m[r]);
                L[i] = af_join(L[i], s_l[r], f);
#pragma unroll
                for (int j = 0; j < 2 * CT; ++j) {
                    total[i][j] = make_float2(af_join(total[i][j].x, o[i][j].x, f), af_join(total[i][j].y, o[i][j].y, f));
                    o[i][j] = make_float2(0.f, 0.f);
                }
            }
            __syncthreads();
            if (tid < ROWS) { s_m[tid] = -INFINITY; s_l[tid] = 0.f; }
        }
        c = next;
        stripe = next_stripe;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!a.stripes_apart) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const int r = lm + 8 * i;
            if (r >= rows) continue;
            const float inv = af_inverse(a, table, s_hi[r], L[i]);
            float* out = a.out + ((size_t)(t0 + r / a.group) * a.nh + kvh * a.group + r % a.group) * d;
#pragma unroll
            for (int j = 0; j < CT; ++j) {
                const int col = cg * 4 + 64 * j;
                if (col < d)
                    *reinterpret_cast<float4*>(out + col) = make_float4(__fmul_rn(total[i][2 * j].x, inv), __fmul_rn(total[i][2 * j].y, inv),
                                                                        __fmul_rn(total[i][2 * j + 1].x, inv), __fmul_rn(total[i][2 * j + 1].y, inv));
            }
        }
        return;
    }
    // the stripes lie in the blocks' shared memory (the keys' buffer is free): every block merges a share of the elements
    __syncthreads();
    float* so = ks;                                   // [ROWS][d]
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) {
            const int col = cg * 4 + 64 * j;
            if (col < d)
                *reinterpret_cast<float4*>(so + (lm + 8 * i) * d + col) = make_float4(o[i][2 * j].x, o[i][2 * j].y, o[i][2 * j + 1].x, o[i][2 * j + 1].y);
        }
    af_cluster_sync();
    const int items = rows * d, per = (items + AF_STRIPES - 1) / AF_STRIPES, stop = min(items, ((int)blockIdx.z + 1) * per);
    for (int e = blockIdx.z * per + tid; e < stop; e += AF_THREADS) {
        const int r = e / d, col = e % d;
        float m[AF_STRIPES], l[AF_STRIPES], x[AF_STRIPES];
#pragma unroll
        for (int s = 0; s < AF_STRIPES; ++s) {
            m[s] = af_ld_cluster(s_m + r, s);
            l[s] = af_ld_cluster(s_l + r, s);
            x[s] = af_ld_cluster(so + r * d + col, s);
        }
        float top = -INFINITY, sum = 0.f, acc = 0.f;
#pragma unroll
        for (int s = 0; s < AF_STRIPES; ++s) {
            const AfMerge f = af_merge(top, m[s]);
            sum = af_join(sum, l[s], f);
            acc = af_join(acc, x[s], f);
        }
        const float inv = af_inverse(a, table, s_hi[r], sum);
        a.out[((size_t)(t0 + r / a.group) * a.nh + kvh * a.group + r % a.group) * d + col] = __fmul_rn(acc, inv);
    }
    af_cluster_sync();                                // no block's stripe goes away while another may still read it
}

template <int RT, int CT>
int af_launch(AttnF32Args a, int blocks, bool apart, cudaStream_t stream) {
    if (blocks == 0) return CE_OK;
    const size_t smem = sizeof(float) * ((size_t)(8 * RT + AF_KEYS) * (a.d + 4) + (size_t)AF_KEYS * a.d + (size_t)8 * RT * AF_SP);
    cudaError_t e;
    static std::atomic<unsigned long long> allowed{0};
    constexpr size_t most = sizeof(float) * ((size_t)(8 * RT + AF_KEYS) * (64 * CT + 4) + (size_t)AF_KEYS * 64 * CT + (size_t)8 * RT * AF_SP);
    e = ce_allow_smem(allowed, attention_f32_kernel<RT, CT>, most);        // (for the largest head size of the instantiation)
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_attention_f32: %s", cudaGetErrorString(e));
    a.stripes_apart = apart && (long long)blocks * a.nkv < 2 * ce_sm_count();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, a.nkv, a.stripes_apart ? AF_STRIPES : 1);
    cfg.blockDim = dim3(AF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    a.overlap = 1;
    if (a.stripes_apart) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = AF_STRIPES;
        cfg.numAttrs = 1;
        cfg.dynamicSmemBytes = most;                             // (one answer for all head sizes)
        static CeRoom room;
        const int at_once = ce_clusters_at_once(room, attention_f32_kernel<RT, CT>, cfg);
        cfg.dynamicSmemBytes = smem;
        a.overlap = (long long)blocks * a.nkv <= at_once;        // see ce_clusters_at_once
        if (at_once == 0) {                                      // (no room for a cluster: the same sums in one block)
            a.stripes_apart = 0;
            a.overlap = 1;
            cfg.gridDim.z = 1;
            cfg.numAttrs = 0;
        }
    }
    if (a.overlap && ce_pdl_enabled()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    ce_note(a.stripes_apart ? "attention_f32_kernel (stripes in a cluster)" : "attention_f32_kernel");
    e = cudaLaunchKernelEx(&cfg, attention_f32_kernel<RT, CT>, a);
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_attention_f32: %s", cudaGetErrorString(e));
    return ce_check_launch("ce_attention_f32");
}

// apart: the stripes may be dealt to clusters (they are while the blocks would not fill the chip)
int af_pick(AttnF32Args a, int rows, int blocks, bool apart, cudaStream_t stream) {
    if (rows <= 8) return a.d <= 64 ? af_launch<1, 1>(a, blocks, apart, stream) : af_launch<1, 2>(a, blocks, apart, stream);
    return a.d <= 64 ? af_launch<4, 1>(a, blocks, apart, stream) : af_launch<4, 2>(a, blocks, apart, stream);
}

}  // namespace

// Heads of up to 128 elements (a multiple of 4), up to 32 query heads a KV head.
extern "C" int ce_attention_f32_supported(int nh, int nkv, int d, int q_stride) {
    return nkv > 0 && nh % nkv == 0 && nh / nkv <= 32 && nkv <= 65535 && d >= 4 && d <= 128 && d % 4 == 0 && q_stride % 4 == 0;
}

// The first n_decode sequences of the step bring one token each; tiles: (sequence, first token) pairs that cover the others 64
// tokens at a time; max_ctx: the longest of those others, its new tokens included.
extern "C" int ce_attention_f32(const float* q, const float* k_pool, const float* v_pool, float* out, const int* positions,
                                const int* seq_slot, const int* q_start, const int* block_table, const int* tiles, int* status,
                                int n_decode, int n_tiles, int nh, int nkv, int d, int q_stride, int page_size, int max_pages,
                                int num_pages, int window, int max_ctx, float scale, cudaStream_t stream) {
    if (n_decode == 0 && n_tiles == 0) return CE_OK;
    if (!q || !k_pool || !v_pool || !out || !positions || !seq_slot || !q_start || !block_table || !status || (n_tiles > 0 && !tiles))
        return ce_fail(CE_ERR_ARG, "ce_attention_f32: null pointer");
    if (!ce_attention_f32_supported(nh, nkv, d, q_stride) || (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15))
        return ce_fail(CE_ERR_SIZE, "ce_attention_f32: %d and %d heads of %d, row stride %d", nh, nkv, d, q_stride);
    AttnF32Args a{q, k_pool, v_pool, out, positions, seq_slot, q_start, block_table, nullptr, status, nh, nkv, d, q_stride, page_size,
                  max_pages, num_pages, window, nh / nkv, 1, 0, 1, scale};
    int rc = af_pick(a, a.group, n_decode, true, stream);
    if (rc) return rc;
    a.tiles = tiles;
    a.tokens = 32 / a.group;
    // Portions whose keys are at most a chunk a stripe gain nothing from a cluster, most of whose blocks would find no key (150 tokens:
    // 30 us in one block, 60 us in clusters; 20 tokens after 3,000: 461 and 78 us).
    return af_pick(a, a.tokens * a.group, n_tiles * ((AF_TILE + a.tokens - 1) / a.tokens), (window > 0 ? min(window, max_ctx) : max_ctx) > AF_KEYS * AF_STRIPES, stream);
}
