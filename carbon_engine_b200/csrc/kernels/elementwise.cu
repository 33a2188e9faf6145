// Memory-bound kernels of a decoder step: embedding gather, RMSNorm, the fused per-head
// q/k norm + rotary embedding + paged K/V write, the residual add and SwiGLU.
//
// The residual stream is float32 in both precisions; norms, rotation and SiLU are computed in
// float32 and rounded once at the store.  The reference gets these ops from its tensor library
// one by one (src/model/layers.rs:140-146 rms_norm, :315-325 rope, :151 silu,
// src/model/mod.rs:781-784 embedding gather, src/kvcache/mod.rs:371-372 K/V scatter).
#include "common.cuh"

// ---------------------------------------------------------------------------------------------
// Embedding: x[t, :] = float(table[token[t], :]) * scale
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void embed_kernel(const T* __restrict__ table, const int* __restrict__ tokens,
                             float* __restrict__ x, int H, int V, int* __restrict__ status, float scale) {
    ce_pdl_begin();
    int t = blockIdx.x;
    int tok = tokens[t];
    if (tok < 0 || tok >= V) {
        if (threadIdx.x == 0) atomicExch(status, 1);
        for (int j = threadIdx.x; j < H; j += blockDim.x) x[(size_t)t * H + j] = 0.f;
        return;
    }
    const T* row = table + (size_t)tok * H;
#pragma unroll 4
    for (int j = threadIdx.x; j < H; j += blockDim.x) x[(size_t)t * H + j] = CeType<T>::load(row + j) * scale;
}

extern "C" int ce_embed(const void* table, int dtype, const int* tokens, float* x, int T, int H, int V,
                        int* status, float scale, cudaStream_t stream) {
    if (T == 0) return CE_OK;
    if (!table || !tokens || !x || !status) return ce_fail(CE_ERR_ARG, "ce_embed: null pointer");
    if (dtype == CE_F32)
        { ce_note("embed_kernel"); ce_launch(embed_kernel<float>, T, H >= 1024 ? 1024 : 256, 0, stream, (const float*)table, tokens, x, H, V, status, scale); }
    else if (dtype == CE_BF16)
        { ce_note("embed_kernel"); ce_launch(embed_kernel<__nv_bfloat16>, T, H >= 1024 ? 1024 : 256, 0, stream, (const __nv_bfloat16*)table, tokens, x, H, V, status, scale); }
    else
        return ce_fail(CE_ERR_ARG, "ce_embed: unknown dtype %d", dtype);
    return ce_check_launch("ce_embed");
}

// ---------------------------------------------------------------------------------------------
// Embedding gather with a norm: x[t, :] = v / sqrt(mean(v^2) + eps) * w,  v = table[tok[t], :] * scale.  xb (or null) receives
// the row rounded to bfloat16 too, for a sublayer that reads the residual itself.
// ---------------------------------------------------------------------------------------------
#define EN_MAX 4
template <typename T, bool VEC>
__global__ void embed_norm_kernel(const T* __restrict__ table, const int* __restrict__ tokens, const float* __restrict__ w,
                                  float* __restrict__ x, __nv_bfloat16* __restrict__ xb, int H, int V, int* status, float scale, float eps) {
    ce_pdl_begin();
    __shared__ float scratch[32];
    int t = blockIdx.x, tok = tokens[t];
    const bool there = tok >= 0 && tok < V;
    if (!there && threadIdx.x == 0) atomicExch(status, 1);
    const T* row = table + (size_t)(there ? tok : 0) * H;
    if (VEC) {                           // four elements at a time, the row in registers
        const int H4 = H >> 2;
        float4 v[EN_MAX];
        float ss = 0.f;
#pragma unroll
        for (int n = 0; n < EN_MAX; ++n) {
            int j = threadIdx.x + n * blockDim.x;
            v[n] = j < H4 ? ce_load4(row + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[n].x *= scale; v[n].y *= scale; v[n].z *= scale; v[n].w *= scale;
            ss += (v[n].x * v[n].x + v[n].y * v[n].y) + (v[n].z * v[n].z + v[n].w * v[n].w);
        }
        const float inv = there ? 1.0f / sqrtf(ce_block_sum(ss, scratch) / (float)H + eps) : 0.f;
#pragma unroll
        for (int n = 0; n < EN_MAX; ++n) {
            int j = threadIdx.x + n * blockDim.x;
            if (j >= H4) continue;
            const float4 ww = ce_load4(w + 4 * j);
            const float4 o = make_float4(v[n].x * inv * ww.x, v[n].y * inv * ww.y, v[n].z * inv * ww.z, v[n].w * inv * ww.w);
            *reinterpret_cast<float4*>(x + (size_t)t * H + 4 * j) = o;
            if (xb) {
                __nv_bfloat162 lo = __floats2bfloat162_rn(o.x, o.y), hi = __floats2bfloat162_rn(o.z, o.w);
                *reinterpret_cast<uint2*>(xb + (size_t)t * H + 4 * j) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
        }
        return;
    }
    float ss = 0.f;
    for (int j = threadIdx.x; j < H; j += blockDim.x) { float v = CeType<T>::load(row + j) * scale; ss = fmaf(v, v, ss); }
    float inv = 1.0f / sqrtf(ce_block_sum(ss, scratch) / (float)H + eps);
    for (int j = threadIdx.x; j < H; j += blockDim.x) {
        float v = there ? CeType<T>::load(row + j) * scale * inv * w[j] : 0.f;
        x[(size_t)t * H + j] = v;
        if (xb) xb[(size_t)t * H + j] = __float2bfloat16_rn(v);
    }
}

template <typename T>
static void embed_norm_launch(const T* table, const int* tokens, const float* w, float* x, __nv_bfloat16* xb, int n, int H, int V, int* status,
                              float scale, float eps, cudaStream_t stream) {
    const int H4 = H / 4, vt = H4 >= 2048 ? 1024 : H4 >= 512 ? 512 : H4 >= 256 ? 256 : 128;
    if (H % 4 == 0 && H4 <= vt * EN_MAX && ((((uintptr_t)table | (uintptr_t)w | (uintptr_t)x | (uintptr_t)xb) & 15) == 0))
        ce_launch(embed_norm_kernel<T, true>, n, vt, 0, stream, table, tokens, w, x, xb, H, V, status, scale, eps);
    else
        ce_launch(embed_norm_kernel<T, false>, n, H >= 1024 ? 1024 : 256, 0, stream, table, tokens, w, x, xb, H, V, status, scale, eps);
}

extern "C" int ce_embed_norm(const void* table, int dtype, const int* tokens, const float* w, float* x, void* xb, int T, int H, int V,
                             int* status, float scale, float eps, cudaStream_t stream) {
    if (T == 0) return CE_OK;
    if (!table || !tokens || !w || !x || !status) return ce_fail(CE_ERR_ARG, "ce_embed_norm: null pointer");
    if (H <= 0 || V <= 0) return ce_fail(CE_ERR_SIZE, "ce_embed_norm: width %d, vocabulary %d", H, V);
    ce_note("embed_norm_kernel");
    if (dtype == CE_F32) embed_norm_launch((const float*)table, tokens, w, x, (__nv_bfloat16*)xb, T, H, V, status, scale, eps, stream);
    else if (dtype == CE_BF16) embed_norm_launch((const __nv_bfloat16*)table, tokens, w, x, (__nv_bfloat16*)xb, T, H, V, status, scale, eps, stream);
    else return ce_fail(CE_ERR_ARG, "ce_embed_norm: unknown dtype %d", dtype);
    return ce_check_launch("ce_embed_norm");
}

// ---------------------------------------------------------------------------------------------
// RMSNorm over the last dimension: out[r, :] = x[row(r), :] * (1/sqrt(mean(x^2) + eps)) * w
// One block of 256 threads per row, so the order of the sum depends on the width only.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w, T* __restrict__ out,
                               const int* __restrict__ rows, int H, float eps) {
    ce_pdl_begin();
    __shared__ float scratch[32];
    int r = blockIdx.x;
    const float* xr = x + (size_t)(rows ? rows[r] : r) * H;
    float ss = 0.f;
    for (int j = threadIdx.x; j < H; j += blockDim.x) {
        float v = xr[j];
        ss = fmaf(v, v, ss);
    }
    ss = ce_block_sum(ss, scratch);
    float inv = 1.0f / sqrtf(ss / (float)H + eps);
    T* o = out + (size_t)r * H;
    for (int j = threadIdx.x; j < H; j += blockDim.x) CeType<T>::store(o + j, xr[j] * inv * w[j]);
}

// The same for widths that are multiples of 4 and at most 4 * 4 * blockDim: every thread keeps its
// float4 elements in registers, so the row is read once and all loads are in flight together.
// four consecutive outputs as one store (the row starts on a 16-byte boundary: H is a multiple of 4)
__device__ __forceinline__ void store4(float* p, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, float a, float b, float c, float d) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    uint2 r;
    r.x = *reinterpret_cast<uint32_t*>(&lo); r.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = r;
}

template <typename T>
__global__ void __launch_bounds__(1024) rmsnorm_vec_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                          T* __restrict__ out, const int* __restrict__ rows, int H,
                                                          float eps) {
    ce_pdl_launch_dependents();          // the weights (and the row list) do not depend on the kernel before
    __shared__ float scratch[32];
    int r = blockIdx.x, n4 = H >> 2;
    const float4* wr = reinterpret_cast<const float4*>(w);
    float4 v[4], g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int j = threadIdx.x + i * blockDim.x;
        g[i] = j < n4 ? wr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)(rows ? rows[r] : r) * H);
    ce_pdl_wait();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int j = threadIdx.x + i * blockDim.x;
        v[i] = j < n4 ? xr[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ss = fmaf(v[i].x, v[i].x, ss); ss = fmaf(v[i].y, v[i].y, ss);
        ss = fmaf(v[i].z, v[i].z, ss); ss = fmaf(v[i].w, v[i].w, ss);
    }
    ss = ce_block_sum(ss, scratch);
    float inv = 1.0f / sqrtf(ss / (float)H + eps);
    T* o = out + (size_t)r * H;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int j = threadIdx.x + i * blockDim.x;
        if (j < n4) store4(o + 4 * j, v[i].x * inv * g[i].x, v[i].y * inv * g[i].y, v[i].z * inv * g[i].z, v[i].w * inv * g[i].w);
    }
}

// Threads per row of the vector kernel: a function of the width only, so that the order of the sum
// never depends on the batch.  0: use the scalar kernel.
static int rmsnorm_vec_threads(int H, const void* x, const void* w, const void* out) {
    if (H % 4 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15)) return 0;
    int n4 = H / 4;
    int threads = ((n4 + 3) / 4 + 31) / 32 * 32;       // four float4 per thread where possible
    if (threads < 128) threads = 128;
    if (threads > 1024) return 0;
    return threads;
}

extern "C" int ce_rmsnorm(const float* x, const float* w, void* out, int out_dtype, const int* rows, int R, int H,
                          float eps, cudaStream_t stream) {
    if (R == 0) return CE_OK;
    if (!x || !w || !out) return ce_fail(CE_ERR_ARG, "ce_rmsnorm: null pointer");
    if (H <= 0) return ce_fail(CE_ERR_SIZE, "ce_rmsnorm: width %d", H);
    int vt = rmsnorm_vec_threads(H, x, w, out);
    if (out_dtype == CE_F32) {
        if (vt) { ce_note("rmsnorm_vec_kernel"); ce_launch(rmsnorm_vec_kernel<float>, R, vt, 0, stream, x, w, (float*)out, rows, H, eps); }
        else { ce_note("rmsnorm_kernel"); ce_launch(rmsnorm_kernel<float>, R, 256, 0, stream, x, w, (float*)out, rows, H, eps); }
    } else if (out_dtype == CE_BF16) {
        if (vt) { ce_note("rmsnorm_vec_kernel"); ce_launch(rmsnorm_vec_kernel<__nv_bfloat16>, R, vt, 0, stream, x, w, (__nv_bfloat16*)out, rows, H, eps); }
        else { ce_note("rmsnorm_kernel"); ce_launch(rmsnorm_kernel<__nv_bfloat16>, R, 256, 0, stream, x, w, (__nv_bfloat16*)out, rows, H, eps); }
    } else
        return ce_fail(CE_ERR_ARG, "ce_rmsnorm: unknown dtype %d", out_dtype);
    return ce_check_launch("ce_rmsnorm");
}

// ---------------------------------------------------------------------------------------------
// Per-head q/k RMSNorm, rotary embedding, and the write of K and V into the paged cache.
//
// Input  qkv [T, (nh + 2*nkv) * d]: q heads, then k heads, then v heads (one GEMM output).
// q heads are normalised and rotated in place.  k heads are normalised, rotated and stored at
// the token's place in the K pool; v heads are copied to the V pool.  Pools are
// [num_pages, nkv, page_size, d].  A token's place is found from its sequence's block-table row:
// page = table[slot, pos / page_size], offset = pos % page_size.
//
// Order follows the reference: norm over the head (weight shared by all heads) BEFORE the
// rotation (src/model/attention.rs:884-889); rotate-half pairing (i, i + rd/2)
// (src/model/layers.rs:159, spelled out in src/kernels/qsa.cu:107-116), or, as a parameter for other
// position encodings, the interleaved pairing (2i, 2i + 1); K is stored after norm and
// rotation, V as projected (src/model/attention.rs:890).
// ---------------------------------------------------------------------------------------------
struct QkRopeArgs {
    void* qkv;
    void* k_pool;
    void* v_pool;
    const float* q_weight;   // [d] or null: no q norm
    const float* k_weight;   // [d] or null: no k norm
    const float* cos_table;  // [max_pos, rd/2] or null: no rotation
    const float* sin_table;
    const int* positions;    // [T]
    const int* seq_of_token; // [T]
    const int* seq_slot;     // [B]
    const int* block_table;  // [slots, max_pages]
    int* status;
    int T, nh, nkv, d, rd, page_size, max_pages, num_pages, max_pos, write_kv;
    float eps;
    int pairing;             // partners of a rotation: 0 = (i, i + rd/2) ("rotate-half"), 1 = (2i, 2i + 1) (interleaved)
    int weights_ready;       // no kernel in front writes q_weight and k_weight
};

template <typename T>
__global__ void qk_rope_kvwrite_kernel(QkRopeArgs a) {
    ce_pdl_begin();
    extern __shared__ float sh[];     // d floats + 32 scratch
    float* vals = sh;
    float* scratch = sh + a.d;
    int t = blockIdx.x, hh = blockIdx.y, j = threadIdx.x;
    int d = a.d;
    bool is_q = hh < a.nh, is_k = !is_q && hh < a.nh + a.nkv;
    if (!is_q && !a.write_kv) return;
    T* src = (T*)a.qkv + (size_t)t * (a.nh + 2 * a.nkv) * d + (size_t)hh * d;
    float v = j < d ? CeType<T>::load(src + j) : 0.f;
    int pos = a.positions[t];

    T* dst = nullptr;
    if (is_q) {
        dst = src;
    } else {
        int slot = a.seq_slot[a.seq_of_token[t]];
        int page = a.block_table[(size_t)slot * a.max_pages + pos / a.page_size];
        if (page < 0 || page >= a.num_pages) {
            if (j == 0) atomicExch(a.status, 2);
            return;
        }
        int kvh = is_k ? hh - a.nh : hh - a.nh - a.nkv;
        T* pool = (T*)(is_k ? a.k_pool : a.v_pool);
        dst = pool + (((size_t)page * a.nkv + kvh) * a.page_size + pos % a.page_size) * d;
    }
    if (!is_q && !is_k) {               // V: plain copy
        if (j < d) CeType<T>::store(dst + j, v);
        return;
    }
    const float* w = is_q ? a.q_weight : a.k_weight;
    if (w) {
        float ss = ce_block_sum(v * v, scratch);
        float inv = 1.0f / sqrtf(ss / (float)d + a.eps);
        if (j < d) v = v * inv * w[j];
    }
    if (a.cos_table) {
        if (pos >= a.max_pos) {
            if (j == 0) atomicExch(a.status, 3);
            return;
        }
        if (j < d) vals[j] = v;
        __syncthreads();
        int half = a.rd / 2;
        const float* c = a.cos_table + (size_t)pos * half;
        const float* s = a.sin_table + (size_t)pos * half;
        if (a.pairing == 1) {           // interleaved: elements 2f and 2f + 1 turn by angle f
            if (j < a.rd) {
                int f = j >> 1;
                v = (j & 1) ? vals[j] * c[f] + vals[j - 1] * s[f] : vals[j] * c[f] - vals[j + 1] * s[f];
            }
        } else if (j < half)
            v = vals[j] * c[j] - vals[j + half] * s[j];
        else if (j < a.rd)
            v = vals[j] * c[j - half] + vals[j - half] * s[j - half];
    }
    if (j < d) CeType<T>::store(dst + j, v);
}

// E consecutive elements to and from float, W of them an access
template <typename T, int W> struct alignas(W * sizeof(T)) RopePiece { T e[W]; };
template <int W, typename T, int E>
__device__ __forceinline__ void rope_load(const T* p, float (&v)[E]) {
#pragma unroll
    for (int i = 0; i < E; i += W) {
        const RopePiece<T, W> piece = *reinterpret_cast<const RopePiece<T, W>*>(p + i);
#pragma unroll
        for (int j = 0; j < W; ++j) v[i + j] = CeType<T>::load(piece.e + j);
    }
}
template <int W, typename T, int E>
__device__ __forceinline__ void rope_store(T* p, const float (&v)[E]) {
#pragma unroll
    for (int i = 0; i < E; i += W) {
        RopePiece<T, W> piece;
#pragma unroll
        for (int j = 0; j < W; ++j) CeType<T>::store(piece.e + j, v[i + j]);
        *reinterpret_cast<RopePiece<T, W>*>(p + i) = piece;
    }
}

// The sum over L lanes with S sums each, as over L * S lanes with one (lane S * l + g: sum g of lane l) that add by halves, the lanes
// furthest apart first.  A lane keeps half of its sums at each step, the other half is its partner's, until one is left (128 elements a
// head: 6 shuffles, 12 with all sums kept); additions commute, so both partners' results are the same bits.
template <int L, int S>
__device__ __forceinline__ void rope_sum(float (&ss)[S], int lane) {
    int n = S;
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool upper = lane & o;
#pragma unroll
            for (int g = 0; g < S / 2; ++g)
                if (g < n) ss[g] = (upper ? ss[g + n] : ss[g]) + __shfl_xor_sync(0xffffffffu, upper ? ss[g] : ss[g + n], o);
        } else {
            ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o);
        }
    }
    // the sums that other lanes kept
#pragma unroll
    for (int o = L / 2, m = S; m > n; o >>= 1, m >>= 1)
#pragma unroll
        for (int g = 0; g < S; ++g)
            if (g < n) ss[g] += __shfl_xor_sync(0xffffffffu, ss[g], o);
#pragma unroll
    for (int o = S / 2; o > 0; o >>= 1)
#pragma unroll
        for (int g = 0; g < o; ++g)
            if (o < n) ss[g] += ss[g + o];
}

// Head sizes that are multiples of 64 (up to 256) with a full rotation.  A head belongs to L neighbouring lanes: a lane holds E
// consecutive elements of the head's first half and the E elements d/2 further on, their partners in the rotation, and moves W at a
// time, 16 bytes where the operands start on them (the launcher says which E, L and W); a warp takes 32 / L heads at a time, and nothing
// is exchanged between lanes but the sum of squares.  The token's position, page, cosines and sines are looked up once per warp; a warp
// takes `hpw` consecutive heads of one token, as few as it takes at a time where tokens are few (decoding: as large a grid as can be),
// a quarter of them all in portions of prompts.  A head's arithmetic does not depend on hpw.
// The sum of squares is that of a warp of 32 lanes with d/64 elements of each half: such a lane's terms in order, first half then
// second, and the lanes' sums by halves (lanes 16 apart, 8, 4, 2, 1).  A lane here holds 32 / L of those lanes' sums.
// What bounds a long portion is the memory (2,048 tokens of 32 + 2 x 8 heads of 128: 50 MB in and out); with accesses of 4 bytes a lane it
// was the instructions.  Measured: a prompt of 203 tokens, 12 layers of 8b sizes, 2,306 -> 2,243 us a pass; eight decode steps with this and
// the attention's merge in one trip 10,330 -> 10,040 (one request), 11,440 -> 11,152 (eight).
template <typename T, int E, int L, int W>
__global__ void __launch_bounds__(128) qk_rope_kvwrite_warp_kernel(QkRopeArgs a, int hpw) {
    // positions, slots, block tables, cosines and sines are inputs of the step or constants: they are looked up while the kernel
    // before this one (the QKV product) still runs.  Its output waits for it, and so do norm weights that a kernel may write.
    ce_pdl_launch_dependents();
    constexpr int AT_ONCE = 32 / L, SUMS = 32 / L, TERMS = E / SUMS;
    constexpr int WF = L == 32 ? W : E % 4 ? 2 : 4;              // of the float32 operands
    const int lane = threadIdx.x & 31, sub = lane / L, heads_per_token = a.nh + 2 * a.nkv;
    const int groups = (heads_per_token + hpw - 1) / hpw;
    const long long wg = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (wg >= (long long)a.T * groups) return;
    const int t = (int)(wg / groups), g = (int)(wg - (long long)t * groups);
    const int hh0 = g * hpw;
    int hh1 = min(hh0 + hpw, heads_per_token);
    if (!a.write_kv) hh1 = min(hh1, a.nh);
    if (hh0 >= hh1) return;
    constexpr int half = E * L, d = 2 * half;
    const int e0 = E * (lane % L);
    const int pos = a.positions[t];
    const bool rotate = a.cos_table != nullptr;
    if (rotate && pos >= a.max_pos && hh0 < a.nh + a.nkv) {
        if (lane == 0) atomicExch(a.status, 3);
        return;
    }
    float cs[E], sn[E];
#pragma unroll
    for (int i = 0; i < E; ++i) { cs[i] = 1.f; sn[i] = 0.f; }
    if (rotate && hh0 < a.nh + a.nkv) {
        rope_load<WF>(a.cos_table + (size_t)pos * half + e0, cs);
        rope_load<WF>(a.sin_table + (size_t)pos * half + e0, sn);
    }
    size_t page_row = 0;
    if (hh1 > a.nh) {                      // a K or V head in this group: where the token's row lies in the pools
        int slot = a.seq_slot[a.seq_of_token[t]];
        int page = a.block_table[(size_t)slot * a.max_pages + pos / a.page_size];
        if (page < 0 || page >= a.num_pages) {
            if (lane == 0) atomicExch(a.status, 2);
            return;
        }
        page_row = (size_t)page * a.nkv * a.page_size + pos % a.page_size;
    }
    T* row = (T*)a.qkv + (size_t)t * heads_per_token * d;
    const float inv_d = 1.0f / (float)d;
    float w1[E], w2[E];
    const float* held = nullptr;           // the norm weights in w1 and w2
    auto hold = [&](const float* w) {
        if (!w || w == held) return;
        rope_load<WF>(w + e0, w1);
        rope_load<WF>(w + half + e0, w2);
        held = w;
    };
    auto weights_of = [&](int hh) { return hh < a.nh ? a.q_weight : hh < a.nh + a.nkv ? a.k_weight : nullptr; };
    if (!a.weights_ready) ce_pdl_wait();
    hold(weights_of(hh0 + sub));
    ce_pdl_wait();
    constexpr int U = E > 4 ? 2 : 4;       // heads of a lane in flight together
    for (int hb = hh0; hb < hh1; hb += U * AT_ONCE) {
        float x1[U][E], x2[U][E];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int hh = hb + u * AT_ONCE + sub;
            if (hh < hh1) {
                rope_load<W>(row + (size_t)hh * d + e0, x1[u]);
                rope_load<W>(row + (size_t)hh * d + half + e0, x2[u]);
            } else {
#pragma unroll
                for (int i = 0; i < E; ++i) x1[u][i] = x2[u][i] = 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (hb + u * AT_ONCE >= hh1) break;
            // query heads stay in place, key and value heads go into the pools; values are copied as they are
            const int hh = hb + u * AT_ONCE + sub, kv = hh - a.nh, v = kv - a.nkv;
            const float* w = weights_of(hh);
            hold(w);
            float ss[SUMS];
#pragma unroll
            for (int g = 0; g < SUMS; ++g) {
                ss[g] = 0.f;
#pragma unroll
                for (int i = g * TERMS; i < (g + 1) * TERMS; ++i) ss[g] = fmaf(x1[u][i], x1[u][i], ss[g]);
#pragma unroll
                for (int i = g * TERMS; i < (g + 1) * TERMS; ++i) ss[g] = fmaf(x2[u][i], x2[u][i], ss[g]);
            }
            rope_sum<L>(ss, lane);
            if (hh >= hh1) continue;
            T* dst = kv < 0 ? row + (size_t)hh * d : (T*)(v < 0 ? a.k_pool : a.v_pool) + (page_row + (size_t)(v < 0 ? kv : v) * a.page_size) * d;
            if (w) {
                const float inv = rsqrtf(fmaf(ss[0], inv_d, a.eps));
#pragma unroll
                for (int i = 0; i < E; ++i) { x1[u][i] = x1[u][i] * inv * w1[i]; x2[u][i] = x2[u][i] * inv * w2[i]; }
            }
            if (rotate && v < 0) {
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const float p = x1[u][i], q = x2[u][i];
                    x1[u][i] = p * cs[i] - q * sn[i];
                    x2[u][i] = q * cs[i] + p * sn[i];
                }
            }
            rope_store<W>(dst + e0, x1[u]);
            rope_store<W>(dst + half + e0, x2[u]);
        }
    }
}

// A head's lanes and accesses, and the elements that an operand must start on (0: not a head size of this kernel).  Operands on 16 bytes:
// 4 float32 or 8 bfloat16 elements an access, and in steps of a few tokens, where latency is all, twice the lanes for a bfloat16 head
// of 128 or 256 (one token of 32 + 2 x 8 heads of 128: 1.42 -> 1.35 us; 203 tokens 2.28 -> 2.6); heads of 192, whose lanes must hold whole
// threes, 2.  Other operands: d / 64 elements an access (1 for heads of 192), 32 lanes (2,048 tokens: 14.2 us against 11.6; a block a
// head took 102).
struct RopeForm {
    void (*kernel)(QkRopeArgs, int);
    int lanes, start;
};
template <typename T>
static RopeForm rope_form(int d, bool narrow, bool few) {
    const bool four = sizeof(T) == 4;
    switch (d) {
        case 64:
            if (narrow) return {qk_rope_kvwrite_warp_kernel<T, 1, 32, 1>, 32, 1};
            if (four) return {qk_rope_kvwrite_warp_kernel<T, 4, 8, 4>, 8, 4};
            return {qk_rope_kvwrite_warp_kernel<T, 8, 4, 8>, 4, 8};
        case 128:
            if (narrow) return {qk_rope_kvwrite_warp_kernel<T, 2, 32, 2>, 32, 2};
            if (four || few) return {qk_rope_kvwrite_warp_kernel<T, 4, 16, 4>, 16, 4};
            return {qk_rope_kvwrite_warp_kernel<T, 8, 8, 8>, 8, 8};
        case 192:
            if (narrow) return {qk_rope_kvwrite_warp_kernel<T, 3, 32, 1>, 32, 1};
            return {qk_rope_kvwrite_warp_kernel<T, 6, 16, 2>, 16, 2};
        case 256:
            if (narrow || four || few) return {qk_rope_kvwrite_warp_kernel<T, 4, 32, 4>, 32, 4};
            return {qk_rope_kvwrite_warp_kernel<T, 8, 16, 8>, 16, 8};
    }
    return {nullptr, 32, 1};
}

template <typename T>
static bool launch_rope_warp(const QkRopeArgs& a, cudaStream_t stream) {
    if (a.cos_table && (a.rd != a.d || a.pairing != 0)) return false;
    const uintptr_t rows = (uintptr_t)a.qkv | (uintptr_t)a.k_pool | (uintptr_t)a.v_pool;
    const uintptr_t floats = (uintptr_t)a.q_weight | (uintptr_t)a.k_weight | (uintptr_t)a.cos_table | (uintptr_t)a.sin_table;
    const RopeForm form = rope_form<T>(a.d, (rows | floats) % 16, a.T < 64);
    if (!form.kernel || rows % 16 % (form.start * sizeof(T)) || floats % 16 % (form.start * sizeof(float))) return false;
    const int heads_per_token = a.nh + 2 * a.nkv, at_once = 32 / form.lanes;
    // few tokens: as many warps as there are, while the chip takes them at once; many: four warps share a token's heads
    int hpw = at_once;
    if (a.T >= 256) hpw = ((heads_per_token + 3) / 4 + at_once - 1) / at_once * at_once;
    else
        while (hpw < 4 && (long long)a.T * ((heads_per_token + hpw - 1) / hpw) > 32 * 148) hpw *= 2;
    const long long warps = (long long)a.T * ((heads_per_token + hpw - 1) / hpw);
    if ((warps + 3) / 4 > 2147483647LL) return false;
    ce_note("qk_rope_kvwrite_warp_kernel");
    ce_launch(form.kernel, (unsigned)((warps + 3) / 4), 128, 0, stream, a, hpw);
    return true;
}

extern "C" int ce_qk_rope_kvwrite(void* qkv, void* k_pool, void* v_pool, int dtype, const float* q_weight,
                                  const float* k_weight, const float* cos_table, const float* sin_table,
                                  const int* positions, const int* seq_of_token, const int* seq_slot,
                                  const int* block_table, int* status, int T, int nh, int nkv, int d, int rd,
                                  int page_size, int max_pages, int num_pages, int max_pos, int write_kv, float eps,
                                  int pairing, int weights_ready, cudaStream_t stream) {
    if (T == 0) return CE_OK;
    if (d <= 0 || d > 1024) return ce_fail(CE_ERR_SIZE, "ce_qk_rope_kvwrite: head_dim %d not in 1..1024", d);
    if (rd < 0 || rd > d || (rd & 1)) return ce_fail(CE_ERR_SIZE, "ce_qk_rope_kvwrite: rotary_dim %d must be even and <= head_dim %d", rd, d);
    if (pairing != 0 && pairing != 1) return ce_fail(CE_ERR_ARG, "ce_qk_rope_kvwrite: pairing %d (0: halves, 1: interleaved)", pairing);
    if (!qkv || !positions || !status) return ce_fail(CE_ERR_ARG, "ce_qk_rope_kvwrite: null pointer");
    if (write_kv && (!k_pool || !v_pool || !seq_of_token || !seq_slot || !block_table))
        return ce_fail(CE_ERR_ARG, "ce_qk_rope_kvwrite: cache pointers missing");
    QkRopeArgs a{qkv, k_pool, v_pool, q_weight, k_weight, cos_table, sin_table, positions, seq_of_token, seq_slot,
                 block_table, status, T, nh, nkv, d, rd, page_size, max_pages, num_pages, max_pos, write_kv, eps, pairing,
                 weights_ready};
    int threads = (d + 31) / 32 * 32;
    dim3 grid(T, nh + 2 * nkv);
    size_t smem = (d + 32) * sizeof(float);
    if (dtype == CE_F32) {
        if (!launch_rope_warp<float>(a, stream)) { ce_note("qk_rope_kvwrite_kernel"); ce_launch(qk_rope_kvwrite_kernel<float>, grid, threads, smem, stream, a); }
    } else if (dtype == CE_BF16) {
        if (!launch_rope_warp<__nv_bfloat16>(a, stream))
            { ce_note("qk_rope_kvwrite_kernel"); ce_launch(qk_rope_kvwrite_kernel<__nv_bfloat16>, grid, threads, smem, stream, a); }
    } else
        return ce_fail(CE_ERR_ARG, "ce_qk_rope_kvwrite: unknown dtype %d", dtype);
    return ce_check_launch("ce_qk_rope_kvwrite");
}

// ---------------------------------------------------------------------------------------------
// x += delta (float32 residual, delta in the activation dtype)
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void add_residual_kernel(float* __restrict__ x, const T* __restrict__ delta, size_t n) {
    ce_pdl_begin();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) x[i] += CeType<T>::load(delta + i);
}

extern "C" int ce_add_residual(float* x, const void* delta, int dtype, long long n, cudaStream_t stream) {
    if (n == 0) return CE_OK;
    if (!x || !delta) return ce_fail(CE_ERR_ARG, "ce_add_residual: null pointer");
    int blocks = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    if (dtype == CE_F32)
        { ce_note("add_residual_kernel"); ce_launch(add_residual_kernel<float>, blocks, 256, 0, stream, x, (const float*)delta, (size_t)n); }
    else if (dtype == CE_BF16)
        { ce_note("add_residual_kernel"); ce_launch(add_residual_kernel<__nv_bfloat16>, blocks, 256, 0, stream, x, (const __nv_bfloat16*)delta, (size_t)n); }
    else
        return ce_fail(CE_ERR_ARG, "ce_add_residual: unknown dtype %d", dtype);
    return ce_check_launch("ce_add_residual");
}

// ---------------------------------------------------------------------------------------------
// SwiGLU: out[t, i] = silu(gu[t, i]) * gu[t, I + i], silu(z) = z / (1 + exp(-z))
// (src/model/layers.rs:568, 625-648)
// ---------------------------------------------------------------------------------------------
template <typename T, bool RELU>
__global__ void swiglu_kernel(const T* __restrict__ gu, T* __restrict__ out, int I, size_t total) {
    ce_pdl_begin();
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < total; i += stride) {
        size_t t = i / I, c = i - t * I;
        float g = CeType<T>::load(gu + t * 2 * I + c);
        float u = CeType<T>::load(gu + t * 2 * I + I + c);
        CeType<T>::store(out + i, RELU ? fmaxf(g, 0.f) * u : g / (1.0f + expf(-g)) * u);
    }
}

// relu != 0: out = relu(gate) * up instead
static int gated_act(const void* gu, void* out, int dtype, int T, int I, int relu, cudaStream_t stream) {
    size_t total = (size_t)T * I;
    if (total == 0) return CE_OK;
    if (!gu || !out) return ce_fail(CE_ERR_ARG, "ce_swiglu: null pointer");
    int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    ce_note("swiglu_kernel");
    if (dtype == CE_F32) {
        if (relu) ce_launch(swiglu_kernel<float, true>, blocks, 256, 0, stream, (const float*)gu, (float*)out, I, total);
        else ce_launch(swiglu_kernel<float, false>, blocks, 256, 0, stream, (const float*)gu, (float*)out, I, total);
    } else if (dtype == CE_BF16) {
        if (relu) ce_launch(swiglu_kernel<__nv_bfloat16, true>, blocks, 256, 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, I, total);
        else ce_launch(swiglu_kernel<__nv_bfloat16, false>, blocks, 256, 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, I, total);
    } else
        return ce_fail(CE_ERR_ARG, "ce_swiglu: unknown dtype %d", dtype);
    return ce_check_launch("ce_swiglu");
}

extern "C" int ce_reluglu(const void* gu, void* out, int dtype, int T, int I, cudaStream_t stream) {
    return gated_act(gu, out, dtype, T, I, 1, stream);
}

extern "C" int ce_swiglu(const void* gu, void* out, int dtype, int T, int I, cudaStream_t stream) {
    return gated_act(gu, out, dtype, T, I, 0, stream);
}

// out[t, i] = the clamped gated activation of gu[t, i] + bias[i] and gu[t, I + i] + bias[I + i] (bias float32 [2I] or null)
template <typename T>
__global__ void clamp_glu_kernel(const T* __restrict__ gu, T* __restrict__ out, const float* __restrict__ bias, float limit, float alpha,
                                 int I, size_t total) {
    ce_pdl_begin();
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        size_t t = i / I, c = i - t * I;
        float g = CeType<T>::load(gu + t * 2 * I + c) + (bias ? bias[c] : 0.f);
        float u = CeType<T>::load(gu + t * 2 * I + I + c) + (bias ? bias[I + c] : 0.f);
        CeType<T>::store(out + i, ce_clamp_glu(g, u, limit, alpha));
    }
}

extern "C" int ce_clamp_glu(const void* gu, void* out, int dtype, const float* bias, float limit, float alpha, int T, int I,
                            cudaStream_t stream) {
    size_t total = (size_t)T * I;
    if (total == 0) return CE_OK;
    if (!gu || !out) return ce_fail(CE_ERR_ARG, "ce_clamp_glu: null pointer");
    int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    ce_note("clamp_glu_kernel");
    if (dtype == CE_F32) ce_launch(clamp_glu_kernel<float>, blocks, 256, 0, stream, (const float*)gu, (float*)out, bias, limit, alpha, I, total);
    else if (dtype == CE_BF16) ce_launch(clamp_glu_kernel<__nv_bfloat16>, blocks, 256, 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, bias, limit, alpha, I, total);
    else return ce_fail(CE_ERR_ARG, "ce_clamp_glu: unknown dtype %d", dtype);
    return ce_check_launch("ce_clamp_glu");
}

// out[t, i] = relu(in[t, i])^2: the epilogue of a library product for the activation of the small experts
template <typename T>
__global__ void relu2_kernel(const T* __restrict__ in, T* __restrict__ out, int I, int ldo, size_t total) {
    ce_pdl_begin();
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        size_t t = i / I, c = i - t * I;
        float v = fmaxf(CeType<T>::load(in + i), 0.f);
        CeType<T>::store(out + t * ldo + c, v * v);
    }
}

extern "C" int ce_relu2(const void* in, void* out, int dtype, int T, int I, int ldo, cudaStream_t stream) {
    size_t total = (size_t)T * I;
    if (total == 0) return CE_OK;
    if (!in || !out) return ce_fail(CE_ERR_ARG, "ce_relu2: null pointer");
    int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    ce_note("relu2_kernel");
    if (dtype == CE_F32) ce_launch(relu2_kernel<float>, blocks, 256, 0, stream, (const float*)in, (float*)out, I, ldo, total);
    else if (dtype == CE_BF16) ce_launch(relu2_kernel<__nv_bfloat16>, blocks, 256, 0, stream, (const __nv_bfloat16*)in, (__nv_bfloat16*)out, I, ldo, total);
    else return ce_fail(CE_ERR_ARG, "ce_relu2: unknown dtype %d", dtype);
    return ce_check_launch("ce_relu2");
}

// ---------------------------------------------------------------------------------------------
// dst[idx[i]] = val[i]: applies the block-table entries that changed since the last step.
// ---------------------------------------------------------------------------------------------
__global__ void scatter_i32_kernel(int* __restrict__ dst, const int* __restrict__ idx, const int* __restrict__ val,
                                   int n, long long dst_len) {
    // No early launch of dependents here: block tables are step inputs, and kernels further down the
    // stream read them BEFORE their own wait (the decode attention looks up pages while the kernels
    // before it still run).  Without the early launch the next kernel starts only when these writes are
    // complete, and so does everything after it.
    ce_pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && idx[i] >= 0 && idx[i] < dst_len) dst[idx[i]] = val[i];
}

extern "C" int ce_scatter_i32(int* dst, const int* idx, const int* val, int n, long long dst_len, cudaStream_t stream) {
    if (n == 0) return CE_OK;
    if (!dst || !idx || !val) return ce_fail(CE_ERR_ARG, "ce_scatter_i32: null pointer");
    { ce_note("scatter_i32_kernel"); ce_launch(scatter_i32_kernel, (n + 255) / 256, 256, 0, stream, dst, idx, val, n, dst_len); }
    return ce_check_launch("ce_scatter_i32");
}
