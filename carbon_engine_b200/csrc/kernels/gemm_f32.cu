// y = x * W^T with float32 FMA arithmetic: the matrix product of the float32 path.  No tensor-core instruction and no
// reduced-precision mode is involved.
//
// THE ORDER OF A SUM is a function of K alone, so a token's result does not depend on M, on the tile it falls in, or on its
// neighbours: K is cut into up to 8 runs (at least 256 long, whole multiples of 32), a run is two chains of fused multiply-adds
// (even k and odd k, each in ascending order) that are added at its end, and the runs are added in order.  Two chains, because
// fma.f32x2 then takes its operand pairs (k, k + 1) as they lie in memory, without a move; up to 8 runs, because they are what a
// cluster of blocks shares when a product has few tiles.  (Shorter chains also round less often: against float64 the error of a
// 2,048-long product is about a third of one running sum's.)
//
// What bounds it: many tokens, the FMA pipes; few tokens (decode), reading the weights once.  One kernel, four tiles, all of 128
// weight rows: 64 tokens (8 x 8 results a thread: 16 shared-memory reads of 16 bytes for 128 fma.f32x2), 32 tokens (8 x 4), and 8
// or 4 tokens where a thread holds one weight row and all tokens, whose values are broadcast reads.  Operands come by cp.async into
// a ring of stages of 32 k, rows as they lie in memory with 16-byte chunks swizzled by the row (chunk ^ row & 7), so that the lanes'
// reads meet no bank twice.  Where a product has too few tiles to fill the chip, a cluster of blocks takes a run of K each and adds
// the partial sums through distributed shared memory, in the order above.  Most products of up to 8 tokens with K of 2,048 and more go to
// gemm_f32_stream.cu instead (the same bits); the small tiles here take the others: shorter or odd K, rows off 16 bytes, few or very many
// weight rows (the vocabulary's, whose clusters are more than the chip holds at once).
//
// Measured (us; 1 and 8 tokens of these two go to gemm_f32_stream.cu now; before: 64 x 64 tiles, 4 x 4 results a thread, one stage of 16 k,
// one block a tile over all of K):
//                          12,288 x 2,048 (gate and up)      2,048 x 6,144 (down)
//     1 token                  485 -> 22 (4.5 TB/s)             985 -> 18
//     8 tokens                 495 -> 28                        987 -> 28
//     32 tokens                499 -> 60                        999 -> 51
//     301 tokens               925 -> 448 (34 TFLOP/s)         1234 -> 234 (32 TFLOP/s)
// At 301 tokens the FMA pipes are 61 % busy (an fma.f32x2 holds one for two cycles): 480 tiles on 296 places make a second wave that is
// 0.62 full, and the two warps of a scheduler leave it without a ready one in half of the cycles.  The same tile with twice the warps
// (8 x 4 results a thread) or with scalar fmaf is 5 to 15 % slower.
#include "gemm_f32.cuh"

namespace {

constexpr int FK = 32;                  // k per stage
constexpr int F_ROWS = 128;             // weight rows per tile
constexpr int F_PITCH = F_ROWS + 4;     // of the partial sums' rows: 8 tokens x 4 features a warp meet 32 banks
constexpr int F_THREADS = 128;
constexpr int F_MAX_RUNS = 8;           // runs of K = blocks of a cluster (the portable limit)

struct F32Args {
    const float* A;
    const float* W;
    float* C;
    int M, N, K, lda, ldc, mode;
    int run, splits;                    // k of a run; blocks a tile's runs are dealt to (1, or one a run)
    int weights_ready;                  // no kernel in front writes W
    int overlap;                        // kernels behind may start before this one ends
    GpGate gate;
};

__device__ __forceinline__ uint32_t f_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void f_cp16(uint32_t dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ float f_ld_cluster(uint32_t local, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void f_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Rows [row0, row0 + ROWS) of a matrix, k of one stage, into a swizzled tile; rows and k that do not exist read zeros.
// row_of(r): the matrix row of tile row r, or -1.
template <int ROWS, bool VEC, typename RowOf>
__device__ __forceinline__ void f_load(float* tile, const float* src, long long ld, int k0, int k_end, RowOf row_of) {
    const int tid = threadIdx.x, c = tid & 7;
#pragma unroll
    for (int p = 0; p < (ROWS + F_THREADS / 8 - 1) / (F_THREADS / 8); ++p) {
        const int r = p * (F_THREADS / 8) + (tid >> 3);
        if (ROWS % (F_THREADS / 8) && r >= ROWS) continue;
        const int row = row_of(r), k = k0 + c * 4;
        float* dst = tile + r * FK + ((c ^ (r & 7)) << 2);
        if (VEC) {
            const bool in = row >= 0 && k < k_end;
            f_cp16(f_smem(dst), in ? src + row * ld + k : src, in);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = row >= 0 && k + e < k_end ? src[row * ld + k + e] : 0.f;
        }
    }
}

// TM tokens x TN weight rows a thread, LM lanes of a warp along the tokens (the rest along the rows), four warps along the rows.
// GATED: the tile's rows are 64 gate rows and the 64 up rows of the same features.  VEC: rows of A and W start on 16 bytes and K
// is a multiple of 4; else operands are fetched one by one.
template <int TM, int LM, int TN, bool GATED, bool VEC>
__global__ void __launch_bounds__(F_THREADS, 2) gemm_f32_kernel(F32Args a, int stages) {
    constexpr int LN = 32 / LM, BM = TM * LM, NF = GATED ? F_ROWS / 2 : F_ROWS;
    constexpr int STAGE = (BM + F_ROWS) * FK;
    static_assert(4 * LN * TN == F_ROWS, "four warps share the tile's rows");
    extern __shared__ __align__(16) float f_smem_raw[];
    float* ring = f_smem_raw;
    float* part = f_smem_raw + stages * STAGE;             // [BM][F_PITCH] sums of the runs finished so far
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane % LM, ln = lane / LM;
    const int n0 = blockIdx.x * NF, m0 = blockIdx.y * BM, rank = blockIdx.z;
    const int k_begin = a.splits > 1 ? rank * a.run : 0, k_end = a.splits > 1 ? min(a.K, k_begin + a.run) : a.K;
    const int slabs = (k_end - k_begin + FK - 1) / FK, run_slabs = a.run / FK;
    auto w_row = [&](int r) { int f = n0 + (r & (NF - 1)); return f < a.N ? (GATED && r >= NF ? a.N + f : f) : -1; };
    auto a_row = [&](int r) { return m0 + r < a.M ? m0 + r : -1; };
    auto load_w = [&](int s) { f_load<F_ROWS, VEC>(ring + (s % stages) * STAGE + BM * FK, a.W, a.K, k_begin + s * FK, k_end, w_row); };
    auto load_a = [&](int s) { f_load<BM, VEC>(ring + (s % stages) * STAGE, a.A, a.lda, k_begin + s * FK, k_end, a_row); };

    // weights that no kernel writes come before the wait for the kernels in front; any other W is read after it, like A
    if (a.overlap) ce_pdl_launch_dependents();
    if (!a.weights_ready) ce_pdl_wait();
    for (int s = 0; s < stages - 1; ++s)
        if (s < slabs) load_w(s);
    ce_pdl_wait();
    for (int s = 0; s < stages - 1; ++s) {
        if (s < slabs) load_a(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    float2 acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
    const int wrow0 = warp * (LN * TN) + ln;
    float* mine = part + lm * F_PITCH + wrow0;
    int in_run = 0;
    bool first_run = true;
    for (int s = 0; s < slabs; ++s) {
        if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncthreads();                                   // the stage has landed, and everyone is done with the one before it
        if (s + stages - 1 < slabs) { load_w(s + stages - 1); load_a(s + stages - 1); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* at = ring + (s % stages) * STAGE;
        const float* wt = at + BM * FK;
#pragma unroll(TM * TN >= 64 ? 2 : 8)
        for (int q = 0; q < FK / 4; ++q) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int r = wrow0 + LN * j;
                w[j] = *reinterpret_cast<const float4*>(wt + r * FK + ((q ^ (r & 7)) << 2));
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const int r = lm + LM * i;
                const float4 x = *reinterpret_cast<const float4*>(at + r * FK + ((q ^ (r & 7)) << 2));
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(x.x, x.y), make_float2(w[j].x, w[j].y), acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(x.z, x.w), make_float2(w[j].z, w[j].w), acc[i][j]);
            }
        }
        if (++in_run == run_slabs || s + 1 == slabs) {     // a run is complete: its sum joins the ones before it
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float* p = mine + LM * i * F_PITCH + LN * j;
                    const float v = acc[i][j].x + acc[i][j].y;
                    *p = first_run ? v : *p + v;
                    acc[i][j] = make_float2(0.f, 0.f);
                }
            in_run = 0;
            first_run = false;
        }
    }
    if (a.splits > 1) f_cluster_sync();
    else __syncthreads();
    // the epilogue: the blocks of a cluster share the tile's results
    const int items = min(BM, a.M - m0) * NF, per = (items + a.splits - 1) / a.splits, stop = min(items, (rank + 1) * per);
    auto total = [&](int at) {
        if (a.splits == 1) return part[at];
        const uint32_t local = f_smem(part + at);
        float v[F_MAX_RUNS];
#pragma unroll
        for (int r = 0; r < F_MAX_RUNS; ++r) v[r] = r < a.splits ? f_ld_cluster(local, r) : 0.f;
        float sum = v[0];
#pragma unroll
        for (int r = 1; r < F_MAX_RUNS; ++r)
            if (r < a.splits) sum += v[r];
        return sum;
    };
    for (int item = rank * per + tid; item < stop; item += F_THREADS) {
        const int m = item / NF, f = item % NF, n = n0 + f;
        if (n >= a.N) continue;
        float v = total(m * F_PITCH + f);
        float* out = a.C + (size_t)(m0 + m) * a.ldc + n;
        if (GATED) {
            float u = total(m * F_PITCH + NF + f);
            if (a.mode == GP_CLAMPGLU) {
                if (a.gate.bias) { v += a.gate.bias[n]; u += a.gate.bias[a.N + n]; }
                *out = ce_clamp_glu(v, u, a.gate.limit, a.gate.alpha);
            } else {
                *out = a.mode == GP_RELUGLU ? fmaxf(v, 0.f) * u : ce_silu_glu(v, u);
            }
        } else if (a.mode == GP_ACCUM_F32) {
            *out += v;
        } else if (a.mode == GP_RELU2) {
            const float r = fmaxf(v, 0.f);
            *out = r * r;
        } else {
            *out = v;
        }
    }
    if (a.splits > 1) f_cluster_sync();                    // nobody's sums go away while another block may still read them
}

template <int TM, int LM, int TN, bool GATED, bool VEC>
int f32_launch(F32Args a, dim3 grid, int stages, cudaStream_t stream) {
    constexpr int BM = TM * LM;
    const size_t smem = sizeof(float) * ((size_t)stages * (BM + F_ROWS) * FK + (size_t)BM * F_PITCH);
    cudaError_t e;
    static std::atomic<unsigned long long> allowed{0};     // (the number of stages, so the size, is the tile's)
    e = ce_allow_smem(allowed, gemm_f32_kernel<TM, LM, TN, GATED, VEC>, smem);
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_gemm_plain: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(F_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    a.overlap = 1;
    if (a.splits > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = a.splits;
        cfg.numAttrs = 1;
        static CeRoom room[F_MAX_RUNS + 1];
        const int at_once = ce_clusters_at_once(room[a.splits], gemm_f32_kernel<TM, LM, TN, GATED, VEC>, cfg);
        a.overlap = (long long)grid.x * grid.y <= at_once;       // see ce_clusters_at_once
        if (at_once == 0) {                                      // (no room for a cluster: the same sums on one block a tile)
            a.splits = cfg.gridDim.z = a.overlap = 1;
            cfg.numAttrs = 0;
        }
    }
    if (a.overlap && ce_pdl_enabled()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    ce_note(a.splits > 1 ? "gemm_f32_kernel (runs of K in a cluster)" : "gemm_f32_kernel");
    e = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<TM, LM, TN, GATED, VEC>, a, stages);
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_gemm_plain: %s", cudaGetErrorString(e));
    return ce_check_launch("ce_gemm_plain");
}

template <int TM, int LM, int TN>
int f32_pick(const F32Args& a, dim3 grid, int stages, bool vec, cudaStream_t stream) {
    if (GP_GATED(a.mode)) return vec ? f32_launch<TM, LM, TN, true, true>(a, grid, stages, stream) : f32_launch<TM, LM, TN, true, false>(a, grid, stages, stream);
    return vec ? f32_launch<TM, LM, TN, false, true>(a, grid, stages, stream) : f32_launch<TM, LM, TN, false, false>(a, grid, stages, stream);
}

}  // namespace

int ce_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int mode, const GpGate& gate,
                bool weights_ready, cudaStream_t stream) {
    const int runs = K / 256 < 1 ? 1 : K / 256 > F_MAX_RUNS ? F_MAX_RUNS : K / 256;
    const int run = ((K + runs - 1) / runs + FK - 1) / FK * FK;
    const bool vec = K % 4 == 0 && lda % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const int features = GP_GATED(mode) ? F_ROWS / 2 : F_ROWS;
    const int tokens = M <= 4 ? 4 : M <= 8 ? 8 : M <= 32 ? 32 : 64;
    const long long tiles = (long long)((N + features - 1) / features) * ((M + tokens - 1) / tokens);
    // Two blocks of the larger tiles share an SM.  With fewer tiles than that a cluster takes a tile's runs (301 tokens, 2,048 x 2,048:
    // 80 tiles, 87 us against 330 on one block a tile); with more it gains nothing (301 tokens, 480 tiles: 448 and 446 us) and
    // later loses (1,000 tokens, 1,536 tiles: 1,193 us on one block a tile, 1,396 in clusters).
    const int splits = runs > 1 && tiles < 2 * ce_sm_count() ? runs : 1;
    F32Args a{A, W, C, M, N, K, lda, ldc, mode, run, splits, weights_ready, 1, gate};
    dim3 grid((N + features - 1) / features, (M + tokens - 1) / tokens, splits);
    switch (tokens) {
        case 4: return f32_pick<4, 1, 1>(a, grid, 4, vec, stream);
        case 8: return f32_pick<8, 1, 1>(a, grid, 4, vec, stream);
        case 32: return f32_pick<8, 4, 4>(a, grid, 4, vec, stream);
        default: return f32_pick<8, 8, 8>(a, grid, 3, vec, stream);
    }
}
