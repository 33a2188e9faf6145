// y = x * W^T in float32 for a few tokens (decode steps), as a stream of weights: the sums of gemm_f32.cu, bit for bit (eight runs of
// K, each two chains of fused multiply-adds, added in order), without a cluster.
//
// What bounds such a product is reading the weights once, and the way from one kernel of a step to the next.  The clusters of
// gemm_f32.cu give a run of K to each of eight blocks, which meet at cluster barriers before and after the sums are added, wait for
// room for eight blocks at once, and keep the next kernel's blocks out meanwhile.  Here a block takes all of K for its share of the
// weight rows (dealt evenly, one block an SM), and a run belongs to a WARP: it copies its run's part of the rows and of the tokens
// into a ring of its own (cp.async, no barrier of the block inside the loop), a lane holds whole rows, and the eight runs meet in
// shared memory once.
// Measured: four decode steps of four layers (width 2,048, 4 requests of 350 to 700 tokens) 1,592 us with the clusters -> 1,430.
#include "gemm_f32.cuh"

namespace {

constexpr int FS_RUNS = 8;                              // runs of K = warps of a block
constexpr int FS_THREADS = 32 * FS_RUNS;
constexpr int FS_BLOCKS = 148;                          // blocks the rows are dealt to

struct FsArgs {
    const float* A;
    const float* W;
    float* C;
    int M, N, K, lda, ldc, mode;
    int rows, stages, weights_ready;                    // output features of a block; stages of a warp's ring; no kernel in front writes W
    GpGate gate;
};

// (half of a 128-byte line a row and stage with 16 k: the first half asks for the whole line)
__device__ __forceinline__ void fs_cp16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// 16 bytes c of row r in a tile of rows of KS floats: eight neighbouring rows' pieces meet all banks
template <int KS>
__device__ __forceinline__ int fs_at(int r, int c) { return r * KS + ((KS == 32 ? c ^ (r & 7) : c ^ ((r >> 1) & 3)) << 2); }

// RT: rows a lane holds; LT: groups of lanes with tokens of their own (2 where a block has at most 16 rows); TOK: tokens; KS: k of a stage.
template <int RT, int LT, int TOK, int KS, bool GATED>
__global__ void __launch_bounds__(FS_THREADS, 2) gemm_f32_stream_kernel(FsArgs a) {
    extern __shared__ __align__(128) float fs_smem[];
    constexpr int PIECES = KS / 4, LR = 32 / LT, TT = TOK / LT, STEP = 32 / PIECES;
    const int tid = threadIdx.x, run = tid >> 5, lane = tid & 31, lr = lane % LR, lt = lane / LR;
    const int n0 = blockIdx.x * a.rows, n_valid = min(a.rows, a.N - n0);
    const int wrows = GATED ? 2 * a.rows : a.rows, stage = (wrows + TOK) * KS, run_k = a.K / FS_RUNS, k0 = run * run_k, slabs = run_k / KS;
    float* ring = fs_smem + run * a.stages * stage;
    const int piece = lane % PIECES, first_row = lane / PIECES;
    const float* w_src = a.W + k0 + piece * 4;
    const float* x_src = a.A + k0 + piece * 4;
    auto load_w = [&](int s, int slot) {
        float* t = ring + slot * stage;
        for (int r = first_row; r < wrows; r += STEP) {
            const int f = GATED && r >= a.rows ? r - a.rows : r;
            const bool in = f < n_valid;
            const size_t row = (size_t)(GATED && r >= a.rows ? a.N : 0) + n0 + (in ? f : 0);
            fs_cp16(t + fs_at<KS>(r, piece), w_src + row * a.K + s * KS, in);
        }
    };
    auto load_x = [&](int s, int slot) {
        float* t = ring + slot * stage + wrows * KS;
#pragma unroll
        for (int r0 = 0; r0 < TOK; r0 += STEP) {
            const int r = r0 + first_row;
            if (r < TOK) fs_cp16(t + fs_at<KS>(r, piece), x_src + (size_t)(r < a.M ? r : 0) * a.lda + s * KS, r < a.M);
        }
    };
    // weights that no kernel writes come before the wait for the kernels in front; any other W is read after it, like A
    ce_pdl_launch_dependents();
    if (!a.weights_ready) ce_pdl_wait();
    for (int s = 0; s < a.stages - 1; ++s)
        if (s < slabs) load_w(s, s);
    ce_pdl_wait();
    for (int s = 0; s < a.stages - 1; ++s) {
        if (s < slabs) load_x(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float2 acc[RT][TT];
#pragma unroll
    for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int m = 0; m < TT; ++m) acc[j][m] = make_float2(0.f, 0.f);
    int row[RT];
#pragma unroll
    for (int j = 0; j < RT; ++j) row[j] = min(lr + LR * j, wrows - 1);               // (lanes beyond the rows: any, not stored)
    int slot = 0, next = a.stages - 1;
    for (int s = 0; s < slabs; ++s) {
        // this warp's copies alone: all but the newest stages - 2 groups have landed
        if (a.stages == 8) asm volatile("cp.async.wait_group 6;" ::: "memory");
        else if (a.stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        if (s + a.stages - 1 < slabs) { load_w(s + a.stages - 1, next); load_x(s + a.stages - 1, next); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* wt = ring + slot * stage;
        const float* xt = wt + wrows * KS;
#pragma unroll(RT * TT >= 8 ? 2 : 4)
        for (int q = 0; q < PIECES; ++q) {
            float4 w[RT];
#pragma unroll
            for (int j = 0; j < RT; ++j) w[j] = *reinterpret_cast<const float4*>(wt + fs_at<KS>(row[j], q));
#pragma unroll
            for (int m = 0; m < TT; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(xt + fs_at<KS>(lt * TT + m, q));
#pragma unroll
                for (int j = 0; j < RT; ++j) {
                    acc[j][m] = __ffma2_rn(make_float2(x.x, x.y), make_float2(w[j].x, w[j].y), acc[j][m]);
                    acc[j][m] = __ffma2_rn(make_float2(x.z, x.w), make_float2(w[j].z, w[j].w), acc[j][m]);
                }
            }
        }
        next = slot;
        if (++slot == a.stages) slot = 0;
        __syncwarp();                                   // the slot just read takes the next copies
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float* part = fs_smem;                              // [run][token][row]
    const int pitch = wrows + 1;
#pragma unroll
    for (int j = 0; j < RT; ++j)
#pragma unroll
        for (int m = 0; m < TT; ++m)
            if (lr + LR * j < wrows) part[(run * TOK + lt * TT + m) * pitch + lr + LR * j] = acc[j][m].x + acc[j][m].y;
    __syncthreads();
    auto total = [&](int m, int r) {
        float v = part[m * pitch + r];
#pragma unroll
        for (int g = 1; g < FS_RUNS; ++g) v += part[(g * TOK + m) * pitch + r];
        return v;
    };
    for (int item = tid; item < a.M * n_valid; item += FS_THREADS) {
        const int m = item / n_valid, r = item - m * n_valid, n = n0 + r;
        float v = total(m, r);
        float* out = a.C + (size_t)m * a.ldc + n;
        if (GATED) {
            float u = total(m, a.rows + r);
            if (a.mode == GP_CLAMPGLU) {
                if (a.gate.bias) { v += a.gate.bias[n]; u += a.gate.bias[a.N + n]; }
                *out = ce_clamp_glu(v, u, a.gate.limit, a.gate.alpha);
            } else {
                *out = a.mode == GP_RELUGLU ? fmaxf(v, 0.f) * u : ce_silu_glu(v, u);
            }
        } else if (a.mode == GP_ACCUM_F32) {
            *out += v;
        } else if (a.mode == GP_RELU2) {
            const float p = fmaxf(v, 0.f);
            *out = p * p;
        } else {
            *out = v;
        }
    }
}

template <int RT, int LT, int TOK, int KS, bool GATED>
int fs_launch(const FsArgs& a, size_t smem, cudaStream_t stream) {
    static std::atomic<unsigned long long> allowed{0};
    cudaError_t e = ce_allow_smem(allowed, gemm_f32_stream_kernel<RT, LT, TOK, KS, GATED>, 200 * 1024);
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_gemm_f32_stream: %s", cudaGetErrorString(e));
    ce_note("gemm_f32_stream_kernel");
    ce_launch(gemm_f32_stream_kernel<RT, LT, TOK, KS, GATED>, (a.N + a.rows - 1) / a.rows, FS_THREADS, smem, stream, a);
    return ce_check_launch("ce_gemm_f32_stream");
}

template <int RT, int LT, int KS>
int fs_pick(const FsArgs& a, size_t smem, cudaStream_t stream) {
    if (a.M <= 4) return GP_GATED(a.mode) ? fs_launch<RT, LT, 4, KS, true>(a, smem, stream) : fs_launch<RT, LT, 4, KS, false>(a, smem, stream);
    return GP_GATED(a.mode) ? fs_launch<RT, LT, 8, KS, true>(a, smem, stream) : fs_launch<RT, LT, 8, KS, false>(a, smem, stream);
}

}  // namespace

// The product of ce_gemm_plain in float32, where this kernel takes its sizes: returns 1 where it does not, else as the other launchers.
// It takes up to 8 tokens, K of eight equal runs (multiples of 32) on 16-byte rows, and as many rows as leave a ring of three stages.
extern "C" int ce_gemm_f32_stream(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int mode, const float* bias,
                                  float limit, float alpha, int weights_ready, cudaStream_t stream) {
    if (M < 1 || M > 8 || K < 2048 || K % 256 || lda % 4 || (((uintptr_t)A | (uintptr_t)W) & 15) || mode < GP_STORE || mode > GP_CLAMPGLU) return 1;
    if (!A || !W || !C || N < 4 * FS_BLOCKS) return 1;
    const int rows = (N + FS_BLOCKS - 1) / FS_BLOCKS, wrows = GP_GATED(mode) ? 2 * rows : rows, rt = (wrows + 31) / 32;
    if (rt > 4) return 1;
    const int tok = M <= 4 ? 4 : 8, ks = rt == 1 ? 32 : 16;
    const size_t stage = sizeof(float) * FS_RUNS * (size_t)(wrows + tok) * ks;
    // Eight stages where 150 KB hold them, else four, else three of what an SM has.  (14 rows and 4 tokens: eight stages, 147 KB, 1,433 us
    // a pass of four decode steps of four layers; four stages, which leave room for the next product's block, 1,579.)
    int stages = (int)(150 * 1024 / stage);
    if (stages < 4) stages = (int)(196 * 1024 / stage);
    if (stages < 3) return 1;
    stages = stages >= 8 ? 8 : stages >= 4 ? 4 : 3;
    size_t smem = stages * stage;
    const size_t sums = sizeof(float) * FS_RUNS * tok * (size_t)(wrows + 1);
    if (sums > smem) smem = sums;
    FsArgs a{A, W, C, M, N, K, lda, ldc, mode, rows, stages, weights_ready, GpGate{bias, limit, alpha}};
    if (wrows <= 16) return fs_pick<1, 2, 32>(a, smem, stream);
    switch (rt) {
        case 1: return fs_pick<1, 1, 32>(a, smem, stream);
        case 2: return fs_pick<2, 1, 16>(a, smem, stream);
        case 3: return fs_pick<3, 1, 16>(a, smem, stream);
        default: return fs_pick<4, 1, 16>(a, smem, stream);
    }
}
