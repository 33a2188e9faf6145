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
// One product (weight rows x K), us with the clusters -> here, weights from memory:
//                   2,048 x 2,048    2,560 x 9,728    4,096 x 4,096    4,096 x 12,288    5,120 x 5,120    12,288 x 2,048 (gated)
//     1 token        7.3 -> 6.1       33.3 -> 25.7     16.4 -> 12.7      42.9 -> 34.9      20.1 -> 19.5     22.5 -> 16.9
//     8 tokens      10.2 -> 7.6       47.1 -> 41.0     22.5 -> 18.1      60.3 -> 49.4      27.9 (there)     28.4 -> 22.3
#include "gemm_f32.cuh"
#include <type_traits>

namespace {

constexpr int FS_RUNS = 8;                              // runs of K = warps of a block
constexpr int FS_THREADS = 32 * FS_RUNS;
constexpr size_t FS_ALONE = 116 * 1024;                  // more than half of an SM's shared memory
constexpr size_t FS_MOST = 196 * 1024;                  // bytes of a block's rings

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

// Stages of a warp's ring: up to eight, as many as 150 KB hold, four or three where those need more.  (14 rows and 4 tokens: eight stages,
// 147 KB, 1,433 us a pass of four decode steps of four layers; four stages, 1,579.  2,560 x 9,728, where six fit: 25.7 us, with four 39.4,
// with the clusters 33.4.)
__host__ __device__ constexpr size_t fs_stage_bytes(int wrows, int tok, int ks) { return sizeof(float) * FS_RUNS * (wrows + tok) * ks; }
__host__ __device__ constexpr int fs_stages(int wrows, int tok, int ks) {
    const size_t stage = fs_stage_bytes(wrows, tok, ks);
    const int n = (int)(150 * 1024 / stage);
    return n > 8 ? 8 : n >= 4 ? n : 4 * stage <= FS_MOST ? 4 : 3;
}

// RT: rows a lane holds; LT: groups of lanes with tokens of their own, so that a warp holds 32 / LT x RT rows (of fewer, lanes
// multiply padding: a block of FIRST rows does the work of 32 / LT x RT); TOK: tokens; KS: k of a stage.
template <int RT, int LT, int FIRST, int TOK, int KS, bool GATED>
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
    auto walk = [&](auto depth) {
        constexpr int ST = decltype(depth)::value;
        int slot = 0, next = ST - 1;
        for (int s = 0; s < slabs; ++s) {
            // this warp's copies alone: all but the newest ST - 2 groups have landed
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncwarp();
            if (s + ST - 1 < slabs) { load_w(s + ST - 1, next); load_x(s + ST - 1, next); }
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
            if (++slot == ST) slot = 0;
            __syncwarp();                               // the slot just read takes the next copies
        }
    };
    // (the number of groups to wait for is part of the instruction: a loop for each depth that these rows can have)
    constexpr int LEAST = fs_stages(32 / LT * RT, TOK, KS), MOST = fs_stages(FIRST, TOK, KS);
    switch (a.stages) {
        case 8: if constexpr (LEAST <= 8 && MOST >= 8) walk(std::integral_constant<int, 8>{}); break;
        case 7: if constexpr (LEAST <= 7 && MOST >= 7) walk(std::integral_constant<int, 7>{}); break;
        case 6: if constexpr (LEAST <= 6 && MOST >= 6) walk(std::integral_constant<int, 6>{}); break;
        case 5: if constexpr (LEAST <= 5 && MOST >= 5) walk(std::integral_constant<int, 5>{}); break;
        case 4: if constexpr (LEAST <= 4 && MOST >= 4) walk(std::integral_constant<int, 4>{}); break;
        case 3: if constexpr (LEAST <= 3 && MOST >= 3) walk(std::integral_constant<int, 3>{}); break;
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

template <int RT, int LT, int FIRST, int TOK, int KS, bool GATED>
int fs_launch(const FsArgs& a, size_t smem, cudaStream_t stream) {
    static std::atomic<unsigned long long> allowed{0};
    cudaError_t e = ce_allow_smem(allowed, gemm_f32_stream_kernel<RT, LT, FIRST, TOK, KS, GATED>, 200 * 1024);
    if (e != cudaSuccess) return ce_fail(CE_ERR_CUDA, "ce_gemm_f32_stream: %s", cudaGetErrorString(e));
    ce_note("gemm_f32_stream_kernel");
    ce_launch(gemm_f32_stream_kernel<RT, LT, FIRST, TOK, KS, GATED>, (a.N + a.rows - 1) / a.rows, FS_THREADS, smem, stream, a);
    return ce_check_launch("ce_gemm_f32_stream");
}

template <int RT, int LT, int FIRST, int KS>
int fs_pick(FsArgs a, bool shared_sm, cudaStream_t stream) {
    const bool gated = GP_GATED(a.mode);
    const int wrows = gated ? 2 * a.rows : a.rows, tok = a.M <= 4 ? 4 : 8;
    a.stages = fs_stages(wrows, tok, KS);
    size_t smem = a.stages * fs_stage_bytes(wrows, tok, KS);
    if (smem > FS_MOST) return 1;
    const size_t sums = sizeof(float) * FS_RUNS * tok * (size_t)(wrows + 1);
    if (sums > smem) smem = sums;
    if (!shared_sm && smem < FS_ALONE) smem = FS_ALONE;
    if (tok == 4) return gated ? fs_launch<RT, LT, FIRST, 4, KS, true>(a, smem, stream) : fs_launch<RT, LT, FIRST, 4, KS, false>(a, smem, stream);
    return gated ? fs_launch<RT, LT, FIRST, 8, KS, true>(a, smem, stream) : fs_launch<RT, LT, FIRST, 8, KS, false>(a, smem, stream);
}

}  // namespace

// The product of ce_gemm_plain in float32, where this kernel takes its sizes: returns 1 where it does not, else as the other launchers.
// It takes up to 8 tokens, K of eight equal runs (multiples of 32) on 16-byte rows, and as many rows as leave a ring of three stages.
// Over 4 to 125 rows a block, 1 to 8 tokens and K of 2,048 to 12,288 it is the faster one but for the rule below.
extern "C" int ce_gemm_f32_stream(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldc, int mode, const float* bias,
                                  float limit, float alpha, int weights_ready, cudaStream_t stream) {
    if (M < 1 || M > 8 || K < 2048 || K % 256 || lda % 4 || (((uintptr_t)A | (uintptr_t)W) & 15) || mode < GP_STORE || mode > GP_CLAMPGLU) return 1;
    const int sms = ce_sm_count();
    if (!A || !W || !C || N < 4 * sms) return 1;
    const int rows = (N + sms - 1) / sms, blocks = (N + rows - 1) / rows, wrows = GP_GATED(mode) ? 2 * rows : rows;
    FsArgs a{A, W, C, M, N, K, lda, ldc, mode, rows, 0, weights_ready, GpGate{bias, limit, alpha}};
    // Up to 48 clusters of the other kernel run side by side, each near the memory's rate; 33 to 41 rows a block here cost nearly as much as 48.
    // (4,884 rows, 1 token: K of 2,048 10.0 us there and 9.1 here, of 12,288 44.7 and 42.3; 5 to 8 tokens 13.3 and 12.7, but 61.9 and 63.5; gated,
    // 2,516 features of 4,096: 16.9 and 17.7.)
    const int tile = GP_GATED(mode) ? 64 : 128;
    if (wrows > 32 && (N + tile - 1) / tile <= 48 && (GP_GATED(mode) || (M > 4 && K > 2048))) return 1;
    // One block an SM where some SMs have none: the next product's blocks would take their places beside others and leave theirs empty
    // (593 x 4,096, one product behind the other: 11.9 us with two blocks an SM, 8.4 with one).
    const bool shared_sm = blocks == sms;
    if (wrows <= 16) return fs_pick<1, 2, 4, 32>(a, shared_sm, stream);
    if (wrows <= 32) return fs_pick<1, 1, 17, 32>(a, shared_sm, stream);
    if (wrows <= 48) return fs_pick<3, 2, 33, 32>(a, shared_sm, stream);
    if (wrows <= 64) return fs_pick<2, 1, 49, 16>(a, shared_sm, stream);
    if (wrows <= 96) return fs_pick<3, 1, 65, 16>(a, shared_sm, stream);
    if (wrows <= 128) return fs_pick<4, 1, 97, 16>(a, shared_sm, stream);
    return 1;
}
