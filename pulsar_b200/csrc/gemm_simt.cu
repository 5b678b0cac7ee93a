// out[M, N] = A[M, K] * W[N, K]^T with float32 multiply-adds on the CUDA cores.
//
// This is the matrix product of the true 32-bit path: no tensor cores and no
// reduced-precision mode.  Each output element is a plain float32 sum over k in
// ascending order (one chain of multiply-adds, in every kernel of this file), so its value
// does not depend on M, on the position of its row in the batch, on which other rows are
// present or on which of the kernels ran.  A and W may be float32 or bfloat16 (read exactly,
// accumulated in float32); the output is float32 or the activation type.  Any M, N, K is accepted.
//
// Three kernels:
//   * simt_rows_kernel (up to 16 rows of A, float32 operands): streams the weights, bound by HBM;
//   * simt_tile_kernel (more rows, float32 operands): bound by the FMA pipes and the register file;
//   * gemm_simt_kernel: everything else (bfloat16 operands, rows of K that are no multiple of 16 bytes).
//
// The reference uses at::linear here (cuBLAS SGEMM in float32,
// pulsar-core/src/model/qwen3.cpp:82-84, 114, 117-119, 128).
#include "mma_common.cuh"

namespace {

using namespace pb;

// ---------------------------------------------------------------- up to 16 rows
// Bound by reading W once, and with more rows of A by shared memory.  The sums stay chains in ascending k: a chain takes 4 cycles
// a step, so 128 blocks of 32 weight rows ask for 8 TB/s, above what HBM gives, and a split of K (which would change the sums)
// is not needed.  W and A come through shared memory in stages of RK k by 16-byte asynchronous copies of four warps that do
// nothing else; CW further warps compute, a thread R rows of W times T rows of A.  Between two stages stands a barrier of the block, and
// behind it a wait for shared memory that nothing covers (150 cycles together, against the 256 of 64 k's chain): long stages.  (A
// warp that copies its own rows needs no barrier, but its copies then stand between its chains: 33 us for 4096 x 4096.)
// A loaded W depends on no earlier kernel: its first
// stages are asked for before griddepcontrol.wait (a W that may just have been computed: the ordinary launch, which begins behind
// it).  A 16-byte read of shared memory costs a warp 4 cycles, 2 where neighbouring lanes read the same place (measured), so lanes
// that share a row of W stand side by side; W's rows stand four floats more than a multiple of 32 apart, which keeps the others off each
// other's banks.
// us on the sizes of an 8B layer (64 x 64 tiles of the general kernel): 6144 x 4096 1 row 19.8 (277), 4 rows 24.4, 8 rows
// 29.6, 16 rows 58; 4096 x 4096 15.1 / 17.7 / 23.2 / 38.5 (282); 24576 x 4096 64 / 69 / 86 / 174 (480); 4096 x 12288
// 39.5 / 45.8 / 59.3 / 108 (851); 151936 x 4096 375 (6.6 TB/s) / 387 / 466 to 540 / 969.
constexpr int RN = 32, RLOAD = 128;

template <int R, int T, int CW, int RST, int RK, typename TO>
__global__ void __launch_bounds__(RLOAD + 32 * CW)
simt_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, TO* __restrict__ out, int M, int N, int K) {
    extern __shared__ __align__(16) float rows_smem[];
    constexpr int RSTRIDE = RK + 4;
    constexpr int LR = RN / R, LT = 32 / LR, MR = LT * T * CW;      // lanes along the rows of W, along those of A; rows of A held
    float* ws = rows_smem;                                  // [RST][RN][RSTRIDE]
    float* as = ws + RST * RN * RSTRIDE;                    // [RST][MR][RK]
    const int tid = threadIdx.x;
    const int row0 = blockIdx.x * RN;
    const int n_kt = (K + RK - 1) / RK;

    if (tid < RLOAD) {                                      // the copying warps
        const uint64_t policy = l2_policy_evict_first();
        const int q = tid % (RK / 4) * 4, r0 = tid / (RK / 4);     // this thread's column of 4 floats and its first row
        auto load_w = [&](int kt) {
            float* dst = ws + (kt % RST) * RN * RSTRIDE;
#pragma unroll
            for (int e = 0; e < RN * RK / 4 / RLOAD; ++e) {
                const int r = r0 + e * (RLOAD / (RK / 4));
                const bool ok = row0 + r < N && kt * RK + q < K;
                cp_async16_policy(smem_u32(dst + r * RSTRIDE + q), ok ? W + (size_t)(row0 + r) * K + kt * RK + q : W, ok, policy);
            }
        };
        auto load_a = [&](int kt) {
            float* dst = as + (kt % RST) * MR * RK;
#pragma unroll
            for (int r = r0; r < MR; r += RLOAD / (RK / 4)) {
                const bool ok = r < M && kt * RK + q < K;
                cp_async16(smem_u32(dst + r * RK + q), ok ? A + (size_t)r * K + kt * RK + q : A, ok);
            }
        };
#pragma unroll
        for (int s = 0; s < RST - 1; ++s) {
            if (s < n_kt) load_w(s);
            if (s < RST - 2) cp_async_commit();
        }
        pdl_wait();
        // A's first stages through registers, beside W's copies (a group of their own would have to wait for all of those)
        for (int s = 0; s < RST - 1 && s < n_kt; ++s)
            for (int r = r0; r < MR; r += RLOAD / (RK / 4)) {
                const bool ok = r < M && s * RK + q < K;
                *reinterpret_cast<float4*>(as + (s * MR + r) * RK + q) =
                    ok ? *reinterpret_cast<const float4*>(A + (size_t)r * K + s * RK + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        cp_async_commit();
        for (int kt = 0; kt < n_kt; ++kt) {
            cp_async_wait<RST - 2>();
            __syncthreads();                                // stage kt has landed; the one before it is done with
            if (kt + RST - 1 < n_kt) {
                load_w(kt + RST - 1);
                load_a(kt + RST - 1);
            }
            cp_async_commit();
        }
        pdl_trigger();
        return;
    }

    const int lane = tid & 31, warp = (tid - RLOAD) >> 5;
    constexpr int RU = R + T <= 3 ? 4 : 2;                  // k of a batch, in fours
    const int lr = LT == 1 ? lane : LT == 2 ? lane >> 1 : (lane & 1) | lane >> 3 << 1;
    const int m0 = warp * LT * T + (LT == 1 ? 0 : LT == 2 ? lane & 1 : lane >> 1 & 3) * T;
    float acc[R][T];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[r][t] = 0.0f;
    pdl_wait();
    for (int kt = 0; kt < n_kt; ++kt) {
        __syncthreads();
        const float* wr = ws + (kt % RST) * RN * RSTRIDE + lr * RSTRIDE;
        const float* ar = as + ((kt % RST) * MR + m0) * RK;
        float4 w[2][RU][R], a[2][RU][T];                    // the operands of a batch of 4 RU k, and of the next one
        auto fetch = [&](int b, int kk) {
#pragma unroll
            for (int u = 0; u < RU; ++u) {
#pragma unroll
                for (int r = 0; r < R; ++r) w[b][u][r] = *reinterpret_cast<const float4*>(wr + r * LR * RSTRIDE + kk + 4 * u);
#pragma unroll
                for (int t = 0; t < T; ++t) a[b][u][t] = *reinterpret_cast<const float4*>(ar + t * RK + kk + 4 * u);
            }
        };
        auto step = [&](float (&c)[R][T], const float4 (&x)[T], const float4 (&y)[R]) {
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int t = 0; t < T; ++t) c[r][t] = fmaf(x[t].x, y[r].x, c[r][t]);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int t = 0; t < T; ++t) c[r][t] = fmaf(x[t].y, y[r].y, c[r][t]);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int t = 0; t < T; ++t) c[r][t] = fmaf(x[t].z, y[r].z, c[r][t]);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int t = 0; t < T; ++t) c[r][t] = fmaf(x[t].w, y[r].w, c[r][t]);
        };
        fetch(0, 0);
#pragma unroll
        for (int kk = 0; kk < RK; kk += 4 * RU) {
            const int b = kk / (4 * RU) & 1;
            if (kk + 4 * RU < RK) fetch(b ^ 1, kk + 4 * RU);
#pragma unroll
            for (int u = 0; u < RU; ++u) step(acc, a[b][u], w[b][u]);
        }
    }
    pdl_trigger();
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int n = row0 + lr + r * LR;
            if (m0 + t < M && n < N) out[(size_t)(m0 + t) * N + n] = from_float<TO>(acc[r][t]);
        }
}

template <int R, int T, int CW, int RST, int RK, typename TO>
int launch_rows(const float* A, const float* W, TO* out, int M, int N, int K, bool loaded, cudaStream_t stream) {
    constexpr int MR = 32 / (RN / R) * T * CW;
    constexpr size_t smem = sizeof(float) * RST * (RN * (RK + 4) + MR * RK);
    static SmemLimit limit;
    if (const int rc = limit.allow(simt_rows_kernel<R, T, CW, RST, RK, TO>, smem)) return rc;
    return launch_early(loaded, simt_rows_kernel<R, T, CW, RST, RK, TO>, dim3((N + RN - 1) / RN), dim3(RLOAD + 32 * CW), smem, stream, A, W, out, M, N, K);
}

// ---------------------------------------------------------------- more rows
// Bound by the FMA pipes and the register file.  A block of 128 threads owns 32 x 128 outputs, a warp 32 x 32, a thread 4 x 8.  Of the
// 8 x 4 lanes of a warp neighbours share a row or a column (see above).  This form, with single multiply-adds, serves where an SM has
// one block, and the last rows: a block whose last rows lie behind M computes 8 or 16.  Both operands stand in shared memory as they do
// in memory, k fastest, so that asynchronous 16-byte copies bring them and a thread reads four k of a row at once (rows ty + 8 i,
// columns tx + 4 j).  Rows stand an odd number of 16-byte units apart (no bank conflicts).  Two stages of 32 k: half the barriers of
// three stages of 16 (24576 x 4096 with 387 rows 2.03 -> 1.90 ms, 4096 x 4096 389 -> 356 us).
constexpr int GM = 32, GN = 128, GK = 32, GST = 2, GSTRIDE = GK + 4;

template <int NI, typename TO>
__device__ __forceinline__ void tile_block(const float* __restrict__ A, const float* __restrict__ W, TO* __restrict__ out,
                                           int M, int N, int K, float* smem) {
    constexpr int LR = 128 / (GK / 4);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane >> 1 & 3, ty = (lane & 1) | lane >> 3 << 1;
    const int row0 = blockIdx.x * GM, col0 = blockIdx.y * GN;
    constexpr int kStage = (GM + GN) * GSTRIDE;
    const int n_kt = (K + GK - 1) / GK;
    const int lq = tid % (GK / 4) * 4, lr = tid / (GK / 4);      // this thread's four k and its row within a copy of LR rows
    auto load = [&](int kt) {
        float* dst = smem + (kt % GST) * kStage + lq;
        const int k = kt * GK + lq;
#pragma unroll
        for (int r = lr; r < 8 * NI; r += LR) {
            const bool ok = k < K && row0 + r < M;
            cp_async16(smem_u32(dst + r * GSTRIDE), ok ? A + (size_t)(row0 + r) * K + k : A, ok);
        }
#pragma unroll
        for (int r = lr; r < GN; r += LR) {
            const bool ok = k < K && col0 + r < N;
            cp_async16(smem_u32(dst + (GM + r) * GSTRIDE), ok ? W + (size_t)(col0 + r) * K + k : W, ok);
        }
    };
    float acc[NI][8];
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
#pragma unroll
    for (int s = 0; s < GST - 1; ++s) {
        if (s < n_kt) load(s);
        cp_async_commit();
    }
    for (int kt = 0; kt < n_kt; ++kt) {
        cp_async_wait<GST - 2>();
        __syncthreads();
        if (kt + GST - 1 < n_kt) load(kt + GST - 1);
        cp_async_commit();
        const float* a_s = smem + (kt % GST) * kStage + ty * GSTRIDE;
        const float* w_s = smem + (kt % GST) * kStage + (GM + warp * 32 + tx) * GSTRIDE;
#pragma unroll
        for (int kk = 0; kk < GK; kk += 4) {
            float4 a[NI];
#pragma unroll
            for (int i = 0; i < NI; ++i) a[i] = *reinterpret_cast<const float4*>(a_s + 8 * i * GSTRIDE + kk);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(w_s + 4 * j * GSTRIDE + kk);
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < NI; ++i) acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int r = row0 + ty + 8 * i;
        if (r >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = col0 + warp * 32 + tx + 4 * j;
            if (c < N) out[(size_t)r * N + c] = from_float<TO>(acc[i][j]);
        }
    }
}

// 32 rows by 128 columns with paired multiply-adds (fma.rn.f32x2: two sums of neighbouring columns, each rounded by itself, so the same
// bits).  From registers alone single multiply-adds reach 52 TFLOP/s here, paired ones 63: three operands a lane and cycle are more than
// the register file gives.  A pair wants neighbouring columns in neighbouring registers, so both operands stand with k slowest in
// shared memory: 16-byte loads of four k bring them to registers while the stage before is computed, and four stores turn them (columns
// shifted by the k's quad, which spreads the stores over the banks).  A thread takes rows 4 ty .. 4 ty + 3 and columns 4 tx .. + 3 and 16 + 4 tx ..
// + 3 of its warp's 32; its a values are doubled into pairs.  us, single multiply-adds before: 24576 x 4096 with 387 rows 1,898 -> 1,732,
// 4096 x 4096 357 -> 338, 6144 x 4096 634 -> 493.  With 64 rows a block 1,838, with pairs along the rows 1,883.
__device__ __forceinline__ unsigned long long pair_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
template <typename TO>
__device__ __forceinline__ void pair_block(const float* __restrict__ A, const float* __restrict__ W, TO* __restrict__ out,
                                           int M, int N, int K, float* smem) {
    constexpr int kStage = GK * (GM + GN), QK = GK / 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane >> 1 & 3, ty = (lane & 1) | lane >> 3 << 1;
    const int row0 = blockIdx.x * GM, col0 = blockIdx.y * GN, n_kt = (K + GK - 1) / GK;
    const int q = tid % QK, r0 = tid / QK;                   // this thread's quad of k and its first row of 16 a round
    float4 ra[GM / 16], rw[GN / 16];
    auto fetch = [&](int kt) {
        const int k = kt * GK + q * 4;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int e = 0; e < GM / 16; ++e) {
            const int r = row0 + r0 + 16 * e;
            ra[e] = r < M && k < K ? *reinterpret_cast<const float4*>(A + (size_t)r * K + k) : zero;
        }
#pragma unroll
        for (int e = 0; e < GN / 16; ++e) {
            const int r = col0 + r0 + 16 * e;
            rw[e] = r < N && k < K ? *reinterpret_cast<const float4*>(W + (size_t)r * K + k) : zero;
        }
    };
    auto put = [&](float* dst, int rows, int at, const float4& v) {
        dst += q * 4 * rows + (at ^ 8 * (q & 3));
        dst[0] = v.x; dst[rows] = v.y; dst[2 * rows] = v.z; dst[3 * rows] = v.w;
    };
    auto stash = [&](int stage) {
        float* as = smem + stage * kStage;
#pragma unroll
        for (int e = 0; e < GM / 16; ++e) put(as, GM, r0 + 16 * e, ra[e]);
#pragma unroll
        for (int e = 0; e < GN / 16; ++e) put(as + GK * GM, GN, r0 + 16 * e, rw[e]);
    };
    unsigned long long acc[4][4];                            // [row][pair of columns]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    fetch(0);
    stash(0);
    __syncthreads();
    for (int kt = 0; kt < n_kt; ++kt) {
        if (kt + 1 < n_kt) fetch(kt + 1);
        const float* as = smem + (kt & 1) * kStage;
        const float* ws = as + GK * GM + warp * 32;
#pragma unroll
        for (int k = 0; k < GK; ++k) {
            const int shift = 8 * (k >> 2 & 3);
            const float4 a = *reinterpret_cast<const float4*>(as + k * GM + ((ty * 4) ^ shift));
            const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + k * GN + ((tx * 4) ^ shift));
            const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(ws + k * GN + ((tx * 4 + 16) ^ shift));
            const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                unsigned long long d;
                asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(av[i]));
                acc[i][0] = pair_fma(d, w0.x, acc[i][0]);
                acc[i][1] = pair_fma(d, w0.y, acc[i][1]);
                acc[i][2] = pair_fma(d, w1.x, acc[i][2]);
                acc[i][3] = pair_fma(d, w1.y, acc[i][3]);
            }
        }
        if (kt + 1 < n_kt) stash((kt + 1) & 1);
        __syncthreads();
    }
    const bool vector = N % 4 == 0 && (uintptr_t)out % (4 * sizeof(TO)) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= M) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = col0 + warp * 32 + tx * 4 + 16 * h;
            float v[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][2 * h]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][2 * h + 1]));
            TO* o = out + (size_t)r * N + c;
            if (vector && c < N) store_quad(o, v);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (c + e < N) o[e] = from_float<TO>(v[e]);
        }
    }
}

template <bool kPairs, typename TO>
__global__ void __launch_bounds__(128, 4)
simt_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, TO* __restrict__ out, int M, int N, int K) {
    __shared__ __align__(16) float tile_smem[GST * (GM + GN) * GSTRIDE];
    const int left = M - (int)blockIdx.x * GM;
    if (kPairs && left > 16) pair_block<TO>(A, W, out, M, N, K, tile_smem);
    else if (left > 16) tile_block<4, TO>(A, W, out, M, N, K, tile_smem);
    else if (left > 8) tile_block<2, TO>(A, W, out, M, N, K, tile_smem);
    else tile_block<1, TO>(A, W, out, M, N, K, tile_smem);
}

template <bool kPairs, typename TO>
int launch_tile(const float* A, const float* W, TO* out, int M, int N, int K, cudaStream_t stream) {
    dim3 grid((M + GM - 1) / GM, (N + GN - 1) / GN);
    if (grid.y > 65535) return PB_ERR_TOO_LARGE;
    simt_tile_kernel<kPairs, TO><<<grid, 128, 0, stream>>>(A, W, out, M, N, K);
    return launch_status();
}

// float32 operands whose rows are multiples of 16 bytes on 16-byte addresses
template <typename TO>
int launch_f32(const float* A, const float* W, TO* out, int M, int N, int K, bool loaded, cudaStream_t stream) {
    // With one block an SM or fewer a block's ring has to keep HBM busy by itself, and its chain is as long as the barriers between its
    // stages make it: four stages of 256 k, where more blocks an SM take four of 128 (five to eight rows: two of 256).  us, 64 k a stage:
    // 4096 x 4096 4 rows 21.2 -> 17.6, 8 rows 27.1 -> 23.2; 24576 x 4096 4 rows 74.9 -> 69.2, 8 rows 103.3 -> 85.7 (93.6 with 128 k),
    // 16 rows 188.5 -> 174; 151936 x 4096 8 rows 562 to 618 -> 466 to 540; 2048 x 2048 one row 11.9 -> 8.1.
    // Stages of 64 k under a short K: a long stage is waited for and multiplied whole however few of its k there are.  us with 64 k / with
    // long stages: 1024 x 64 1 row 1.4 / 1.8, 8 rows 1.3 / 2.8, x 128 2 rows 1.8 / 1.9, 4 rows 1.9 / 2.1, 8 rows 1.9 / 2.7, 16 rows 3.0 / 3.5,
    // x 192 4 rows 2.3 / 2.1, x 320 8 rows 3.6 / 4.7, x 512 4.9 / 4.7, x 576 6.2 / 7.2, 16 rows 10.3 / 8.7; 8192 x 192 16 rows 5.4 / 6.4.
    const bool few = (N + RN - 1) / RN <= 148;
    const bool brief = M <= 2 ? K <= 64 : M <= 4 ? K <= (few ? 128 : 64) : M <= 8 ? K < (few ? 640 : 384) && K % 256 != 0
                              : K <= 128 || (!few && K < 384 && K % 128 != 0);
#define PB_ROWS(R, T, CW, ST, RK) return launch_rows<R, T, CW, ST, RK>(A, W, out, M, N, K, loaded, stream)
    if (brief) {
        if (M == 1) PB_ROWS(1, 1, 1, 8, 64);
        if (M == 2) PB_ROWS(2, 1, 1, 8, 64);
        if (M <= 4) PB_ROWS(2, 1, 2, 8, 64);
        if (M <= 8) { if (few) PB_ROWS(2, 1, 4, 16, 64); PB_ROWS(2, 2, 2, 8, 64); }
        if (M <= 16) { if (few) PB_ROWS(2, 1, 8, 16, 64); PB_ROWS(4, 2, 2, 8, 64); }
    }
    if (M == 1) { if (few) PB_ROWS(1, 1, 1, 4, 256); PB_ROWS(1, 1, 1, 4, 128); }
    if (M == 2) { if (few) PB_ROWS(2, 1, 1, 4, 256); PB_ROWS(2, 1, 1, 4, 128); }
    if (M <= 4) { if (few) PB_ROWS(2, 1, 2, 4, 256); PB_ROWS(2, 1, 2, 4, 128); }
    if (M <= 8) { if (few) PB_ROWS(2, 1, 4, 4, 256); PB_ROWS(2, 2, 2, 2, 256); }
    if (M <= 16) { if (few) PB_ROWS(2, 1, 8, 4, 256); PB_ROWS(4, 2, 2, 4, 128); }
#undef PB_ROWS
    // Pairs where an SM has two blocks and more, whose loads then cover each other's (4096 x 12288, 200 rows: 773 us both ways;
    // 151936 x 4096, 387 rows: 10.1 ms, 11.2 with single multiply-adds, 11.3 with single ones and 64 rows a block): with one, the
    // asynchronous copies are ahead (100 rows 448 against 608; 6144 x 4096, 64 rows 153 against 217).
    if ((long)((M + GM - 1) / GM) * ((N + GN - 1) / GN) > 148) return launch_tile<true>(A, W, out, M, N, K, stream);
    return launch_tile<false>(A, W, out, M, N, K, stream);
}

// ---------------------------------------------------------------- any operands
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;   // 256 threads, 4x4 outputs each

template <typename TA, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ out, int M, int N, int K) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int tr = (tid / 16) * TM, tc = (tid % 16) * TN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k per operand = 1024 elements, 4 per thread, k fastest for coalescing.
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;
            const int r = idx / BK, kk = idx % BK;
            const int gr = row0 + r, gk = k0 + kk;
            As[kk][r] = (gr < M && gk < K) ? to_float(A[(size_t)gr * K + gk]) : 0.0f;
            const int gc = col0 + r;
            Ws[kk][r] = (gc < N && gk < K) ? to_float(W[(size_t)gc * K + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][tr + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tc + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gr = row0 + tr + i;
        if (gr >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gc = col0 + tc + j;
            if (gc < N) out[(size_t)gr * N + gc] = from_float<TO>(acc[i][j]);
        }
    }
}

template <typename TA, typename TW, typename TO>
int launch(const void* A, const void* W, void* out, int M, int N, int K, cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return PB_ERR_TOO_LARGE;
    gemm_simt_kernel<TA, TW, TO><<<grid, 256, 0, stream>>>((const TA*)A, (const TW*)W, (TO*)out, M, N, K);
    return launch_status();
}

}  // namespace

static int gemm_simt(int a_dtype, int w_dtype, int out_dtype, const void* A, const void* W, void* out, int M, int N, int K, bool loaded,
                     cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return PB_ERR_BAD_SIZE;
    if ((a_dtype | w_dtype | out_dtype) & ~1) return PB_ERR_BAD_DTYPE;
    typedef __nv_bfloat16 bf;
    if (a_dtype == PB_F32 && w_dtype == PB_F32 && K % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0) {
        const int status = out_dtype == PB_F32 ? launch_f32((const float*)A, (const float*)W, (float*)out, M, N, K, loaded, stream)
                                               : launch_f32((const float*)A, (const float*)W, (bf*)out, M, N, K, loaded, stream);
        if (status != PB_ERR_TOO_LARGE) return status;
    }
    const int key = a_dtype * 4 + w_dtype * 2 + out_dtype;
    switch (key) {
        case 0: return launch<float, float, float>(A, W, out, M, N, K, stream);
        case 1: return launch<float, float, bf>(A, W, out, M, N, K, stream);
        case 2: return launch<float, bf, float>(A, W, out, M, N, K, stream);
        case 3: return launch<float, bf, bf>(A, W, out, M, N, K, stream);
        case 4: return launch<bf, float, float>(A, W, out, M, N, K, stream);
        case 5: return launch<bf, float, bf>(A, W, out, M, N, K, stream);
        case 6: return launch<bf, bf, float>(A, W, out, M, N, K, stream);
        case 7: return launch<bf, bf, bf>(A, W, out, M, N, K, stream);
    }
    return PB_ERR_BAD_DTYPE;
}

// a_dtype / w_dtype / out_dtype: PB_F32 or PB_BF16.
PB_EXPORT int pb_gemm_simt(int a_dtype, int w_dtype, int out_dtype, const void* A, const void* W, void* out,
                           int M, int N, int K, cudaStream_t stream) {
    return gemm_simt(a_dtype, w_dtype, out_dtype, A, W, out, M, N, K, false, stream);
}

// The same for a W that no kernel still on the stream writes (a loaded weight): it may be read before those have ended.
PB_EXPORT int pb_gemm_simt_loaded(int a_dtype, int w_dtype, int out_dtype, const void* A, const void* W, void* out,
                                  int M, int N, int K, cudaStream_t stream) {
    return gemm_simt(a_dtype, w_dtype, out_dtype, A, W, out, M, N, K, true, stream);
}
