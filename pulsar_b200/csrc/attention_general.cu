// Paged attention in its general form: keys and values of different widths, an optional
// distance bias per head, a sliding window and a chunk mask, float32 queries.
//
// What the kinds of attention that the head-size-specific kernels do not cover share:
//   * key rows `Dk` wide and value rows `Dv` wide, each with a row stride of its own, so that
//     the value may be a leading part of the cached key row (attention over a compressed
//     latent: key = [latent | rotated part], value = latent, one cached tensor);
//   * score = (q . k) * scale - slope[h] * (p - j) where `slopes` is given (a linear distance
//     bias; p the query's position, j the key's);
//   * visible keys lo .. p with lo the largest of 0, p - window + 1 (window > 0) and
//     floor(p / chunk) * chunk (chunk > 0; chunks are counted from position 0 of the sequence);
//     with keep_first > 0 the keys 0 .. keep_first - 1 stay visible below lo as well (at their true positions);
//   * with softcap > 0 the scaled score becomes softcap * tanh(score / softcap) (before the distance bias);
//   * with `sinks` [Hq] the softmax's denominator holds one more term per head, exp(sinks[h]), that has no value;
//   * with `sigmoid` there is no softmax: a visible key's weight is 1 / (1 + exp(-(score + score_bias[h]))) (score_bias
//     optional), and the weights are not normalised over the keys;
//   * with `out_cos` / `out_sin` [N, Dv / 2] the finished output row of a token turns back by the token's angles: columns
//     2m and 2m + 1 are a pair (u, v) -> (u cos + v sin, v cos - u sin), before the one rounding (values that were cached
//     turned by their own positions then enter by the difference of the two).
// Queries come in float32 (rotation and score are 32-bit arithmetic whatever the cache holds);
// scores, the running maximum, the sums and the output accumulate in float32 with expf.
//
// One block per (query token, query head); key tiles of 32 aligned to absolute key indices,
// tile i handled by warp i mod 4, warps combined in index order: the result at a position does
// not depend on how the tokens were cut into steps, on what else is in the batch or on which
// pages hold the keys.  Prompt portions and single decoded tokens take the same kernel.
//
// Layouts: q [N, Hq, Dk] float32; out [N, Hq, Dv] T (float32 with out_f32); pools [pages, Hkv, page_size, stride] T;
// block_table [S, table_stride]; cu_q [S+1]; kv_len [S] (after this step); seq_of_token [N].
//
// Also here: the kernel that splits a fused projection row [q | k | v] of such widths into float32
// queries and the pages.
#include "mma_common.cuh"

namespace {

using namespace pb;

constexpr int kWarps = 4;

template <typename T> struct Vec;
template <> struct Vec<float> { static constexpr int n = 4; };
template <> struct Vec<__nv_bfloat16> { static constexpr int n = 8; };

__device__ __forceinline__ void load16(const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
__device__ __forceinline__ void load16(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

struct GeneralShape {
    int Hq, Hkv, Dk, Dv, k_stride, v_stride, page_size, window, chunk, table_stride;
    int k_vec;          // leading key elements that 16-byte loads may take (0 when rows are not 16-byte aligned)
    float scale;
    int keep_first;     // keys below this stay visible whatever the window or chunk says; 0: none
    float softcap;      // > 0: scaled scores are capped to softcap * tanh(score / softcap)
    int v_share;        // consecutive key heads that read one value head (the value pool has Hkv / v_share heads); 1: a value head per key head
    int out_f32;        // the output rows are float32 whatever the pools' type (what follows subtracts them from one another)
    int sigmoid;        // a key's weight is the sigmoid of its score (+ score_bias[head]) and nothing is normalised
    const float *score_bias, *out_cos, *out_sin;
};

__device__ __forceinline__ float sigmoid_weight(float s) { return 1.0f / (1.0f + expf(-s)); }

// Columns 2m and 2m + 1 of a finished row turn back by angle m of the row's token; `even`: this is the pair's first column.
__device__ __forceinline__ float turned_back(float own, float other, int m, int even, const float* cos_row, const float* sin_row) {
    return even ? own * cos_row[m] + other * sin_row[m] : own * cos_row[m] - other * sin_row[m];
}

template <typename T>
__device__ __forceinline__ void store_out(T* out, size_t at, float v, int out_f32) {
    if (out_f32) reinterpret_cast<float*>(out)[at] = v;
    else out[at] = from_float<T>(v);
}

// Tiles of 32 keys that a query (or a block of queries) with lowest key `lo` walks over: the tiles that hold kept first
// keys and lie wholly below the tile of `lo`, then the tiles from that of `lo` on.  n_kept is the count of the former.
__device__ __forceinline__ int kept_tiles(int lo, int keep_first) {
    return min((keep_first + 31) >> 5, lo >> 5);
}
__device__ __forceinline__ float cap_score(float s, float softcap) {
    return softcap > 0.0f ? softcap * tanhf(s / softcap) : s;
}

template <typename T, int ACC>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_general_kernel(const float* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                               T* __restrict__ out, const int* __restrict__ block_table, const int* __restrict__ cu_q,
                               const int* __restrict__ kv_len, const int* __restrict__ seq_of_token,
                               const float* __restrict__ slopes, const float* __restrict__ sinks, const GeneralShape sh,
                               const PoolBounds bounds) {
    extern __shared__ float smem[];
    const int Dk = sh.Dk, Dv = sh.Dv;
    float* q_s = smem;                         // [Dk] query times scale
    float* p_s = q_s + Dk;                     // [kWarps][32]
    float* m_s = p_s + kWarps * 32;            // [kWarps]
    float* l_s = m_s + kWarps;                 // [kWarps]
    float* acc_s = l_s + kWarps;               // [kWarps][Dv]

    const int t = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int s = seq_of_token[t];
    const int q0 = cu_q[s], q1 = cu_q[s + 1];
    const int p = kv_len[s] - (q1 - q0) + (t - q0);
    int lo = 0;
    if (sh.window > 0 && p - sh.window + 1 > lo) lo = p - sh.window + 1;
    if (sh.chunk > 0 && (p / sh.chunk) * sh.chunk > lo) lo = (p / sh.chunk) * sh.chunk;
    const int g = h / (sh.Hq / sh.Hkv);
    const int* table = block_table + (size_t)s * sh.table_stride;
    const float slope = slopes ? slopes[h] : 0.0f;

    const float* qv = q + ((size_t)t * sh.Hq + h) * Dk;
    for (int i = threadIdx.x; i < Dk; i += blockDim.x) q_s[i] = qv[i] * sh.scale;
    __syncthreads();

    const float bias = (sh.sigmoid && sh.score_bias) ? sh.score_bias[h] : 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;
    float acc[ACC];
#pragma unroll
    for (int i = 0; i < ACC; ++i) acc[i] = 0.0f;

    const int first_tile = lo >> 5, last_tile = p >> 5;
    const int n_kept = kept_tiles(lo, sh.keep_first);
    const int n_walk = n_kept + last_tile - first_tile + 1;
    for (int idx = warp; idx < n_walk; idx += kWarps) {
        const int tile = idx < n_kept ? idx : first_tile + idx - n_kept;
        const int j = (tile << 5) + lane;
        const bool valid = j <= p && (j >= lo || j < sh.keep_first);
        float sc = -INFINITY;
        if (valid) {
            int page = table[j / sh.page_size];
            if (!page_ok(page, bounds)) page = 0;
            const T* kr = k_pool + (((size_t)page * sh.Hkv + g) * sh.page_size + j % sh.page_size) * sh.k_stride;
            float dot = 0.0f;
            int d = 0;
            for (; d < sh.k_vec; d += Vec<T>::n) {
                float kf[Vec<T>::n];
                load16(kr + d, kf);
#pragma unroll
                for (int e = 0; e < Vec<T>::n; ++e) dot = fmaf(q_s[d + e], kf[e], dot);
            }
            for (; d < Dk; ++d) dot = fmaf(q_s[d], to_float(kr[d]), dot);
            sc = cap_score(dot, sh.softcap) - slope * (float)(p - j);
        }
        float pv;
        if (sh.sigmoid) {                                     // uniform over the grid
            pv = valid ? sigmoid_weight(sc + bias) : 0.0f;
        } else {
            const float m_new = fmaxf(m_run, warp_max(sc));   // finite: every tile in range has a visible key
            pv = valid ? expf(sc - m_new) : 0.0f;
            const float corr = expf(m_run - m_new);           // 0 on the first tile (m_run = -inf)
            l_run = l_run * corr + warp_sum(pv);
            m_run = m_new;
#pragma unroll
            for (int i = 0; i < ACC; ++i) acc[i] *= corr;
        }
        __syncwarp();
        p_s[warp * 32 + lane] = pv;
        __syncwarp();
        const int j0 = tile << 5;
        const int k_end = (p - j0 < 31) ? p - j0 : 31;
        for (int kk = 0; kk <= k_end; ++kk) {
            const int jj = j0 + kk;
            if (jj < lo && jj >= sh.keep_first) continue;      // uniform over the warp
            int page = table[jj / sh.page_size];
            if (!page_ok(page, bounds)) page = 0;
            const T* vr = v_pool + (((size_t)page * (sh.Hkv / sh.v_share) + g / sh.v_share) * sh.page_size + jj % sh.page_size) * sh.v_stride;
            const float pk = p_s[warp * 32 + kk];
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                const int d = lane + 32 * i;
                if (d < Dv) acc[i] = fmaf(pk, to_float(vr[d]), acc[i]);
            }
        }
    }

    if (lane == 0) { m_s[warp] = m_run; l_s[warp] = l_run; }
#pragma unroll
    for (int i = 0; i < ACC; ++i) {
        const int d = lane + 32 * i;
        if (d < Dv) acc_s[warp * Dv + d] = acc[i];
    }
    __syncthreads();
    float m_all = m_s[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) m_all = fmaxf(m_all, m_s[w]);
    float l_all = 0.0f;
    float f[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) { f[w] = (m_s[w] == -INFINITY) ? 0.0f : expf(m_s[w] - m_all); l_all += l_s[w] * f[w]; }
    if (sinks) l_all += expf(sinks[h] - m_all);
    if (sh.sigmoid) {                                         // the warps' sums add up as they are
        l_all = 1.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) f[w] = 1.0f;
    }
    const size_t ov = ((size_t)t * sh.Hq + h) * Dv;
    auto column = [&](int d) {
        float o = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) o += acc_s[w * Dv + d] * f[w];
        return o / l_all;
    };
    for (int d = threadIdx.x; d < Dv; d += blockDim.x) {
        float o = column(d);
        if (sh.out_cos) {
            const size_t at = (size_t)t * (Dv >> 1);
            o = turned_back(o, column(d ^ 1), d >> 1, !(d & 1), sh.out_cos + at, sh.out_sin + at);
        }
        store_out(out, ov + d, o, sh.out_f32);
    }
}

template <typename T, int ACC>
int launch_general(const float* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, const int* cu_q,
                   const int* kv_len, const int* seq_of_token, const float* slopes, const float* sinks, int n_tokens,
                   const GeneralShape& sh, cudaStream_t stream) {
    const size_t smem = sizeof(float) * (sh.Dk + kWarps * 32 + 2 * kWarps + (size_t)kWarps * sh.Dv);
    dim3 grid(n_tokens, sh.Hq);
    paged_attention_general_kernel<T, ACC><<<grid, kWarps * 32, smem, stream>>>(q, (const T*)k_pool, (const T*)v_pool, (T*)out,
        block_table, cu_q, kv_len, seq_of_token, slopes, sinks, sh, pb::pool_bounds_now());
    return launch_status();
}

template <typename T>
int dispatch_general(const float* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, const int* cu_q,
                     const int* kv_len, const int* seq_of_token, const float* slopes, const float* sinks, int n_tokens,
                     GeneralShape sh, cudaStream_t stream) {
    const bool aligned = ((uintptr_t)k_pool % 16 == 0) && ((size_t)sh.k_stride * sizeof(T)) % 16 == 0;
    sh.k_vec = aligned ? sh.Dk - sh.Dk % Vec<T>::n : 0;
#define PB_GENERAL(A) return launch_general<T, A>(q, k_pool, v_pool, out, block_table, cu_q, kv_len, seq_of_token, slopes, sinks, n_tokens, sh, stream)
    if (sh.Dv <= 64) PB_GENERAL(2);
    if (sh.Dv <= 128) PB_GENERAL(4);
    if (sh.Dv <= 256) PB_GENERAL(8);
    if (sh.Dv <= 512) PB_GENERAL(16);
    PB_GENERAL(32);
#undef PB_GENERAL
}

// ---------------------------------------------------------------- the tiled form
// The same arithmetic with the keys and values of a tile staged in shared memory and shared by 16 query rows: the rows of
// a block are consecutive (token, head) pairs of one sequence and one key/value head (index = token * group + head in
// group), so a step of single tokens shares a tile among the heads of a group and a prompt portion among tokens as well.
// Warp w owns rows 4w .. 4w+3; its lane l scores key l of the tile against the four rows (the key's elements come from
// shared memory 16 bytes at a time, the queries by broadcast), the warp reduces maxima and sums over its lanes, and lane l
// then owns value columns l, l + 32, ... of the four rows' outputs.  Tiles of 32 keys are aligned to absolute key
// indices and taken in ascending order; a tile in which a row sees nothing leaves that row's state untouched, so a row's
// result depends on its own position alone.  With splits (grid z) each block takes a contiguous share of the tiles and
// writes (maximum, sum, unnormalised output) per row to a float32 workspace that general_combine_kernel merges in split
// order.  Needs key and value rows that are multiples of 16 bytes; other sizes take the kernel above.
constexpr int kRows = 16;
constexpr int kTile = 32;

struct TiledShape {
    GeneralShape g;
    int n_seqs, n_splits, k_row, v_row;      // rows of the staged tiles in elements (k_row padded; v_row = k_row when the value is part of the key row)
    int v_in_k;
};


template <typename T, int ACC>
__global__ void __launch_bounds__(128)
general_tiled_kernel(const float* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool, T* __restrict__ out,
                     float* __restrict__ partial, const int* __restrict__ block_table, const int* __restrict__ cu_q,
                     const int* __restrict__ kv_len, const float* __restrict__ slopes, const float* __restrict__ sinks,
                     const TiledShape ts, const PoolBounds bounds) {
    pdl_wait();         // may have come onto the SMs while the kernel before it was ending: nothing is touched before that one is done
    constexpr int V = Vec<T>::n;
    const GeneralShape& sh = ts.g;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Dk = sh.Dk, Dv = sh.Dv, GH = sh.Hq / sh.Hkv;
    float* q_s = reinterpret_cast<float*>(smem_raw);                         // [kRows][Dk]
    float* p_s = q_s + kRows * Dk;                                            // [kRows][kTile]
    T* k_s = reinterpret_cast<T*>(p_s + kRows * kTile);                       // [kTile][k_row]
    T* v_s = ts.v_in_k ? k_s : k_s + (size_t)kTile * ts.k_row;                // [kTile][v_row]

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.y, split = blockIdx.z;
    int tile = blockIdx.x, s = 0, q0 = 0, q_len = 0;
    for (; s < ts.n_seqs; ++s) {
        q0 = cu_q[s];
        q_len = cu_q[s + 1] - q0;
        const int nt = (q_len * GH + kRows - 1) / kRows;
        if (tile < nt) break;
        tile -= nt;
    }
    if (s >= ts.n_seqs) return;
    const int ctx0 = kv_len[s] - q_len;
    const int idx0 = tile * kRows;
    const int n_rows = min(kRows, q_len * GH - idx0);
    const int* table = block_table + (size_t)s * sh.table_stride;

    // the block's span of keys: from the lowest key any row sees to the highest
    int lo_blk = 0x7fffffff, hi_blk = 0;
    for (int r = 0; r < n_rows; ++r) {
        const int p = ctx0 + (idx0 + r) / GH;
        int lo = 0;
        if (sh.window > 0 && p - sh.window + 1 > lo) lo = p - sh.window + 1;
        if (sh.chunk > 0 && (p / sh.chunk) * sh.chunk > lo) lo = (p / sh.chunk) * sh.chunk;
        lo_blk = min(lo_blk, lo);
        hi_blk = max(hi_blk, p);
    }
    // the tiles the block walks over, in ascending order: those of kept first keys below the span, then the span's
    const int kt0 = lo_blk / kTile, n_kept = kept_tiles(lo_blk, sh.keep_first);
    const int n_tiles = n_kept + hi_blk / kTile - kt0 + 1;
    const int per = (n_tiles + ts.n_splits - 1) / ts.n_splits;
    const int t_begin = split * per, t_end = min(n_tiles, t_begin + per);

    // this thread's four rows
    int pos[4], lo_r[4], tok[4], head[4];
    float slope[4], bias[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = warp * 4 + r;
        const bool on = row < n_rows;
        const int idx = idx0 + (on ? row : 0);
        tok[r] = q0 + idx / GH;
        head[r] = g * GH + idx % GH;
        pos[r] = on ? ctx0 + idx / GH : -1;                  // -1: sees no key
        int lo = 0;
        if (sh.window > 0 && pos[r] - sh.window + 1 > lo) lo = pos[r] - sh.window + 1;
        if (sh.chunk > 0 && pos[r] >= 0 && (pos[r] / sh.chunk) * sh.chunk > lo) lo = (pos[r] / sh.chunk) * sh.chunk;
        lo_r[r] = lo;
        slope[r] = slopes ? slopes[head[r]] : 0.0f;
        bias[r] = (sh.sigmoid && sh.score_bias) ? sh.score_bias[head[r]] : 0.0f;
    }
    // the rows' queries, 16 bytes at a time, all copies in flight at once (the scale enters with the scores)
    {
        const int q_chunks = Dk / 4;
        for (int c = threadIdx.x; c < kRows * q_chunks; c += blockDim.x) {
            const int row = c / q_chunks, part = c % q_chunks;
            const bool on = row < n_rows;
            const int idx = idx0 + (on ? row : 0);
            const float* src = q + ((size_t)(q0 + idx / GH) * sh.Hq + g * GH + idx % GH) * Dk + part * 4;
            cp_async16(smem_u32(q_s + (size_t)row * Dk + part * 4), src, on);
        }
        cp_async_commit();
    }

    float m_run[4], l_run[4], acc[4][ACC];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m_run[r] = -INFINITY;
        l_run[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < ACC; ++i) acc[r][i] = 0.0f;
    }

    const int k_chunks = Dk / V, v_chunks = Dv / V;
    for (int ti = t_begin; ti < t_end; ++ti) {
        const int kt = ti < n_kept ? ti : kt0 + ti - n_kept;
        const int j0 = kt * kTile;
        __syncthreads();                                   // the tile before is done with
        {
            // four threads per key: one look into the block table, then the row's 16-byte pieces, all in flight at once
            const int key = threadIdx.x >> 2, sub = threadIdx.x & 3;
            const int j = j0 + key;
            const bool ok = j <= hi_blk && (j >= lo_blk || j < sh.keep_first);   // rows outside the block's span are filled with zeros
            const T* k_src = k_pool;
            const T* v_src = v_pool;
            if (ok) {
                int page = table[j / sh.page_size];
                if (!page_ok(page, bounds)) page = 0;
                const size_t at = ((size_t)page * sh.Hkv + g) * sh.page_size + j % sh.page_size;
                const size_t v_at = ((size_t)page * (sh.Hkv / sh.v_share) + g / sh.v_share) * sh.page_size + j % sh.page_size;
                k_src = k_pool + at * sh.k_stride;
                v_src = v_pool + v_at * sh.v_stride;
            }
            for (int part = sub; part < k_chunks; part += 4)
                cp_async16(smem_u32(k_s + (size_t)key * ts.k_row + part * V), k_src + part * V, ok);
            if (!ts.v_in_k)
                for (int part = sub; part < v_chunks; part += 4)
                    cp_async16(smem_u32(v_s + (size_t)key * ts.v_row + part * V), v_src + part * V, ok);
            cp_async_commit();
            cp_async_wait<0>();
        }
        __syncthreads();

        if (warp * 4 >= n_rows) continue;                  // a warp without rows only helps to load (a step of single tokens: the group's heads are all the rows there are)
        // scores of key `lane` against the warp's four rows
        float sc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const T* kr = k_s + (size_t)lane * ts.k_row;
        const float* qr = q_s + (size_t)(warp * 4) * Dk;
        for (int d = 0; d < Dk; d += V) {
            float kf[V];
            load16(kr + d, kf);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
#pragma unroll
                for (int e = 0; e < V; e += 4) {
                    const float4 qv = *reinterpret_cast<const float4*>(qr + r * Dk + d + e);
                    sc[r] = fmaf(qv.x, kf[e], sc[r]);
                    sc[r] = fmaf(qv.y, kf[e + 1], sc[r]);
                    sc[r] = fmaf(qv.z, kf[e + 2], sc[r]);
                    sc[r] = fmaf(qv.w, kf[e + 3], sc[r]);
                }
            }
        }
        const int j = j0 + lane;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const bool vis = j <= pos[r] && (j >= lo_r[r] || j < sh.keep_first);
            const float v = vis ? (sh.softcap > 0.0f ? cap_score(sc[r] * sh.scale, sh.softcap) - slope[r] * (float)(pos[r] - j)
                                                     : fmaf(sc[r], sh.scale, -slope[r] * (float)(pos[r] - j)))
                                : -INFINITY;
            if (sh.sigmoid) {                               // uniform over the grid
                p_s[(warp * 4 + r) * kTile + lane] = vis ? sigmoid_weight(v + bias[r]) : 0.0f;
                continue;
            }
            const float m_new = fmaxf(m_run[r], warp_max(v));
            float pv = 0.0f, corr = 1.0f;
            if (m_new != -INFINITY) {                       // uniform over the warp
                pv = vis ? expf(v - m_new) : 0.0f;
                corr = expf(m_run[r] - m_new);              // 0 while the row had seen nothing
            }
            l_run[r] = l_run[r] * corr + warp_sum(pv);
            m_run[r] = m_new;
            if (corr != 1.0f) {
#pragma unroll
                for (int i = 0; i < ACC; ++i) acc[r][i] *= corr;
            }
            p_s[(warp * 4 + r) * kTile + lane] = pv;
        }
        __syncwarp();
        // outputs: lane owns value columns lane + 32 i of the four rows
        const float* pr = p_s + (warp * 4) * kTile;
        for (int kk = 0; kk < kTile; kk += 4) {
            float4 pw[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) pw[r] = *reinterpret_cast<const float4*>(pr + r * kTile + kk);
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                const int c = lane + 32 * i;
                if (c < Dv) {
                    const float v0 = to_float(v_s[(size_t)(kk + 0) * ts.v_row + c]), v1 = to_float(v_s[(size_t)(kk + 1) * ts.v_row + c]);
                    const float v2 = to_float(v_s[(size_t)(kk + 2) * ts.v_row + c]), v3 = to_float(v_s[(size_t)(kk + 3) * ts.v_row + c]);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        acc[r][i] = fmaf(pw[r].x, v0, acc[r][i]);
                        acc[r][i] = fmaf(pw[r].y, v1, acc[r][i]);
                        acc[r][i] = fmaf(pw[r].z, v2, acc[r][i]);
                        acc[r][i] = fmaf(pw[r].w, v3, acc[r][i]);
                    }
                }
            }
        }
        __syncwarp();
    }

    cp_async_wait<0>();                                    // a block without tiles still has its queries on their way
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (warp * 4 + r >= n_rows) continue;
        const size_t row = (size_t)tok[r] * sh.Hq + head[r];
        if (ts.n_splits == 1) {
            const float inv = sh.sigmoid ? 1.0f : 1.0f / (sinks ? l_run[r] + expf(sinks[head[r]] - m_run[r]) : l_run[r]);
            const size_t at = (size_t)tok[r] * (Dv >> 1);
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                const int c = lane + 32 * i;
                float o = acc[r][i] * inv;
                if (sh.out_cos) {                           // uniform over the grid; the pair's other column is the neighbouring lane's
                    const float other = __shfl_xor_sync(0xffffffffu, o, 1);
                    if (c < Dv) o = turned_back(o, other, c >> 1, !(c & 1), sh.out_cos + at, sh.out_sin + at);
                }
                if (c < Dv) store_out(out, row * Dv + c, o, sh.out_f32);
            }
        } else {
            float* pp = partial + (row * ts.n_splits + split) * (Dv + 2);
            if (lane == 0) { pp[0] = m_run[r]; pp[1] = l_run[r]; }
#pragma unroll
            for (int i = 0; i < ACC; ++i) {
                const int c = lane + 32 * i;
                if (c < Dv) pp[2 + c] = acc[r][i];
            }
        }
    }
}

// out[row] = sum over the splits, in their order, of their partial outputs weighted by exp(m_split - m_all), over the
// weighted sum of their sums.  One block per (token, head).
// (With `sigmoid` the partial outputs are added as they are; a row's columns turn back where the launch says so.)
// Every warp takes the weights of up to 32 splits side by side, a lane one; a thread's columns of those splits are asked for before the
// weights are known, so that one trip to L2 brings all of it.  kSplits (4, 8, 16, 32): the splits a round takes, kCols: the columns a
// thread takes; both no larger than the launch needs, since every round runs through all its places (us with the attention itself, a loop
// over the splits, rounds of 32 with two columns always, now: 128 sequences at 300 keys, 16 heads on one of 32 / 64, 4 splits 29.4,
// 31.3, 27.1; 8 at 500, 128 / 128, 8 splits 24.8, 14.3, 13.4; 32 at 1,000, 16 on one of 576 / 512, 16 splits 111, 43.1, 40.9).
template <typename T, int kSplits, int kCols>
__global__ void general_combine_kernel(const float* __restrict__ partial, T* __restrict__ out, const float* __restrict__ sinks,
                                       int n_splits, const GeneralShape sh) {
    pdl_trigger();
    pdl_wait();
    const size_t row = blockIdx.x;
    const int Hq = sh.Hq, Dv = sh.Dv, lane = threadIdx.x & 31;
    const float* pp = partial + row * n_splits * (Dv + 2);
    float m_all = -INFINITY, l_all = 0.0f;
    if (!sh.sigmoid && n_splits > kSplits) {
        for (int z = lane; z < n_splits; z += 32) m_all = fmaxf(m_all, pp[(size_t)z * (Dv + 2)]);
        m_all = warp_max(m_all);
    }
    float o[kCols];                                          // this thread's columns
#pragma unroll
    for (int i = 0; i < kCols; ++i) o[i] = 0.0f;
    for (int z0 = 0; z0 < n_splits; z0 += kSplits) {
        const int nz = min(kSplits, n_splits - z0);
        float v[kCols][kSplits];
#pragma unroll
        for (int i = 0; i < kCols; ++i) {
            const int c = threadIdx.x + i * blockDim.x;
#pragma unroll
            for (int z = 0; z < kSplits; ++z) v[i][z] = (z < nz && c < Dv) ? pp[(size_t)(z0 + z) * (Dv + 2) + 2 + c] : 0.0f;
        }
        float w = lane < nz ? 1.0f : 0.0f;
        if (!sh.sigmoid) {                                   // uniform over the grid
            const float* mine = pp + (size_t)(z0 + min(lane, nz - 1)) * (Dv + 2);
            const float m = lane < nz ? mine[0] : -INFINITY, l = mine[1];
            if (n_splits <= kSplits) m_all = warp_max(m);
            w = m != -INFINITY ? expf(m - m_all) : 0.0f;
            l_all += warp_sum(w != 0.0f ? l * w : 0.0f);
        }
#pragma unroll
        for (int z = 0; z < kSplits; ++z) {
            const float wz = __shfl_sync(0xffffffffu, w, z);
            if (wz != 0.0f) {                                // uniform over the warp
#pragma unroll
                for (int i = 0; i < kCols; ++i) o[i] = fmaf(v[i][z], wz, o[i]);
            }
        }
    }
    if (sh.sigmoid) l_all = 1.0f;
    else if (sinks) l_all += expf(sinks[row % Hq] - m_all);
#pragma unroll
    for (int i = 0; i < kCols; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        float v = o[i] / l_all;
        if (sh.out_cos) {                                    // uniform over the grid; the pair's other column is the neighbouring lane's
            const float other = __shfl_xor_sync(0xffffffffu, v, 1);
            const size_t at = row / Hq * (Dv >> 1);
            if (c < Dv) v = turned_back(v, other, c >> 1, !(c & 1), sh.out_cos + at, sh.out_sin + at);
        }
        if (c < Dv) store_out(out, row * Dv + c, v, sh.out_f32);
    }
}

// ---------------------------------------------------------------- the tiled form on the tensor cores
// The same blocks, tiles, splits and partial results as above for bfloat16 pools, with both products on mma.sync (m16n8k16: a
// block's 16 rows are one fragment).  Queries and softmax weights keep their 24 bits: each is the sum of three bfloat16 numbers
// (x = hi + mid + lo, exact to float32's last bit or one below) and every product is three MMAs into one float32 accumulator;
// keys and values are bfloat16 in the cache and exact as they are.  Where the time went before: shared memory, which a
// multiply-add on the CUDA cores reads half a word for; the matrix instruction reads a staged row once per 16 rows.
// The four warps share the key's width for the scores (a warp holds its share of the 16 queries in registers from the start, KS
// steps of 16 elements, and adds its part to the others' through shared memory, in warp order) and the value's width for the
// outputs (VT tiles of 8 columns).  Every warp takes the same softmax.  Tiles are fetched one ahead.
constexpr int kSRow = kTile + 4;        // floats of a row of partial scores

// x as a sum of three bfloat16 pairs: element pairs packed as mma wants them.  An infinite number is its own first part and
// has nothing left.  kLarge: x may be a finite number above bfloat16's largest, which would round to infinity (queries; softmax
// weights are at most one).
__device__ __forceinline__ float to_bf16_range(float x) {
    constexpr float most = 3.3895313892515355e38f;          // bfloat16's largest
    return fabsf(x) < INFINITY ? fminf(fmaxf(x, -most), most) : x;      // (what is no number stays none)
}
template <bool kLarge>
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = kLarge ? pack_bf16(to_bf16_range(x), to_bf16_range(y)) : pack_bf16(x, y);
    x = fabsf(x) == INFINITY ? 0.0f : x - __uint_as_float(hi << 16);
    y = fabsf(y) == INFINITY ? 0.0f : y - __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(x, y);
    x -= __uint_as_float(mid << 16);
    y -= __uint_as_float(mid & 0xffff0000u);
    lo = pack_bf16(x, y);
}

// A product from its first part and the rest.  An infinite key or value makes the first part what the whole product is; the rest, where
// it meets zeros and numbers of the other sign, is then NaN or infinite itself and says nothing.
__device__ __forceinline__ float with_rest(float first, float rest) { return fabsf(first) == INFINITY ? first : first + rest; }

template <int KS, int VT>
__global__ void __launch_bounds__(128)
general_rows_tc_kernel(const float* __restrict__ q, const bf16* __restrict__ k_pool, const bf16* __restrict__ v_pool, bf16* __restrict__ out,
                       float* __restrict__ partial, const int* __restrict__ block_table, const int* __restrict__ cu_q,
                       const int* __restrict__ kv_len, const float* __restrict__ slopes, const float* __restrict__ sinks,
                       const TiledShape ts, const PoolBounds bounds) {
    pdl_wait();
    const GeneralShape& sh = ts.g;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Dk = sh.Dk, Dv = sh.Dv, GH = sh.Hq / sh.Hkv;
    float* s_s = reinterpret_cast<float*>(smem_raw);                          // [4 warps][kRows][kSRow] partial scores
    bf16* kv_s = reinterpret_cast<bf16*>(s_s + 4 * kRows * kSRow);            // two stages of [kTile][k_row] (and [kTile][v_row])
    const size_t stage = (size_t)kTile * (ts.k_row + (ts.v_in_k ? 0 : ts.v_row));

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.y, split = blockIdx.z;
    int tile = blockIdx.x, s = 0, q0 = 0, q_len = 0;
    for (; s < ts.n_seqs; ++s) {
        q0 = cu_q[s];
        q_len = cu_q[s + 1] - q0;
        const int nt = (q_len * GH + kRows - 1) / kRows;
        if (tile < nt) break;
        tile -= nt;
    }
    if (s >= ts.n_seqs) return;
    const int ctx0 = kv_len[s] - q_len;
    const int idx0 = tile * kRows;
    const int n_rows = min(kRows, q_len * GH - idx0);
    const int* table = block_table + (size_t)s * sh.table_stride;

    // the block's span of keys: lowest keys ascend with the rows' positions, so the first row sees the lowest key, the last the highest
    auto lowest = [&](int p) {
        int lo = 0;
        if (sh.window > 0 && p - sh.window + 1 > lo) lo = p - sh.window + 1;
        if (sh.chunk > 0 && (p / sh.chunk) * sh.chunk > lo) lo = (p / sh.chunk) * sh.chunk;
        return lo;
    };
    const int lo_blk = lowest(ctx0 + idx0 / GH), hi_blk = ctx0 + (idx0 + n_rows - 1) / GH;
    const int kt0 = lo_blk / kTile, n_kept = kept_tiles(lo_blk, sh.keep_first);
    const int n_tiles = n_kept + hi_blk / kTile - kt0 + 1;
    const int per = (n_tiles + ts.n_splits - 1) / ts.n_splits;
    const int t_begin = split * per, t_end = min(n_tiles, t_begin + per);

    auto load = [&](int ti) {
        const int j0 = (ti < n_kept ? ti : kt0 + ti - n_kept) * kTile;
        bf16* k_s = kv_s + (ti & 1) * stage;
        bf16* v_s = k_s + (size_t)kTile * ts.k_row;
        const int key = threadIdx.x >> 2, sub = threadIdx.x & 3, j = j0 + key;
        const bool ok = j <= hi_blk && (j >= lo_blk || j < sh.keep_first);   // rows outside the block's span are filled with zeros
        const bf16* k_src = k_pool;
        const bf16* v_src = v_pool;
        if (ok) {
            int page = table[j / sh.page_size];
            if (!page_ok(page, bounds)) page = 0;
            k_src += (((size_t)page * sh.Hkv + g) * sh.page_size + j % sh.page_size) * sh.k_stride;
            v_src += (((size_t)page * (sh.Hkv / sh.v_share) + g / sh.v_share) * sh.page_size + j % sh.page_size) * sh.v_stride;
        }
        for (int part = sub; part < Dk / 8; part += 4) cp_async16(smem_u32(k_s + (size_t)key * ts.k_row + part * 8), k_src + part * 8, ok);
        if (!ts.v_in_k)
            for (int part = sub; part < Dv / 8; part += 4) cp_async16(smem_u32(v_s + (size_t)key * ts.v_row + part * 8), v_src + part * 8, ok);
    };
    if (t_begin < t_end) load(t_begin);
    cp_async_commit();

    // this thread's two rows of the fragments
    int pos[2], lo_r[2], tok[2], head[2];
    float slope[2], bias[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = (lane >> 2) + 8 * r;
        const bool on = row < n_rows;
        const int idx = idx0 + (on ? row : 0);
        tok[r] = q0 + idx / GH;
        head[r] = g * GH + idx % GH;
        pos[r] = on ? ctx0 + idx / GH : -1;                  // -1: sees no key
        lo_r[r] = on ? lowest(pos[r]) : 0;
        slope[r] = slopes ? slopes[head[r]] : 0.0f;
        bias[r] = (sh.sigmoid && sh.score_bias) ? sh.score_bias[head[r]] : 0.0f;
    }
    // this warp's share of the queries, split: [step][a register of the fragment: (row, row + 8) x (8 columns, the next 8)]
    const int steps = Dk / 16;
    uint32_t qf[3][KS][4];
#pragma unroll
    for (int i = 0; i < KS; ++i) {
        const int ks = warp * KS + i;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const int r = f & 1, col = ks * 16 + (f >> 1) * 8 + (lane & 3) * 2;
            float2 v = make_float2(0.0f, 0.0f);
            if (ks < steps && pos[r] >= 0) v = *reinterpret_cast<const float2*>(q + ((size_t)tok[r] * sh.Hq + head[r]) * Dk + col);
            split3<true>(v.x, v.y, qf[0][i][f], qf[1][i][f], qf[2][i][f]);
        }
    }

    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f}, acc[VT][4];
#pragma unroll
    for (int i = 0; i < VT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.0f;

    for (int ti = t_begin; ti < t_end; ++ti) {
        cp_async_wait<0>();
        __syncthreads();                                   // the tile has landed; the one before it, and its scores, are done with
        if (ti + 1 < t_end) load(ti + 1);
        cp_async_commit();
        const int j0 = (ti < n_kept ? ti : kt0 + ti - n_kept) * kTile;
        const bf16* k_s = kv_s + (ti & 1) * stage;
        const bf16* v_s = ts.v_in_k ? k_s : k_s + (size_t)kTile * ts.k_row;

        // this warp's part of the scores of 32 keys; the queries' first parts and the small rest in accumulators of their own
        // (an MMA cuts off what falls below its accumulator's last bits)
        float sc[4][4], sr[4][4];
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[n][e] = sr[n][e] = 0.0f;
#pragma unroll
        for (int i = 0; i < KS; ++i) {
            const int ks = warp * KS + i;
            if (ks < steps) {                               // uniform over the warp
#pragma unroll
                for (int n2 = 0; n2 < 2; ++n2) {
                    uint32_t b[4];                          // keys 16 n2 .. + 7: two registers, the next 8 keys: two more
                    const int key = n2 * 16 + (lane & 7) + (lane >> 4) * 8, col = ks * 16 + (lane >> 3 & 1) * 8;
                    ldmatrix_x4(b, smem_u32(k_s + (size_t)key * ts.k_row + col));
#pragma unroll
                    for (int p = 2; p >= 0; --p) {
                        mma_bf16(p ? sr[2 * n2] : sc[2 * n2], qf[p][i], b[0], b[1]);
                        mma_bf16(p ? sr[2 * n2 + 1] : sc[2 * n2 + 1], qf[p][i], b[2], b[3]);
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                *reinterpret_cast<float2*>(s_s + (warp * kRows + (lane >> 2) + 8 * r) * kSRow + n * 8 + (lane & 3) * 2) =
                    make_float2(with_rest(sc[n][2 * r], sr[n][2 * r]), with_rest(sc[n][2 * r + 1], sr[n][2 * r + 1]));
        __syncthreads();

        // the softmax weights of this thread's two rows: keys 8 n + 2 (lane mod 4) + {0, 1}, the columns of the scores' fragments
        float pw[4][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float m_tile = -INFINITY;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float2 x = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const float2 y = *reinterpret_cast<const float2*>(s_s + (w * kRows + (lane >> 2) + 8 * r) * kSRow + n * 8 + (lane & 3) * 2);
                    x.x += y.x;
                    x.y += y.y;
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int j = j0 + n * 8 + (lane & 3) * 2 + e;
                    const float raw = e ? x.y : x.x;
                    const bool vis = j <= pos[r] && (j >= lo_r[r] || j < sh.keep_first);
                    const float v = vis ? (sh.softcap > 0.0f ? cap_score(raw * sh.scale, sh.softcap) - slope[r] * (float)(pos[r] - j)
                                                             : fmaf(raw, sh.scale, -slope[r] * (float)(pos[r] - j)))
                                        : -INFINITY;
                    pw[n][2 * r + e] = v;
                    m_tile = fmaxf(m_tile, v);
                }
            }
            if (sh.sigmoid) {                               // uniform over the grid
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float v = pw[n][2 * r + e];
                        pw[n][2 * r + e] = v == -INFINITY ? 0.0f : sigmoid_weight(v + bias[r]);
                    }
                continue;
            }
            m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 1));
            m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 2));
            const float m_new = fmaxf(m_run[r], m_tile);
            float corr = 1.0f, sum = 0.0f;
            if (m_new != -INFINITY) corr = expf(m_run[r] - m_new);      // 0 while the row had seen nothing
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float v = pw[n][2 * r + e];
                    const float p = v == -INFINITY ? 0.0f : expf(v - m_new);
                    pw[n][2 * r + e] = p;
                    sum += p;
                }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l_run[r] = l_run[r] * corr + sum;
            m_run[r] = m_new;
            if (corr != 1.0f) {
#pragma unroll
                for (int i = 0; i < VT; ++i) {
                    acc[i][2 * r] *= corr;
                    acc[i][2 * r + 1] *= corr;
                }
            }
        }
        // outputs: this warp's columns.  A tile's sums begin at zero and join the others in an addition of their own, rounded to
        // nearest: the MMAs' cut-off would add up over a long row of keys.
        uint32_t pf[2][3][4];                               // [16 keys][part][register: (row, row + 8) of the first 8 keys, of the next 8]
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2)
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const int n = 2 * k2 + (f >> 1), r = f & 1;
                split3<false>(pw[n][2 * r], pw[n][2 * r + 1], pf[k2][0][f], pf[k2][1][f], pf[k2][2][f]);
            }
#pragma unroll
        for (int i = 0; i < VT; i += 2) {
            const int col = (warp * VT + i) * 8;
            if (col >= Dv) break;                           // uniform over the warp; Dv is a multiple of 16
            float o[2][4], rest[2][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[0][e] = o[1][e] = rest[0][e] = rest[1][e] = 0.0f;
#pragma unroll
            for (int k2 = 0; k2 < 2; ++k2) {
                uint32_t b[4];                              // columns col .. + 7: two registers (8 keys each), the next 8 columns: two more
                const int key = k2 * 16 + (lane & 7) + (lane >> 3 & 1) * 8;
                ldmatrix_x4_trans(b, smem_u32(v_s + (size_t)key * ts.v_row + col + (lane >> 4) * 8));
#pragma unroll
                for (int p = 2; p >= 0; --p) {
                    mma_bf16(p ? rest[0] : o[0], pf[k2][p], b[0], b[1]);
                    mma_bf16(p ? rest[1] : o[1], pf[k2][p], b[2], b[3]);
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[i][e] += with_rest(o[0][e], rest[0][e]);
                acc[i + 1][e] += with_rest(o[1][e], rest[1][e]);
            }
        }
    }
    cp_async_wait<0>();
    pdl_trigger();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (pos[r] < 0) continue;
        const size_t row = (size_t)tok[r] * sh.Hq + head[r];
        if (ts.n_splits == 1) {
            const float inv = sh.sigmoid ? 1.0f : 1.0f / (sinks ? l_run[r] + expf(sinks[head[r]] - m_run[r]) : l_run[r]);
            const size_t at = (size_t)tok[r] * (Dv >> 1);
#pragma unroll
            for (int i = 0; i < VT; ++i) {
                const int c = (warp * VT + i) * 8 + (lane & 3) * 2;
                if (c >= Dv) break;
                float u = acc[i][2 * r] * inv, v = acc[i][2 * r + 1] * inv;
                if (sh.out_cos) {                           // uniform over the grid; both columns of a pair are this thread's
                    const float a = turned_back(u, v, c >> 1, 1, sh.out_cos + at, sh.out_sin + at);
                    v = turned_back(v, u, c >> 1, 0, sh.out_cos + at, sh.out_sin + at);
                    u = a;
                }
                store_out(out, row * Dv + c, u, sh.out_f32);
                store_out(out, row * Dv + c + 1, v, sh.out_f32);
            }
        } else {
            float* pp = partial + (row * ts.n_splits + split) * (Dv + 2);
            if (warp == 0 && (lane & 3) == 0) { pp[0] = m_run[r]; pp[1] = l_run[r]; }
#pragma unroll
            for (int i = 0; i < VT; ++i) {
                const int c = (warp * VT + i) * 8 + (lane & 3) * 2;
                if (c >= Dv) break;
                *reinterpret_cast<float2*>(pp + 2 + c) = make_float2(acc[i][2 * r], acc[i][2 * r + 1]);
            }
        }
    }
}

// Shared memory of the kernel above; 0 where it does not take the sizes (key and value widths in steps of 16 up to 576 and 512).
size_t rows_tc_smem(const TiledShape& ts) {
    const GeneralShape& sh = ts.g;
    if (sh.Dk % 16 || sh.Dv % 16 || sh.Dk > 576 || sh.Dv > 512) return 0;
    return sizeof(float) * 4 * kRows * kSRow + 2 * sizeof(bf16) * kTile * ((size_t)ts.k_row + (ts.v_in_k ? 0 : ts.v_row));
}

template <int KS, int VT>
int launch_rows_tc(const float* q, const void* k_pool, const void* v_pool, void* out, float* partial, const int* block_table,
                   const int* cu_q, const int* kv_len, const float* slopes, const float* sinks, int row_tiles, const TiledShape& ts,
                   size_t smem, cudaStream_t stream) {
    static SmemLimit limit;
    if (const int rc = limit.allow(general_rows_tc_kernel<KS, VT>, 200 * 1024)) return rc;
    return launch_pdl(general_rows_tc_kernel<KS, VT>, dim3(row_tiles, ts.g.Hkv, ts.n_splits), dim3(128), smem, stream, q, (const bf16*)k_pool,
                      (const bf16*)v_pool, (bf16*)out, partial, block_table, cu_q, kv_len, slopes, sinks, ts, pb::pool_bounds_now());
}

template <typename T>
size_t tiled_smem(const TiledShape& ts) {
    return sizeof(float) * (kRows * ts.g.Dk + kRows * kTile) + sizeof(T) * kTile * ((size_t)ts.k_row + (ts.v_in_k ? 0 : ts.v_row));
}

template <typename T, int ACC>
int launch_tiled(const float* q, const void* k_pool, const void* v_pool, void* out, float* partial, const int* block_table,
                 const int* cu_q, const int* kv_len, const float* slopes, const float* sinks, int row_tiles, const TiledShape& ts,
                 cudaStream_t stream) {
    const size_t smem = tiled_smem<T>(ts);
    static SmemLimit limit;
    if (const int rc = limit.allow(general_tiled_kernel<T, ACC>, smem)) return rc;
    dim3 grid(row_tiles, ts.g.Hkv, ts.n_splits);
    return launch_pdl(general_tiled_kernel<T, ACC>, grid, dim3(128), smem, stream, q, (const T*)k_pool, (const T*)v_pool, (T*)out, partial,
                      block_table, cu_q, kv_len, slopes, sinks, ts, pb::pool_bounds_now());
}

template <typename T>
bool tiled_shape(TiledShape& ts, const void* k_pool, const void* v_pool) {
    const GeneralShape& sh = ts.g;
    const size_t e = sizeof(T);
    if ((sh.Dk * e) % 16 || (sh.Dv * e) % 16 || (sh.k_stride * e) % 16 || (sh.v_stride * e) % 16) return false;
    if (((uintptr_t)k_pool | (uintptr_t)v_pool) % 16) return false;
    ts.v_in_k = (k_pool == v_pool && sh.k_stride == sh.v_stride && sh.Dv <= sh.Dk) ? 1 : 0;
    const int unit = 16 / (int)e;                           // elements in 16 bytes
    int k_units = sh.Dk / unit;
    if (k_units % 2 == 0) ++k_units;                        // rows an odd number of 16-byte units apart: lanes on different rows do not collide
    ts.k_row = k_units * unit;
    ts.v_row = ts.v_in_k ? ts.k_row : sh.Dv;
    return tiled_smem<T>(ts) <= 200 * 1024;
}

template <typename T>
int dispatch_tiled(const float* q, const void* k_pool, const void* v_pool, void* out, float* partial, const int* block_table,
                   const int* cu_q, const int* kv_len, const float* slopes, const float* sinks, int row_tiles, const TiledShape& ts,
                   cudaStream_t stream) {
#define PB_TILED(A) return launch_tiled<T, A>(q, k_pool, v_pool, out, partial, block_table, cu_q, kv_len, slopes, sinks, row_tiles, ts, stream)
    if (ts.g.Dv <= 64) PB_TILED(2);
    if (ts.g.Dv <= 128) PB_TILED(4);
    if (ts.g.Dv <= 256) PB_TILED(8);
    PB_TILED(16);
#undef PB_TILED
}

// bfloat16 pools take the tensor-core form where it takes the widths, else the CUDA-core form.  us with the merge, CUDA cores -> tensor
// cores, 8 sequences at 1,900 keys: 16 heads on one row of 576 / 512, 32 splits 60.5 -> 22.7; 16 on 4 heads of 128 / 128, chunks of
// 1,024, 16 splits 26.7 -> 15.1; the smallest (2 sequences, 8 heads on 4 of 64 / 64, 90 and 333 keys) 7.6 -> 8.2.  Relative error of
// float32 rows against 64 bits on the first: 5.7e-7 -> 2.0e-7.
// Keys of 32 and fewer with fewer than four heads to a key/value head stay on the CUDA cores: so few sums a tile do not pay for the
// tensor-core form's larger blocks once these fill the SMs (4 heads of 32 / 32, 32 sequences at 1,000 keys 32.7 against 34.7, 128 at 300
// 42.1 against 47.1; one at 1,000 9.9 against 10.9).  With four heads or more, and from keys of 48 on, it is level or ahead.
int dispatch_tiled_bf16(const float* q, const void* k_pool, const void* v_pool, void* out, float* partial, const int* block_table,
                        const int* cu_q, const int* kv_len, const float* slopes, const float* sinks, int row_tiles, TiledShape ts,
                        cudaStream_t stream) {
    const int v_row = ts.v_row;
    if (!ts.v_in_k) ts.v_row = (ts.g.Dv / 8 | 1) * 8;       // value rows an odd number of 16-byte units apart as well
    const size_t smem = rows_tc_smem(ts);
#define PB_ROWS_TC(K, V) return launch_rows_tc<K, V>(q, k_pool, v_pool, out, partial, block_table, cu_q, kv_len, slopes, sinks, row_tiles, ts, smem, stream)
    const bool thin = ts.g.Dk <= 32 && ts.g.Hq / ts.g.Hkv < 4;
    if (smem > 0 && smem <= 200 * 1024 && !thin && (uintptr_t)partial % 8 == 0) {        // partial results are written two floats at a time
        if (ts.g.Dk <= 128 && ts.g.Dv <= 128) PB_ROWS_TC(2, 4);
        if (ts.g.Dk <= 192 && ts.g.Dv <= 128) PB_ROWS_TC(3, 4);
        if (ts.g.Dk <= 320 && ts.g.Dv <= 256) PB_ROWS_TC(5, 8);
        PB_ROWS_TC(9, 16);
    }
#undef PB_ROWS_TC
    ts.v_row = v_row;
    return dispatch_tiled<bf16>(q, k_pool, v_pool, out, partial, block_table, cu_q, kv_len, slopes, sinks, row_tiles, ts, stream);
}

template <typename T>
int launch_combine(const float* partial, void* out, const float* sinks, int n_tokens, const TiledShape& ts, cudaStream_t stream) {
    int b = 32;
    while (b < ts.g.Dv && b < 256) b <<= 1;
#define PB_COMBINE(S, C) return launch_pdl(general_combine_kernel<T, S, C>, dim3(n_tokens * ts.g.Hq), dim3(b), 0, stream, partial, (T*)out, sinks, ts.n_splits, ts.g)
#define PB_COMBINE_COLS(C) { if (ts.n_splits <= 4) PB_COMBINE(4, C); if (ts.n_splits <= 8) PB_COMBINE(8, C); if (ts.n_splits <= 16) PB_COMBINE(16, C); PB_COMBINE(32, C); }
    if (ts.g.Dv <= b) PB_COMBINE_COLS(1)
    PB_COMBINE_COLS(2)                                      // widths up to 512 in blocks of 256
#undef PB_COMBINE_COLS
#undef PB_COMBINE
}

// One warp per (token, head) of the fused projection row [q: Hq*Dk | k: Hk*Dk | v: Hv*Dv]:
// queries to float32 [N, Hq, Dk], keys and values into the pages of the token's slot (pools of Hk and of Hv heads).
// With temp_coef != 0 a query at position p is multiplied by 1 + temp_coef * ln(floor((p + 1) / temp_every) + 1).
template <typename T>
__global__ void qkv_split_write_kernel(const T* __restrict__ qkv, float* __restrict__ q_out, T* __restrict__ k_pool,
                                       T* __restrict__ v_pool, const int* __restrict__ slots, int Hq, int Hk, int Hv, int Dk, int Dv,
                                       int page_size, const int* __restrict__ positions, float temp_coef, int temp_every,
                                       const PoolBounds bounds) {
    // A short kernel: the next one may fetch its weights now.  Not where the blocks come in rounds: the next kernel could only come in
    // the last one, and what every block pays for the word adds up (us, 48 heads of 64 and 16 of 128: 2,048 tokens 21.4 without, 35.6
    // with it; 256 tokens, 4,096 blocks, 5.1 and 6.1; 64 tokens, 1,024 blocks, 3.4 either way).
    if (gridDim.x * gridDim.y <= 16 * 148) pdl_trigger();
    pdl_wait();         // may have come onto the SMs while the product before it was ending: nothing is touched before that one is done
    const int t = blockIdx.x, lane = threadIdx.x & 31;
    const int head = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (head >= Hq + Hk + Hv) return;
    const size_t row = (size_t)Hq * Dk + (size_t)Hk * Dk + (size_t)Hv * Dv;
    const T* base = qkv + (size_t)t * row;
    if (head < Hq) {
        const T* src = base + (size_t)head * Dk;
        float* dst = q_out + ((size_t)t * Hq + head) * Dk;
        float f = 1.0f;
        if (temp_coef != 0.0f) f = 1.0f + temp_coef * logf((float)((positions[t] + 1) / temp_every + 1));
        for (int i = lane; i < Dk; i += 32) dst[i] = to_float(src[i]) * f;
        return;
    }
    const int slot = slots[t];
    if (slot < 0 || !slot_ok(slot, page_size, bounds)) return;
    const bool is_k = head < Hq + Hk;
    const int kvh = is_k ? head - Hq : head - Hq - Hk;
    const int D = is_k ? Dk : Dv, Hp = is_k ? Hk : Hv;
    const T* src = base + (size_t)Hq * Dk + (is_k ? (size_t)kvh * Dk : (size_t)Hk * Dk + (size_t)kvh * Dv);
    T* dst = (is_k ? k_pool : v_pool) + (((size_t)(slot / page_size) * Hp + kvh) * page_size + slot % page_size) * D;
    for (int i = lane; i < D; i += 32) dst[i] = src[i];
}

// Sigmoid weights have no denominator that a sink could join; turning back pairs the columns of a row.
bool weighting_ok(int sigmoid, const float* score_bias, const float* sinks, const float* out_cos, const float* out_sin, int Dv) {
    return !(sigmoid && sinks) && !(score_bias && !sigmoid) && ((out_cos == nullptr) == (out_sin == nullptr)) && !(out_cos && Dv % 2);
}

}  // namespace

// sigmoid, score_bias (float32 [Hq] or null), out_cos / out_sin (float32 [n_tokens, Dv / 2] or null): see the head of this file.
PB_EXPORT int pb_paged_attention_general(int dtype, const float* q, const void* k_pool, const void* v_pool, void* out,
                                         const int* block_table, int table_stride, const int* cu_q, const int* kv_len,
                                         const int* seq_of_token, const float* slopes, int n_tokens, int Hq, int Hkv, int Dk,
                                         int Dv, int k_stride, int v_stride, int page_size, float scale, int window, int chunk,
                                         int keep_first, float softcap, const float* sinks, int v_share, int out_f32, int sigmoid,
                                         const float* score_bias, const float* out_cos, const float* out_sin, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (!weighting_ok(sigmoid, score_bias, sinks, out_cos, out_sin, Dv)) return PB_ERR_BAD_SIZE;
    if (Dk <= 0 || Dv <= 0 || Dk > 4096 || Dv > 1024 || Hkv <= 0 || Hq <= 0 || Hq % Hkv || page_size <= 0 || k_stride < Dk ||
        v_stride < Dv || window < 0 || chunk < 0 || keep_first < 0 || !(softcap >= 0.0f) || v_share <= 0 || Hkv % v_share)
        return PB_ERR_BAD_SIZE;
    if (Hq > 65535) return PB_ERR_TOO_LARGE;
    GeneralShape sh{Hq, Hkv, Dk, Dv, k_stride, v_stride, page_size, window, chunk, table_stride, 0, scale, keep_first, softcap, v_share,
                    out_f32 != 0, sigmoid != 0, score_bias, out_cos, out_sin};
    if (dtype == PB_F32)
        return dispatch_general<float>(q, k_pool, v_pool, out, block_table, cu_q, kv_len, seq_of_token, slopes, sinks, n_tokens, sh,
                                       stream);
    if (dtype == PB_BF16)
        return dispatch_general<__nv_bfloat16>(q, k_pool, v_pool, out, block_table, cu_q, kv_len, seq_of_token, slopes, sinks, n_tokens,
                                               sh, stream);
    return PB_ERR_BAD_DTYPE;
}

PB_EXPORT int pb_qkv_split_write(int dtype, const void* qkv, float* q_out, void* k_pool, void* v_pool, const int* slots,
                                 int n_tokens, int Hq, int Hk, int Hv, int Dk, int Dv, int page_size, const int* positions,
                                 float temp_coef, int temp_every, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (Hq <= 0 || Hk < 0 || Hv < 0 || Dk <= 0 || Dv <= 0 || page_size <= 0) return PB_ERR_BAD_SIZE;
    if (temp_coef != 0.0f && (positions == nullptr || temp_every <= 0)) return PB_ERR_BAD_SIZE;
    const int heads = Hq + Hk + Hv;
    dim3 grid(n_tokens, (heads + 3) / 4);
    if (dtype == PB_F32)
        launch_pdl(qkv_split_write_kernel<float>, grid, 128, 0, stream, (const float*)qkv, q_out, (float*)k_pool, (float*)v_pool, slots, Hq,
                                                                Hk, Hv, Dk, Dv, page_size, positions, temp_coef, temp_every, pb::pool_bounds_now());
    else if (dtype == PB_BF16)
        launch_pdl(qkv_split_write_kernel<__nv_bfloat16>, grid, 128, 0, stream, (const __nv_bfloat16*)qkv, q_out, (__nv_bfloat16*)k_pool,
                                                                        (__nv_bfloat16*)v_pool, slots, Hq, Hk, Hv, Dk, Dv, page_size,
                                                                        positions, temp_coef, temp_every, pb::pool_bounds_now());
    else return PB_ERR_BAD_DTYPE;
    return launch_status();
}

PB_EXPORT int pb_attention_general_tiled_supported(int dtype, const void* k_pool, const void* v_pool, int Hq, int Hkv, int Dk, int Dv,
                                                   int k_stride, int v_stride) {
    if (Dk <= 0 || Dv <= 0 || Dv > 512 || Hkv <= 0 || Hq <= 0 || Hq % Hkv || k_stride < Dk || v_stride < Dv) return 0;
    TiledShape ts{};
    ts.g = GeneralShape{Hq, Hkv, Dk, Dv, k_stride, v_stride, 1, 0, 0, 0, 0, 1.0f, 0, 0.0f, 1};
    if (dtype == PB_F32) return tiled_shape<float>(ts, k_pool, v_pool) ? 1 : 0;
    if (dtype == PB_BF16) return tiled_shape<__nv_bfloat16>(ts, k_pool, v_pool) ? 1 : 0;
    return 0;
}

// The tiled form of pb_paged_attention_general.  row_tiles: the sum over the sequences of ceil(new tokens * (Hq / Hkv) / 16).
// n_splits > 1 needs `partial`: float32, n_tokens * Hq * n_splits * (Dv + 2) elements.
PB_EXPORT int pb_paged_attention_general_tiled(int dtype, const float* q, const void* k_pool, const void* v_pool, void* out,
                                               float* partial, const int* block_table, int table_stride, const int* cu_q,
                                               const int* kv_len, const float* slopes, int n_tokens, int n_seqs, int row_tiles,
                                               int n_splits, int Hq, int Hkv, int Dk, int Dv, int k_stride, int v_stride,
                                               int page_size, float scale, int window, int chunk, int keep_first, float softcap,
                                               const float* sinks, int v_share, int out_f32, int sigmoid, const float* score_bias,
                                               const float* out_cos, const float* out_sin, cudaStream_t stream) {
    if (n_tokens <= 0 || row_tiles <= 0) return 0;
    if (!weighting_ok(sigmoid, score_bias, sinks, out_cos, out_sin, Dv)) return PB_ERR_BAD_SIZE;
    if (v_share <= 0 || Hkv % v_share) return PB_ERR_BAD_SIZE;
    if (!pb_attention_general_tiled_supported(dtype, k_pool, v_pool, Hq, Hkv, Dk, Dv, k_stride, v_stride)) return PB_ERR_BAD_SIZE;
    if (page_size <= 0 || window < 0 || chunk < 0 || keep_first < 0 || !(softcap >= 0.0f) || n_splits < 1 || n_splits > 65535 ||
        (n_splits > 1 && partial == nullptr) || (uintptr_t)q % 16)
        return PB_ERR_BAD_SIZE;
    if (Hkv > 65535) return PB_ERR_TOO_LARGE;
    TiledShape ts{};
    ts.g = GeneralShape{Hq, Hkv, Dk, Dv, k_stride, v_stride, page_size, window, chunk, table_stride, 0, scale, keep_first, softcap, v_share,
                        out_f32 != 0, sigmoid != 0, score_bias, out_cos, out_sin};
    ts.n_seqs = n_seqs;
    ts.n_splits = n_splits;
    int status;
    if (dtype == PB_F32) {
        tiled_shape<float>(ts, k_pool, v_pool);
        status = dispatch_tiled<float>(q, k_pool, v_pool, out, partial, block_table, cu_q, kv_len, slopes, sinks, row_tiles, ts, stream);
        if (status == 0 && n_splits > 1) status = launch_combine<float>(partial, out, sinks, n_tokens, ts, stream);
    } else {
        tiled_shape<bf16>(ts, k_pool, v_pool);
        status = dispatch_tiled_bf16(q, k_pool, v_pool, out, partial, block_table, cu_q, kv_len, slopes, sinks, row_tiles, ts, stream);
        if (status == 0 && n_splits > 1) status = launch_combine<bf16>(partial, out, sinks, n_tokens, ts, stream);
    }
    return status;
}
