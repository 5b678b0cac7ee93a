// Paged attention for any batch of query tokens: prompt portions and single decoded
// tokens side by side, causal, optional sliding window, grouped-query heads, any head
// size that is a multiple of 16 up to 256, float32 or bfloat16 storage.
//
// This is the exact kernel of the engine: scores, running maximum, sums and the output
// accumulate in float32 with expf.  The reduction order of a (token, head) pair depends
// only on that token's position (key tiles of 32 aligned to absolute key indices, tile i
// handled by warp i mod 4, the warps' shares combined from that of the row's first tile
// on), so logits do not depend on how tokens were cut into steps or batched.  The float32
// path of the model runs it for every step but those of single tokens (the split-key
// decode attention); the bfloat16 path uses it wherever no tensor-core kernel applies.
//
// Role in the reference: pulsar-core/src/kernels/paged_common.cu:21-142
// (attn_scalar_kernel, one CTA per (query token, q head), online softmax).  Unlike it,
// keys are stored rotated and are not rotated again on read, and partial results are
// combined in a fixed order instead of with atomics.
//
// Layouts: q, out [N, Hq, D]; pools [pages, Hkv, page_size, D]; block_table
// [S, table_stride] of page ids indexed by logical page (entries of pages that a window
// has released are never read); cu_q [S+1]; kv_len [S] (length after this step);
// seq_of_token [N].  Query token t of sequence s sits at position
// kv_len[s] - (cu_q[s+1]-cu_q[s]) + (t - cu_q[s]) and sees keys lo..p,
// lo = max(0, p - window + 1) when window > 0.
#include "common.cuh"

namespace {

using namespace pb;

constexpr int kWarps = 4;
constexpr int kMaxD = 256;

template <typename T> struct Vec;   // 16-byte vector of T
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

// The rows of one block: n_rows of at most R query rows of one sequence that share a key/value head, GP heads of the group for each of
// the tokens t0, t0 + 1, ...  Warp w takes the key tiles i with i mod 4 = w for all of them: lane l reads key l of the tile once and
// scores it against every row (the rows' queries come from shared memory by broadcast), then lane l owns the columns l, l + 32, ... of
// the rows' outputs and every value row is read once for all of them.  Bound by the latency of a tile's steps.  A row's sums do not
// depend on R or on the other rows.
template <typename T, int R, int ACC>
__device__ __forceinline__ void
rows_of_block(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool, T* __restrict__ out,
              const int* __restrict__ table, int t0, int n_rows, int p0, int Hq, int Hkv, int D, int page_size, float scale, int window,
              int GP, int g, int head0, const PoolBounds& bounds, float* smem) {
    float* q_s = smem;                         // [R][D] queries, multiplied by scale
    float* p_s = q_s + R * D;                  // [kWarps][R][32]
    float* m_s = p_s + kWarps * R * 32;        // [kWarps][R]
    float* l_s = m_s + kWarps * R;             // [kWarps][R]
    int* lo_s = reinterpret_cast<int*>(l_s + kWarps * R);       // [R] lowest visible key
    int* pos_s = lo_s + R;                                      // [R] the query's position
    float* acc_s = reinterpret_cast<float*>(pos_s + R);         // [kWarps][R][D]

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const int p = p0 + r / GP;
        pos_s[r] = p;
        lo_s[r] = (window > 0 && p - window + 1 > 0) ? p - window + 1 : 0;
    }
    // every row's query is asked for before the first is used
    constexpr int kParts = (32 * ACC + kWarps * 32 - 1) / (kWarps * 32);
    float qv[R][kParts];
    int token = t0, head = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const T* row = q + ((size_t)token * Hq + head0 + head) * D;
        if (++head == GP) { head = 0; ++token; }
#pragma unroll
        for (int i = 0; i < kParts; ++i) {
            const int d = threadIdx.x + i * kWarps * 32;
            qv[r][i] = (r < n_rows && d < D) ? to_float(row[d]) * scale : 0.0f;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kParts; ++i)
            if (threadIdx.x + i * kWarps * 32 < D) q_s[r * D + threadIdx.x + i * kWarps * 32] = qv[r][i];
    __syncthreads();

    float m_run[R], l_run[R], acc[R][ACC];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m_run[r] = -INFINITY;
        l_run[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < ACC; ++i) acc[r][i] = 0.0f;
    }

    const int lo_min = lo_s[0], p_max = pos_s[n_rows - 1];              // positions ascend along the rows
    const int first = lo_min >> 5, last = p_max >> 5;
    for (int tile = first + ((warp - first) & (kWarps - 1)); tile <= last; tile += kWarps) {
        const int j0 = tile << 5, j = j0 + lane;
        const bool any = j >= lo_min && j <= p_max;
        size_t at = 0;                                             // where the key's row begins in the pools
        float sc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) sc[r] = 0.0f;
        if (any) {
            int page = table[j / page_size];
            if (!page_ok(page, bounds)) page = 0;
            at = (((size_t)page * Hkv + g) * page_size + j % page_size) * D;
        }
        const T* kr = k_pool + at;
        for (int d = 0; d < D; d += 16) {                          // 16 elements of the key asked for at once
            constexpr int V = Vec<T>::n;
            float kf[16 / V][V];
#pragma unroll
            for (int u = 0; u < 16 / V; ++u) load16(kr + d + u * V, kf[u]);
#pragma unroll
            for (int u = 0; u < 16; u += 4) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 a = *reinterpret_cast<const float4*>(q_s + r * D + d + u);
                    sc[r] = fmaf(a.x, kf[u / V][u % V], sc[r]);
                    sc[r] = fmaf(a.y, kf[(u + 1) / V][(u + 1) % V], sc[r]);
                    sc[r] = fmaf(a.z, kf[(u + 2) / V][(u + 2) % V], sc[r]);
                    sc[r] = fmaf(a.w, kf[(u + 3) / V][(u + 3) % V], sc[r]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int lo = lo_s[r], p = pos_s[r];
            if (r >= n_rows || p < j0 || lo > j0 + 31) continue;   // uniform: the row sees nothing of this tile
            const bool valid = j >= lo && j <= p;
            const float m_new = fmaxf(m_run[r], warp_max(valid ? sc[r] : -INFINITY));
            const float pv = valid ? expf(sc[r] - m_new) : 0.0f;
            const float corr = expf(m_run[r] - m_new);             // 0 on the row's first tile (m_run = -inf)
            l_run[r] = l_run[r] * corr + warp_sum(pv);
            m_run[r] = m_new;
#pragma unroll
            for (int i = 0; i < ACC; ++i) acc[r][i] *= corr;
            p_s[(warp * R + r) * 32 + lane] = pv;
        }
        __syncwarp();
        for (int k0 = 0; k0 < 32; k0 += 4) {
            if (j0 + k0 > p_max) break;
            float vf[4][ACC];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const T* vr = v_pool + __shfl_sync(0xffffffffu, at, k0 + u);    // keys nobody sees read the pool's first row, unused
#pragma unroll
                for (int i = 0; i < ACC; ++i) vf[u][i] = lane + 32 * i < D ? to_float(vr[lane + 32 * i]) : 0.0f;
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int b = lo_s[r] - j0, e = pos_s[r] - j0;     // the row sees the keys b .. e of the tile
                if (r >= n_rows || e < k0 || b > k0 + 3) continue;
                const float4 pk = *reinterpret_cast<const float4*>(p_s + (warp * R + r) * 32 + k0);
                const float w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (k0 + u < b || k0 + u > e) continue;        // uniform; what the row does not see may be anything
#pragma unroll
                    for (int i = 0; i < ACC; ++i) acc[r][i] = fmaf(w[u], vf[u][i], acc[r][i]);
                }
            }
        }
        __syncwarp();
    }

#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r >= n_rows) continue;
        if (lane == 0) { m_s[warp * R + r] = m_run[r]; l_s[warp * R + r] = l_run[r]; }
#pragma unroll
        for (int i = 0; i < ACC; ++i) {
            const int d = lane + 32 * i;
            if (d < D) acc_s[(warp * R + r) * D + d] = acc[r][i];
        }
    }
    __syncthreads();
    for (int r = 0; r < n_rows; ++r) {
        const int turn = lo_s[r] >> 5;         // the warps' shares are added from that of the row's first tile on
        float m[kWarps], f[kWarps], m_all = -INFINITY, l_all = 0.0f;
#pragma unroll
        for (int c = 0; c < kWarps; ++c) {
            m[c] = m_s[((c + turn) & (kWarps - 1)) * R + r];
            m_all = fmaxf(m_all, m[c]);
        }
#pragma unroll
        for (int c = 0; c < kWarps; ++c) {
            f[c] = expf(m[c] - m_all);
            l_all += l_s[((c + turn) & (kWarps - 1)) * R + r] * f[c];
        }
        T* row = out + ((size_t)(t0 + r / GP) * Hq + head0 + r % GP) * D;
        for (int d = threadIdx.x; d < D; d += blockDim.x) {
            float o = 0.0f;
#pragma unroll
            for (int c = 0; c < kWarps; ++c) o += acc_s[(((c + turn) & (kWarps - 1)) * R + r) * D + d] * f[c];
            row[d] = from_float<T>(o / l_all);
        }
    }
}

// ROWS query rows that share a key/value head: GP heads of the group times TQ = ROWS / GP neighbouring tokens, counted from the first
// token of their sequence, so that a block's tokens belong to one sequence.  There is a block for every token; those that are not the
// first of their TQ end at once.  Every TQ-th token comes first in the grid, then every TQ-th of the rest: what stays is spread over
// the SMs and not on each TQ-th of them (16 heads of 64, 64 tokens at 2,064 keys: 167 us, 242 with the tokens in their order).  A block
// with four rows or fewer runs the loops for four.
// us, float32: a block per row, blocks over TQ tokens that walked their sequences one after the other, now: 32 heads on 8 of 128, 32
// single tokens at 2,000 keys beside a prompt of 200 679, 1,775, 438; 8 at 2,000 beside 505 tokens at 2,041 5,186, 2,867, 1,403; 16
// heads of 64, 32 at 500 beside 100 tokens 123, 259, 85; a prompt of 387 tokens (32 on 8 of 128) 498, 268, 177; 600 1,110, 448, 349.
template <typename T, int ROWS, int ACC>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                               T* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                               const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                               const int* __restrict__ seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                               float scale, int window, int GP, const PoolBounds bounds) {
    extern __shared__ __align__(16) float smem[];
    const int TQ = ROWS / GP;
    int t0 = blockIdx.x;
    if (ROWS > 1) {
        const int n_tiles = gridDim.x / TQ;
        t0 = blockIdx.x % n_tiles * TQ + blockIdx.x / n_tiles;
        if (t0 >= n_tokens) return;
    }
    const int s = seq_of_token[t0], q0 = cu_q[s];
    if (ROWS > 1 && (t0 - q0) % TQ) return;
    const int q1 = cu_q[s + 1];
    const int G = Hq / Hkv, g = blockIdx.y, g0 = blockIdx.z * GP;
    const int n_tok = max(1, min(min(TQ, q1 - t0), n_tokens - t0));
    // heads of the last part of a group may be fewer than GP: their rows are then those of one token (GP = ROWS)
    const int n_rows = min(n_tok * GP, G - g0 < GP ? G - g0 : ROWS);
    const int p0 = kv_len[s] - (q1 - q0) + (t0 - q0);
    const int* table = block_table + (size_t)s * table_stride;
    if (ROWS > 4 && n_rows <= 4)
        rows_of_block<T, 4, ACC>(q, k_pool, v_pool, out, table, t0, n_rows, p0, Hq, Hkv, D, page_size, scale, window, GP, g, g * G + g0, bounds, smem);
    else
        rows_of_block<T, ROWS, ACC>(q, k_pool, v_pool, out, table, t0, n_rows, p0, Hq, Hkv, D, page_size, scale, window, GP, g, g * G + g0, bounds, smem);
}

template <typename T, int ROWS, int ACC>
int launch_rows(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, int table_stride,
                const int* cu_q, const int* kv_len, const int* seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                float scale, int window, cudaStream_t stream) {
    const int G = Hq / Hkv, GP = G < ROWS ? G : ROWS, TQ = ROWS / GP;
    const size_t smem = sizeof(float) * ((size_t)ROWS * D + kWarps * ROWS * 32 + 2 * kWarps * ROWS + 2 * ROWS + (size_t)kWarps * ROWS * D);
    static SmemLimit limit;
    if (const int rc = limit.allow(paged_attention_generic_kernel<T, ROWS, ACC>, smem)) return rc;
    dim3 grid((n_tokens + TQ - 1) / TQ * TQ, Hkv, (G + GP - 1) / GP);
    if (grid.y > 65535 || grid.z > 65535) return PB_ERR_TOO_LARGE;
    paged_attention_generic_kernel<T, ROWS, ACC><<<grid, kWarps * 32, smem, stream>>>((const T*)q, (const T*)k_pool,
        (const T*)v_pool, (T*)out, block_table, table_stride, cu_q, kv_len, seq_of_token, n_tokens, Hq, Hkv, D, page_size, scale,
        window, GP, pb::pool_bounds_now());
    return launch_status();
}

// Sixteen rows a block (eight of heads wider than 128) where that leaves two blocks for every SM, else four: with few rows a row's
// own chain of tiles is what takes the time, and more blocks hide more of it.  One row a block up to two rows for every SM, and up to
// four where the block table names no more than 80 tokens: there the loops over rows cost more than the shared keys save (32 heads on 8
// of 128, float32, one row against four: 8 tokens at 256 keys 22.9 and 23.5 us, 16 at 256 31.5 and 23.7, 16 at 64 12.8 and 13.5, 2 at
// 2 5.4 and 8.2).
template <typename T>
int dispatch_generic(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, int table_stride,
                     const int* cu_q, const int* kv_len, const int* seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                     float scale, int window, cudaStream_t stream) {
#define PB_GENERIC(R, A) return launch_rows<T, R, A>(q, k_pool, v_pool, out, block_table, table_stride, cu_q, kv_len, seq_of_token, \
                                                     n_tokens, Hq, Hkv, D, page_size, scale, window, stream)
    const long rows = (long)n_tokens * Hq;
    const bool many = rows >= 16 * 2 * 148;
    if (rows <= 2 * 148 || (rows <= 4 * 148 && (long)table_stride * page_size <= 80)) {
        if (D <= 64) PB_GENERIC(1, 2);
        if (D <= 128) PB_GENERIC(1, 4);
        PB_GENERIC(1, 8);
    }
    if (D <= 64) { if (many) PB_GENERIC(16, 2); PB_GENERIC(4, 2); }
    if (D <= 128) { if (many) PB_GENERIC(16, 4); PB_GENERIC(4, 4); }
    if (many) PB_GENERIC(8, 8);
    PB_GENERIC(4, 8);
#undef PB_GENERIC
}

}  // namespace

PB_EXPORT int pb_paged_attention_generic(int dtype, const void* q, const void* k_pool, const void* v_pool, void* out,
                                         const int* block_table, int table_stride, const int* cu_q, const int* kv_len,
                                         const int* seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                                         float scale, int window, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (D <= 0 || D % 16 || D > kMaxD || Hkv <= 0 || Hq % Hkv || page_size <= 0) return PB_ERR_BAD_SIZE;
    if (Hkv > 65535) return PB_ERR_TOO_LARGE;
    if (dtype == PB_F32)
        return dispatch_generic<float>(q, k_pool, v_pool, out, block_table, table_stride, cu_q, kv_len, seq_of_token, n_tokens, Hq, Hkv, D,
                                       page_size, scale, window, stream);
    if (dtype == PB_BF16)
        return dispatch_generic<__nv_bfloat16>(q, k_pool, v_pool, out, block_table, table_stride, cu_q, kv_len, seq_of_token, n_tokens, Hq,
                                               Hkv, D, page_size, scale, window, stream);
    return PB_ERR_BAD_DTYPE;
}
