// Paged attention for any batch of query tokens: prompt portions and single decoded
// tokens side by side, causal, optional sliding window, grouped-query heads, any head
// size that is a multiple of 16 up to 256, float32 or bfloat16 storage.
//
// This is the exact kernel of the engine: scores, running maximum, sums and the output
// accumulate in float32 with expf.  The reduction order of a (token, head) pair depends
// only on that token's position (key tiles of 32 aligned to absolute key indices, tile i
// handled by warp i mod 4, the warps' shares combined from that of the row's first tile
// on), so logits do not depend on how tokens were cut into steps or batched.  The float32 path of the model always runs it; the bfloat16 path uses
// it wherever no tensor-core kernel applies.
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

// A block takes up to ROWS query rows that share a key/value head: GP heads of the group times ROWS / GP neighbouring tokens.
// Warp w takes the key tiles i with i mod 4 = w for all of them: lane l reads key l of the tile once and scores it against every
// row (the rows' queries come from shared memory by broadcast), then lane l owns the columns l, l + 32, ... of the rows' outputs
// and every value row is read once for all of them.  Bound by the latency of a tile's steps; with a block per row instead by reading
// K and V again for each row (8 kv heads of 4 query heads, head size 128, float32: a prompt of 387 tokens 268 us, 498 with a block per
// row; 600 tokens 455, 1,119).  A row's sums do not depend on ROWS or on the other rows.
template <typename T, int ROWS, int ACC>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                               T* __restrict__ out, const int* __restrict__ block_table, int table_stride,
                               const int* __restrict__ cu_q, const int* __restrict__ kv_len,
                               const int* __restrict__ seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                               float scale, int window, int GP, const PoolBounds bounds) {
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;                         // [ROWS][D] queries, multiplied by scale
    float* p_s = q_s + ROWS * D;               // [kWarps][ROWS][32]
    float* m_s = p_s + kWarps * ROWS * 32;     // [kWarps][ROWS]
    float* l_s = m_s + kWarps * ROWS;          // [kWarps][ROWS]
    int* lo_s = reinterpret_cast<int*>(l_s + kWarps * ROWS);    // [ROWS] lowest visible key
    int* pos_s = lo_s + ROWS;                                   // [ROWS] the query's position; -1: no such row
    float* acc_s = reinterpret_cast<float*>(pos_s + ROWS);      // [kWarps][ROWS][D]

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = Hq / Hkv, g = blockIdx.y, g0 = blockIdx.z * GP;
    const int TQ = ROWS / GP;
    const int t0 = blockIdx.x * TQ, t1 = min(n_tokens, t0 + TQ);

    for (int r = threadIdx.x; r < ROWS; r += blockDim.x) {
        const int t = t0 + r / GP;
        const bool on = r < TQ * GP && t < t1 && g0 + r % GP < G;
        int p = -1, lo = 0;
        if (on) {
            const int s = seq_of_token[t], q0 = cu_q[s], q1 = cu_q[s + 1];
            p = kv_len[s] - (q1 - q0) + (t - q0);
            if (window > 0 && p - window + 1 > 0) lo = p - window + 1;
        }
        pos_s[r] = p;
        lo_s[r] = lo;
    }
    for (int i = threadIdx.x; i < ROWS * D; i += blockDim.x) {
        const int r = i / D, d = i % D, t = t0 + r / GP, h = g0 + r % GP;
        const bool on = r < TQ * GP && t < t1 && h < G;
        q_s[i] = on ? to_float(q[((size_t)t * Hq + g * G + h) * D + d]) * scale : 0.0f;
    }
    __syncthreads();

    float m_run[ROWS], l_run[ROWS], acc[ROWS][ACC];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        m_run[r] = -INFINITY;
        l_run[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < ACC; ++i) acc[r][i] = 0.0f;
    }

    // the block's tokens sequence by sequence (as a rule there is one): their rows are neighbours
    for (int ta = t0; ta < t1;) {
        const int s = seq_of_token[ta];
        const int te = max(ta + 1, min(t1, cu_q[s + 1]));
        const int r0 = (ta - t0) * GP, r1 = (te - t0) * GP;
        const int lo_min = lo_s[r0], p_max = pos_s[r1 - GP];           // positions ascend along a sequence's tokens
        const int* table = block_table + (size_t)s * table_stride;
        ta = te;
        const int first = lo_min >> 5, last = p_max >> 5;
        for (int tile = first + ((warp - first) & (kWarps - 1)); tile <= last; tile += kWarps) {
            const int j0 = tile << 5, j = j0 + lane;
            const bool any = j >= lo_min && j <= p_max;
            size_t at = 0;                                             // where the key's row begins in the pools
            float sc[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) sc[r] = 0.0f;
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
                    for (int r = 0; r < ROWS; ++r) {
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
            for (int r = 0; r < ROWS; ++r) {
                const int lo = lo_s[r], p = pos_s[r];
                if (r < r0 || r >= r1 || p < j0 || lo > j0 + 31) continue;          // uniform: the row sees nothing of this tile
                const bool valid = j >= lo && j <= p;
                const float m_new = fmaxf(m_run[r], warp_max(valid ? sc[r] : -INFINITY));
                const float pv = valid ? expf(sc[r] - m_new) : 0.0f;
                const float corr = expf(m_run[r] - m_new);             // 0 on the row's first tile (m_run = -inf)
                l_run[r] = l_run[r] * corr + warp_sum(pv);
                m_run[r] = m_new;
#pragma unroll
                for (int i = 0; i < ACC; ++i) acc[r][i] *= corr;
                p_s[(warp * ROWS + r) * 32 + lane] = pv;
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
                for (int r = 0; r < ROWS; ++r) {
                    const int b = lo_s[r] - j0, e = pos_s[r] - j0;     // the row sees the keys b .. e of the tile
                    if (r < r0 || r >= r1 || e < k0 || b > k0 + 3) continue;
                    const float4 pk = *reinterpret_cast<const float4*>(p_s + (warp * ROWS + r) * 32 + k0);
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
    }

#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        if (lane == 0) { m_s[warp * ROWS + r] = m_run[r]; l_s[warp * ROWS + r] = l_run[r]; }
#pragma unroll
        for (int i = 0; i < ACC; ++i) {
            const int d = lane + 32 * i;
            if (d < D) acc_s[(warp * ROWS + r) * D + d] = acc[r][i];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ROWS * D; i += blockDim.x) {
        const int r = i / D, d = i % D;
        if (pos_s[r] < 0) continue;
        const int turn = lo_s[r] >> 5;         // the warps' shares are added from that of the row's first tile on
        float m[kWarps], m_all = -INFINITY;
#pragma unroll
        for (int c = 0; c < kWarps; ++c) {
            m[c] = m_s[((c + turn) & (kWarps - 1)) * ROWS + r];
            m_all = fmaxf(m_all, m[c]);
        }
        float l_all = 0.0f, o = 0.0f;
#pragma unroll
        for (int c = 0; c < kWarps; ++c) {
            const int w = (c + turn) & (kWarps - 1);
            const float f = expf(m[c] - m_all);
            l_all += l_s[w * ROWS + r] * f;
            o += acc_s[(w * ROWS + r) * D + d] * f;
        }
        out[((size_t)(t0 + r / GP) * Hq + g * G + g0 + r % GP) * D + d] = from_float<T>(o / l_all);
    }
}

template <typename T, int ROWS, int ACC>
int launch_rows(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, int table_stride,
                const int* cu_q, const int* kv_len, const int* seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                float scale, int window, cudaStream_t stream) {
    const int G = Hq / Hkv, GP = G < ROWS ? G : ROWS, TQ = ROWS / GP;
    const size_t smem = sizeof(float) * ((size_t)ROWS * D + kWarps * ROWS * 32 + 2 * kWarps * ROWS + 2 * ROWS + (size_t)kWarps * ROWS * D);
    constexpr size_t most = sizeof(float) * (ROWS * 32 * ACC + kWarps * ROWS * 32 + 2 * kWarps * ROWS + 2 * ROWS + kWarps * ROWS * 32 * ACC);
    static const cudaError_t allowed =
        cudaFuncSetAttribute(paged_attention_generic_kernel<T, ROWS, ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (allowed != cudaSuccess) return (int)allowed;
    dim3 grid((n_tokens + TQ - 1) / TQ, Hkv, (G + GP - 1) / GP);
    if (grid.y > 65535 || grid.z > 65535) return PB_ERR_TOO_LARGE;
    paged_attention_generic_kernel<T, ROWS, ACC><<<grid, kWarps * 32, smem, stream>>>((const T*)q, (const T*)k_pool,
        (const T*)v_pool, (T*)out, block_table, table_stride, cu_q, kv_len, seq_of_token, n_tokens, Hq, Hkv, D, page_size, scale,
        window, GP, pb::pool_bounds_now());
    return launch_status();
}

// Sixteen rows a block (eight of heads wider than 128) where that leaves two blocks for every SM, else four: with few rows a row's
// own chain of tiles is what takes the time, and more blocks hide more of it.
template <typename T>
int dispatch_generic(const void* q, const void* k_pool, const void* v_pool, void* out, const int* block_table, int table_stride,
                     const int* cu_q, const int* kv_len, const int* seq_of_token, int n_tokens, int Hq, int Hkv, int D, int page_size,
                     float scale, int window, cudaStream_t stream) {
#define PB_GENERIC(R, A) return launch_rows<T, R, A>(q, k_pool, v_pool, out, block_table, table_stride, cu_q, kv_len, seq_of_token, \
                                                     n_tokens, Hq, Hkv, D, page_size, scale, window, stream)
    const bool many = (long)n_tokens * Hq >= 16 * 2 * 148;
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
