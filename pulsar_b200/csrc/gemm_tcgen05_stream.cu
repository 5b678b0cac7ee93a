// out[M, N] = x[M, K] * W[N, K]^T for 17 to 128 tokens in bfloat16: the projections of a step of dozens of single
// tokens or of a short prompt, where every weight is still read once and the time is the time to stream W from HBM,
// but there are too many tokens for the kernel that keeps them in MMA fragments (gemm_skinny.cu).
//
// The operands change places against gemm_tcgen05.cu: rows of W are the 128-row operand of tcgen05.mma (the lanes of
// the accumulator in tensor memory), the tokens are its narrow one (16 to 128 columns).
//
// Bound by HBM; what it takes to get there, at 48 tokens and the 8B sizes.  Bytes on their way: a load takes 2 us under full load, so an
// SM needs some 100 KB of W asked for; the ring takes what shared memory is left, and until x is there (the kernel before still
// runs) further W comes to L2.  Issue: a stage costs the thread that asks for it or multiplies it 350 to 500 cycles however small it
// is, so stages are 128 k deep and W and x have a thread each (64 k and one thread: 285 ns a stage, 27 GB/s an SM).  Splitting:
// 4096 output features are only 32 tiles of 128 rows, so K is cut into `slices`, one block of a thread-block cluster each.  A
// cluster walks over tiles (cluster i: tiles i, i + clusters, ...) without a pause, two accumulators in tensor memory take turns, and a
// finished tile's partial sums meet in the cluster's shared memory: every block sends each quad of tokens, float32, to the block whose
// share it is (asynchronous stores that count on the receiver's barrier), which adds them in the order of the slices.  No partial
// sum travels through L2.  Tail behind the last stage: 2.5 us (4.4 with sums fetched from the peers instead of sent by them).
// us (the library's product, with the gating kernel behind gate/up; both in a graph of launches over weights larger than L2):
//   48 tokens: 6144 x 4096 11.3 (11.7), 4096 x 4096 9.0 (9.9), gate/up 24576 x 4096 32.2 (38.0), 4096 x 12288 19.1 (21.2),
//   151936 x 4096 181 (206; 6.9 TB/s); 111 tokens: gate/up 39.5 (46.0), most others behind the library's (the tokens' tile is read
//   again from L2 with every tile: at 111 tokens as many bytes as W's).  Between other kernels some 3 us more of this one's time is
//   hidden than of the library's.
//
// Roles in a block (224 threads): warp 0 / one thread issues the TMA loads of W (with an evict-first L2 hint: weights are read once
// per step and are far larger than L2), before the kernel waits for its predecessor; warp 6 / one thread those of x, behind it; warp
// 1 / one lane issues the MMAs, warps 2-5 read the accumulators.  Gated product: a tile holds gate rows and the up rows that belong
// to them, and the gating is applied where the sums are complete, so the [M, 2I] intermediate never exists.
//
// Every wait on a barrier is bounded by a clock limit; a role that gives up sets the error word, lets its copies
// land, and the block frees its tensor memory and returns.  A block ends when it has all that its peers send it, and one that gave up
// waits for its peers to end or give up, so nothing is sent to a block that has gone.  No TMA load uses cluster multicast.
//
// The reference calls at::linear (cuBLAS) for all of these (pulsar-core/src/model/qwen3.cpp:82-84, 114, 117-119).
#include "tcgen05_common.cuh"

#include <algorithm>
#include <cstdlib>

namespace {

using namespace pb;
typedef __nv_bfloat16 bf16;

constexpr int kRows = 128;            // rows of one MMA (lanes of tensor memory)
constexpr int kAtom = 64;             // k of a box: one 128-byte swizzle atom of bfloat16
constexpr int kBK = 128;              // k per stage
constexpr int kThreads = 224;
constexpr int kTmemColumns = 256;     // two accumulators of up to 128 columns
constexpr int kMaxStages = 16;
constexpr int kAhead = 2;             // stages whose W is fetched to L2 while x is not there
constexpr int kMaxSlices = 8;         // blocks of a cluster (the portable limit)
constexpr int kSmem = 226 * 1024;     // dynamic shared memory of a block, at most

enum { kPlain = 0, kSwiGLU = 1 };

__device__ unsigned int g_stream_error = 0;       // 0 = fine; else 1 + the role that gave up

__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {      // K-major, 128-byte rows, 128-byte swizzle
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3fff);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int c0, int c1) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}

// A barrier, or 16 bytes, of the cluster's block `rank` at this block's shared-memory address `addr`.
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void peer_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// 16 bytes to a block of the cluster; they count towards what that block's barrier `bar` expects.
__device__ __forceinline__ void peer_push(uint32_t addr, uint32_t bar, const uint32_t* v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}
// mbar_wait on a barrier that other blocks of the cluster arrive at: what they wrote or read before is ordered before what follows.
// (By the wait itself: a fence behind both waits costs every thread, gate/up 24576 x 4096 with 48 tokens 34.9 us against 32.2.)
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    const long long t0 = clock64(), limit = __ldg(&g_wait_limit);
    while (!mbar_try_wait_cluster(bar, parity)) {
        if (*abort_flag) return false;
        if (clock64() - t0 > limit) return false;
    }
    return true;
}

struct StreamArgs {
    int M, N, K;
    int n_pad;          // tokens rounded up to a multiple of 16: columns of an accumulator, rows of an x box
    int stages;         // TMA stages of the ring
    int slices;         // slices of K per tile, blocks of a cluster
    int rows;           // rows of W in a tile, a multiple of 16, at most 128
    int pass;           // tokens whose partial sums are laid down at once
    int n_tiles;        // tiles of W's rows
    int part_offset;    // bytes from the ring's start to the partial sums [pass tokens][tile rows] float32
    int bar_offset;     // bytes from the ring's start to the barriers
    GatedInter inter;   // gated product: its width and gating
};

// Barrier of `threads` threads that returns whether `ok` held for all of them: the epilogue warps decide together
// whether a wait ran out, so that none of them goes on to a barrier that the others have left.
__device__ __forceinline__ bool named_barrier_all(int id, int threads, bool ok) {
    uint32_t all;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %3, 0;\nbar.red.and.pred p, %1, %2, q;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(all) : "r"(id), "r"(threads), "r"((uint32_t)ok) : "memory");
    return all != 0;
}

// The end of a pass: this block's share of the pass's tokens, `own` quads from token `first`, summed over the cluster's slices in their
// order, gated where the product is gated, and stored.  128 threads, a thread four tokens of one output column at a time.
// part: [slices][stride quads][rows] of four tokens' partial sums each.
template <int MODE, typename OutT>
__device__ __forceinline__ void add_up(const float4* part, int rows, int slices, int stride, int own, int first, int M, int col0, int width,
                                       int etid, OutT* __restrict__ out, const GatedInter& gate) {
    const int cols = MODE == kSwiGLU ? rows / 2 : rows;
    const bool halves = cols <= 64;                                  // two quads side by side
    const int c = halves ? etid & 63 : etid, step = halves ? 2 : 1;
    if (c >= cols || col0 + c >= width) return;
    int q = halves ? etid >> 6 : 0;
    const float4* p = part + q * rows + c;
    OutT* o = out + (size_t)(first + q * 4) * width + col0 + c;
    int left = M - first - q * 4;
#pragma unroll 2
    for (; q < own; q += step, p += step * rows, o += (size_t)(4 * step) * width, left -= 4 * step) {
        float4 sum = p[0], up = MODE == kSwiGLU ? p[cols] : sum;
        for (int s = 1; s < slices; ++s) {
            const float4 v = p[s * stride * rows];
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            if (MODE == kSwiGLU) {
                const float4 u = p[s * stride * rows + cols];
                up.x += u.x; up.y += u.y; up.z += u.z; up.w += u.w;
            }
        }
        if (MODE == kSwiGLU) {
            sum.x = gated(sum.x, up.x, gate); sum.y = gated(sum.y, up.y, gate);
            sum.z = gated(sum.z, up.z, gate); sum.w = gated(sum.w, up.w, gate);
        }
        o[0] = from_float<OutT>(sum.x);
        if (left > 1) o[width] = from_float<OutT>(sum.y);
        if (left > 2) o[2 * (size_t)width] = from_float<OutT>(sum.z);
        if (left > 3) o[3 * (size_t)width] = from_float<OutT>(sum.w);
    }
}

template <int MODE, typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tcgen05_stream_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                           OutT* __restrict__ out, const __grid_constant__ StreamArgs a) {
    extern __shared__ unsigned char smem_raw[];
    const int tile_cols = MODE == kSwiGLU ? a.rows / 2 : a.rows;
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int w_bytes = a.rows * kBK * 2, x_bytes = a.n_pad * kBK * 2, stage_bytes = w_bytes + x_bytes;
    const float4* part = reinterpret_cast<const float4*>(smem + a.part_offset);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + a.bar_offset);            // full, empty [kMaxStages], then pairs and singles
    const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * kMaxStages;
    const uint32_t acc_full0 = empty0 + 8 * kMaxStages, acc_empty0 = acc_full0 + 16;
    const uint32_t part_full = acc_full0 + 32, part_empty = acc_full0 + 40;       // all blocks' sums are laid down; all have read mine
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 6);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)(blockIdx.x % a.slices), cluster = (int)(blockIdx.x / a.slices), clusters = (int)(gridDim.x / a.slices);
    const int k_tiles = (a.K + kBK - 1) / kBK;
    const int kt0 = (int)((long long)k_tiles * rank / a.slices), kt1 = (int)((long long)k_tiles * (rank + 1) / a.slices);

    const uint64_t policy = policy_evict_first();
    auto load_w = [&](int s, int kt, int tile) {
        const uint32_t bar = full0 + 8 * s, dst = smem_addr(smem) + s * stage_bytes;
        mbar_expect_tx(bar, w_bytes);
#pragma unroll
        for (int h = 0; h < kBK / kAtom; ++h) {
            const uint32_t d = dst + h * (w_bytes / 2);
            tma_load_2d_hint(d, &map_w, bar, kt * kBK + h * kAtom, tile * tile_cols, policy);
            if (MODE == kSwiGLU) tma_load_2d_hint(d + w_bytes / 4, &map_w, bar, kt * kBK + h * kAtom, a.inter.n + tile * tile_cols, policy);
        }
    };
    auto prefetch_w = [&](int kt, int tile) {
#pragma unroll
        for (int h = 0; h < kBK / kAtom; ++h) {
            tma_prefetch_2d(&map_w, kt * kBK + h * kAtom, tile * tile_cols);
            if (MODE == kSwiGLU) tma_prefetch_2d(&map_w, kt * kBK + h * kAtom, a.inter.n + tile * tile_cols);
        }
    };
    // The weights depend on no earlier kernel: the first stages' W is on its way before anything else is done.
    const int early = min(kt1 - kt0, a.stages);
    if (tid == 0) {
        for (int s = 0; s < a.stages; ++s) { mbar_init(full0 + 8 * s, 2); mbar_init(empty0 + 8 * s, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(acc_full0 + 8 * i, 1); mbar_init(acc_empty0 + 8 * i, 4); }
        mbar_init(part_full, 1);
        mbar_init(part_empty, a.slices);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < early; ++i) load_w(i, kt0 + i, cluster);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(kTmemColumns));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (a.slices > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;

    if (warp == 0) {
        // ---------------- TMA producer of W: stage s of the ring's turn `phase`; the first `early` loads are asked for above
        if (lane == 0) {
            int s = early == a.stages ? 0 : early, kt = kt0 + early;
            uint32_t phase = early == a.stages ? 1 : 0;
            // HBM has time to spare until x is there: the W of two stages more comes to L2 (a layer's products, 48 tokens: 3 us of 83)
            for (int i = 0; i < kAhead && kt + i < kt1; ++i) prefetch_w(kt + i, cluster);
            for (int tile = cluster; tile < a.n_tiles && ok; tile += clusters, kt = kt0)
                for (; kt < kt1; ++kt) {
                    if (!mbar_wait(empty0 + 8 * s, phase ^ 1, abort_flag)) { ok = false; break; }
                    load_w(s, kt, tile);
                    if (++s == a.stages) { s = 0; phase ^= 1; }
                }
            if (!ok) atomicMax(&g_stream_error, 2u);
        }
    } else if (warp == 6) {
        // ---------------- TMA producer of x, behind the kernels that write it
        if (lane == 0) {
            const uint32_t x0 = smem_addr(smem) + w_bytes;
            int s = 0;
            uint32_t phase = 0;
            pdl_wait();
            for (int tile = cluster; tile < a.n_tiles && ok; tile += clusters)
                for (int kt = kt0; kt < kt1; ++kt) {
                    const uint32_t bar = full0 + 8 * s, dst = x0 + s * stage_bytes;
                    if (!mbar_wait(empty0 + 8 * s, phase ^ 1, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(bar, x_bytes);
#pragma unroll
                    for (int h = 0; h < kBK / kAtom; ++h) tma_load_2d(dst + h * (x_bytes / 2), &map_x, bar, kt * kBK + h * kAtom, 0);
                    if (++s == a.stages) { s = 0; phase ^= 1; }
                }
            if (!ok) atomicMax(&g_stream_error, 2u);
            pdl_trigger();                                               // every load is asked for: the next kernel's may come
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: the warp walks the loop uniformly, one elected lane issues
        const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t desc0 = umma_desc(smem_addr(smem));
        // float32 accumulator, bfloat16 A and B, both K-major, N >> 3, M >> 4
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.n_pad >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
        uint32_t phase = 0;
        int j = 0, s = 0;
        for (int tile = cluster; tile < a.n_tiles && ok; tile += clusters, ++j) {
            const int acc = j & 1;
            ok = mbar_wait(acc_empty0 + 8 * acc, ((j >> 1) & 1) ^ 1, abort_flag);
            const uint32_t tmem_d = tmem_u + acc * 128;
            for (int kt = kt0; kt < kt1 && ok; ++kt) {
                if (!mbar_wait(full0 + 8 * s, phase, abort_flag)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t w_desc = desc0 + (uint64_t)((uint32_t)(s * stage_bytes) >> 4);
                const uint64_t x_desc = w_desc + (uint64_t)(w_bytes >> 4);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k)         // four steps of 16 k lie in each atom
                        umma_bf16(tmem_d, w_desc + (uint64_t)(k / 4 * (w_bytes >> 5) + k % 4 * 2), x_desc + (uint64_t)(k / 4 * (x_bytes >> 5) + k % 4 * 2),
                                  idesc, (kt > kt0 || k > 0) ? 1u : 0u);
                    umma_commit(empty0 + 8 * s);
                    if (kt == kt1 - 1) umma_commit(acc_full0 + 8 * acc);
                }
                __syncwarp();
                if (++s == a.stages) { s = 0; phase ^= 1; }
            }
        }
        if (!ok && lane == 0) atomicMax(&g_stream_error, 3u);
    } else {
        // ---------------- epilogue: this thread holds weight row `row`, one token per column
        if (a.slices > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");       // the peers' barriers are set up
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const int etid = tid - 64;                                              // 0 .. 127 among the epilogue threads
        const uint32_t part_addr = smem_addr(part);
        uint32_t pass = 0;                                                      // passes so far: the phase of both barriers
        int j = 0;
        for (int tile = cluster; tile < a.n_tiles && ok; tile += clusters, ++j) {
            const int acc = j & 1;
            ok = named_barrier_all(4, 128, mbar_wait(acc_full0 + 8 * acc, (j >> 1) & 1, abort_flag));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t lane_base = tmem_base + acc * 128 + ((uint32_t)(quarter * 32) << 16);
            for (int first = 0; first < a.M && ok; first += a.pass, ++pass) {
                // quads of tokens in this pass, of each block's share, and of this block's
                const int quads = (min(a.pass, a.M - first) + 3) / 4, share = (quads + a.slices - 1) / a.slices;
                const int own = max(0, min(share, quads - rank * share));
                // what the pass before laid down has been read by all blocks of the cluster
                ok = named_barrier_all(4, 128, mbar_wait_cluster(part_empty, (pass & 1) ^ 1, abort_flag));
                if (!ok) break;
                if (etid == 0) mbar_expect_tx(part_full, a.slices * own * a.rows * 16);
                int owner = 0, slot = 0;
                const uint32_t mine = part_addr + (rank * share * a.rows + row) * 16;
                uint32_t to = peer_addr(mine, 0), bar = peer_addr(part_full, 0);
                for (int c0 = 0; c0 < quads; c0 += 8) {
                    uint32_t v[32];
                    tmem_ld32(lane_base + first + c0 * 4, v);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        if (c0 + i >= quads) break;
                        if (slot == share) {
                            slot = 0;
                            to = peer_addr(mine, ++owner);
                            bar = peer_addr(part_full, owner);
                        }
                        if (row < a.rows) peer_push(to, bar, v + 4 * i);
                        to += a.rows * 16;
                        ++slot;
                    }
                }
                const bool last = first + a.pass >= a.M;
                if (last) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty0 + 8 * acc);           // the accumulator is free again
                }
                ok = named_barrier_all(4, 128, mbar_wait_cluster(part_full, pass & 1, abort_flag));
                if (!ok) break;
                add_up<MODE, OutT>(part, a.rows, a.slices, share, own, first + rank * share * 4, a.M, tile * tile_cols,
                                   MODE == kSwiGLU ? a.inter.n : a.N, etid, out, a.inter);
                if (last && tile + clusters >= a.n_tiles) break;                // nobody waits for it, and the block may be gone
                named_barrier_all(4, 128, true);
                if (etid < a.slices) peer_arrive(peer_addr(part_empty, etid));
            }
        }
        if (!ok && lane == 0) atomicMax(&g_stream_error, 4u);
    }
    if (!ok) *abort_flag = 1;
    __syncwarp();
    if (a.slices > 1 && (warp < 2 || warp == 6)) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // A block that gave up lets its copies and products in flight land before it frees what they write.
    const bool gave_up = *abort_flag != 0;
    if (gave_up)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemColumns));
    // A block that ends has what its peers sent it, and sends nothing to one that has ended.  One that gave up waits for its peers, which
    // may still send to it.
    if (gave_up && a.slices > 1) {
        __syncthreads();
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    }
}

// Row-major [rows, K] bfloat16 matrix, boxes of box_rows x 64 columns, 128-byte swizzle, zero fill outside.
int make_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return (int)cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {kAtom, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rc == CUDA_SUCCESS ? 0 : PB_ERR_BAD_SIZE;
}

int forced(const char* name) {
    const char* v = getenv(name);
    return v ? atoi(v) : 0;
}

cudaLaunchConfig_t stream_config(cudaLaunchAttribute (&attr)[2], int slices, int grid, size_t smem, bool early, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = kThreads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early && pdl_enabled() ? 2 : 1;
    return cfg;
}

// Clusters of `slices` blocks that the device holds at once (one block an SM; clusters do not cross the chip's GPU processing
// clusters, so not every SM can be used by every size).
template <int MODE, typename OutT>
int resident_clusters(int slices, int dev) {
    static DeviceCount known[kMaxSlices + 1];
    return known[slices].get(dev, [&](int* n) {
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = stream_config(attr, slices, slices, kSmem, false, nullptr);
        const cudaError_t rc = cudaOccupancyMaxActiveClusters(n, gemm_tcgen05_stream_kernel<MODE, OutT>, &cfg);
        if (rc != cudaSuccess) (void)cudaGetLastError();
        return (int)rc;
    });
}

// Shared memory of a block besides the alignment of its ring: barriers, and what is left for stages and partial sums.
constexpr int kBarBytes = (2 * kMaxStages + 6) * 8 + 16, kRoom = kSmem - 1024 - kBarBytes;

// Bytes of the partial sums of `pass` tokens.
inline int sum_bytes(int pass, int slices, int rows) { return (pass / 4 + slices - 1) / slices * slices * rows * 16; }

// Tokens whose partial sums are laid down at once: all, or 64 where all leave fewer than three stages.
inline int pass_tokens(int n_pad, int slices, int rows) {
    return n_pad > 64 && kRoom - sum_bytes(n_pad, slices, rows) < 3 * (rows + n_pad) * kBK * 2 ? 64 : n_pad;
}

// How a problem is cut: slices of K, rows of a tile.  The cost is what a block walks through one after the other, in rows of 128 k:
//   - the k-tiles of its slice times the tile's rows and half a row for every token, for its first tile;
//   - that for every further tile, or what the sums of a tile take where that is longer.  All of a tile's sums pass through every
//     block's epilogue however many slices there are, once for each pass (gate/up 28672 x 4096, 111 tokens, tiles of 128 rows: 4.7 rounds of 3
//     slices 73 us, 3 of 2 slices 48; 76000 x 2048, 128 tokens: 1, 2, 4, 8 slices 65, 90, 142, 297);
//   - the last round by how full it is, but as no less than half a round (an SM alone pulls twice its share of HBM; with many tokens,
//     whose loads come from L2, less);
//   - the exchange behind the last tile, by the block's share of the tokens.
// The weights of these were fitted to the times of all cuts of 30 products with 32 to 128 tokens: the chosen one is on average 2.7 % behind
// the best (9.0 % while the sums were taken to cost less the more slices share them).  us at 48 tokens: 4096 x 4096 4 slices x 128 rows
// 8.9; 6144 x 4096 2 x 96 11.3; gate/up 24576 x 4096 2 x 112 32.2; 4096 x 12288 4 x 128 19.1.
template <int MODE, typename OutT>
int cut(StreamArgs& a, int k_tiles) {          // the clusters that the device holds, 0: none of any size
    static const int slices_forced = forced("PULSAR_STREAM_SLICES");
    const int width = MODE == kSwiGLU ? a.inter.n : a.N, quads = a.n_pad / 4;
    float best = 0.0f;
    int clusters = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    for (int s = 1; s <= kMaxSlices && s <= k_tiles; ++s) {
        if (slices_forced > 0 && s != std::min(slices_forced, std::min(kMaxSlices, k_tiles))) continue;
        const int n = resident_clusters<MODE, OutT>(s, dev);
        if (n == 0) continue;
        const int slice_tiles = (k_tiles + s - 1) / s, share = (quads + s - 1) / s;
        for (int rows = kRows; rows >= 48; rows -= 16) {
            const int cols = MODE == kSwiGLU ? rows / 2 : rows, tiles = (width + cols - 1) / cols, rest = tiles % n;
            const int passes = pass_tokens(a.n_pad, s, rows) < a.n_pad ? 2 : 1;
            float rounds = (float)(tiles / n);
            if (rest > 0) rounds += fminf(1.0f, fmaxf((float)rest / n, 0.5f + a.n_pad / 256.0f));
            const float walk = (float)(slice_tiles * (rows + a.n_pad / 2));
            const float sums = s > 1 ? 600.0f * passes + 80.0f * quads : 450.0f * passes + 64.0f * quads;
            const float cost = fminf(rounds, 1.0f) * walk + fmaxf(rounds - 1.0f, 0.0f) * fmaxf(walk, sums) + 150.0f * passes + 20.0f * share;
            if (best == 0.0f || cost < best) { best = cost; clusters = n; a.slices = s; a.rows = rows; a.n_tiles = tiles; }
        }
    }
    return clusters;
}

template <int MODE, typename OutT>
int launch(const void* x, const void* w, void* out, StreamArgs a, bool loaded, cudaStream_t stream) {
    static SmemLimit limit;
    if (const int rc = limit.allow(gemm_tcgen05_stream_kernel<MODE, OutT>, kSmem)) return rc;
    const int n = cut<MODE, OutT>(a, (a.K + kBK - 1) / kBK);
    if (n == 0) return PB_ERR_BAD_SIZE;            // declined: the caller has another product
    const int stage_bytes = (a.rows + a.n_pad) * kBK * 2;
    // The MMAs read kRows rows from an atom's first: what lies behind the last stage, up to there, belongs to the block as well.
    const int beyond = (a.rows + kRows) * kAtom * 2 + 1024;
    a.pass = pass_tokens(a.n_pad, a.slices, a.rows);
    const int part_bytes = sum_bytes(a.pass, a.slices, a.rows);
    int stages = std::min((kRoom - part_bytes) / stage_bytes, kMaxStages);
    while (stages > 0 && (stages - 1) * stage_bytes + beyond > kSmem) --stages;
    static const int stages_forced = forced("PULSAR_STREAM_STAGES");
    if (stages_forced > 0 && stages_forced < stages) stages = stages_forced;
    if (stages < 2) return PB_ERR_BAD_SIZE;
    a.stages = stages;
    a.part_offset = stages * stage_bytes;
    a.bar_offset = a.part_offset + part_bytes;
    int smem = a.bar_offset + kBarBytes + 1024;
    if (smem < (stages - 1) * stage_bytes + beyond) smem = (stages - 1) * stage_bytes + beyond;
    CUtensorMap mx, mw;
    if (const int rc = make_map(&mx, x, a.M, a.K, a.n_pad)) return rc;
    if (const int rc = make_map(&mw, w, a.N, a.K, MODE == kSwiGLU ? a.rows / 2 : a.rows)) return rc;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = stream_config(attr, a.slices, (a.n_tiles < n ? a.n_tiles : n) * a.slices, smem, loaded, stream);
    return (int)cudaLaunchKernelEx(&cfg, gemm_tcgen05_stream_kernel<MODE, OutT>, mx, mw, (OutT*)out, (const StreamArgs)a);
}

}  // namespace

// 1 if pb_gemm_tcgen05_stream takes this problem: 1 to 128 tokens, K a multiple of 8 (TMA strides are multiples of
// 16 bytes); a gated product additionally needs the gate/up halves to split evenly.
PB_EXPORT int pb_gemm_tcgen05_stream_supported(int mode, int M, int N, int K) {
    if (M <= 0 || M > 128 || N <= 0 || K <= 0 || (K % 8)) return 0;
    if (mode == kSwiGLU) return (N % 2 == 0) ? 1 : 0;
    return mode == kPlain ? 1 : 0;
}

// slices and rows: how the product is cut on the current device.  Returns the clusters that it holds, 0 where the product is declined.
PB_EXPORT int pb_gemm_tcgen05_stream_cut(int mode, int M, int N, int K, int* slices, int* rows) {
    if (!pb_gemm_tcgen05_stream_supported(mode, M, N, K)) return 0;
    StreamArgs a{};
    a.N = N;
    a.n_pad = (M + 15) / 16 * 16;
    a.inter = GatedInter(mode == kSwiGLU ? N / 2 : 0);
    static SmemLimit limits[2];
    if (mode == kSwiGLU ? limits[0].allow(gemm_tcgen05_stream_kernel<kSwiGLU, bf16>, kSmem) : limits[1].allow(gemm_tcgen05_stream_kernel<kPlain, bf16>, kSmem)) return 0;
    const int n = mode == kSwiGLU ? cut<kSwiGLU, bf16>(a, (K + kBK - 1) / kBK) : cut<kPlain, bf16>(a, (K + kBK - 1) / kBK);
    *slices = a.slices;
    *rows = a.rows;
    return n;
}

// limit > 0: the new limit of the kernel's bounded waits in clock cycles; error >= 0: the new value of the error
// word; address: receives the word's device address.  Returns 0, or -1 when a CUDA call failed.
PB_EXPORT int pb_gemm_tcgen05_stream_wait_control(long long limit, int error, void** address) {
    return wait_control(g_stream_error, limit, error, address);
}

// mode 0: out[M, N] = x W^T (out_dtype bfloat16 or float32).  mode 1: W = [gate rows; up rows], N = 2 * inter,
// out[M, inter] = the gating that pb_set_gating set last (SwiGLU: silu(x Wg^T) * (x Wu^T)).  x [M, K] and W [N, K] bfloat16, 16-byte
// aligned, M <= 128.  loaded: no kernel still on the stream writes W, and it may be read before those have ended.
PB_EXPORT int pb_gemm_tcgen05_stream(int mode, int out_dtype, const void* x, const void* w, void* out, int M, int N, int K, int loaded,
                                     cudaStream_t stream) {
    if (!pb_gemm_tcgen05_stream_supported(mode, M, N, K)) return PB_ERR_BAD_SIZE;
    if ((((uintptr_t)x | (uintptr_t)w) & 15) != 0) return PB_ERR_BAD_SIZE;
    if (out_dtype != PB_BF16 && out_dtype != PB_F32) return PB_ERR_BAD_DTYPE;
    StreamArgs a{};
    a.M = M;
    a.N = N;
    a.K = K;
    a.n_pad = (M + 15) / 16 * 16;
    a.inter = mode == kSwiGLU ? gating_now(N / 2) : GatedInter(0);
    if (mode == kSwiGLU) return out_dtype == PB_BF16 ? launch<kSwiGLU, bf16>(x, w, out, a, loaded != 0, stream) : launch<kSwiGLU, float>(x, w, out, a, loaded != 0, stream);
    return out_dtype == PB_BF16 ? launch<kPlain, bf16>(x, w, out, a, loaded != 0, stream) : launch<kPlain, float>(x, w, out, a, loaded != 0, stream);
}
