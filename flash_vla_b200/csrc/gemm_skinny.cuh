// Weight-streaming GEMM for the action-expert decoder (M <= 128 tokens): out = x[M,K] @ W[K,N].
//
// These GEMMs are bound by the HBM read of W (5-17 MB per call, read once, always cold), so the
// kernel is built around getting every byte of W in flight at once:
//   * the problem is transposed: the 128-wide slice of N is the MMA's M (TMEM lanes), the tokens
//     are its N (TMEM columns): 32, 64, 96 or 128 slots, whichever hold the rows, so no tensor-core or shared-memory work is
//     spent on padding 51 rows to 128, and of the activations only the rows there are (in eights) are fetched;
//   * grid = (N / 128 tiles) x (S K-splits); each CTA owns a W[KC, 128] block, asks TMA for all
//     of it at kernel start (<= 8 boxes of 64 k x 128 n, 128B-swizzled, used in place as an
//     MN-major operand) and issues KC/16 tcgen05.mma into one TMEM accumulator;
//   * the S CTAs of a K-split form a thread-block cluster. Each reads its partial accumulator
//     from TMEM and sends it, registers to distributed shared memory, so that CTA r receives the
//     partials of its slice of tokens; once its barrier has counted them CTA r sums them in rank order
//     (deterministic) and runs the fused epilogue: RMS-factor + RoPE + scatter to Q/K/V, GeGLU,
//     bias, or in-place residual add into the fp32 stream.
// The activation operand arrives by TMA as bf16 rows: either the activation itself (bf16) or the bf16
// shadow that the kernels writing the fp32 residual stream keep beside it; the per-token sum of
// squares for the RMS factor is read back from that operand tile in shared memory while the MMAs run
// and is reduced with the partials. What remains is a chain of latencies (dependency 0.9 us after the
// last CTA of the kernel before, X tile 0.5, MMAs 0.6 to 1.5, exchange 0.5, epilogue 0.6), in which every instruction behind the
// exchange counts, hence the cluster size and the token slots as template parameters. Per launch inside the chain at 51 rows:
// QKV 4.3 us (5.7 with an exchange through bulk copies, run-time sizes and a lane test before the MMAs), attention output 3.9 (5.0),
// gate / up 6.3 (8.2), down 4.6 (6.2); 65 rows, which the general GEMM took before, 77.7 -> 33 us per layer-step. A layer-step by
// token slots: 11 rows 24.1 us on 64 slots and 512 threads, 21.6 on 32 and 256; 32 rows 24.2 -> 22.8; 65 rows 33.3 us on 128 slots with whole
// tiles of 128 activation rows (five k-blocks at a time), 31.1 on 96 with tiles of 72 (seven); 51 rows 25.03 -> 24.96. (256 threads on 64 slots:
// 26.1 at 51 rows; 33 to 64 rows as two parts of 32 slots: no difference.) (An fp32 activation without a shadow is still accepted: the CTA
// then converts its slice in registers.) No separate norm kernel, no global-memory scratch, no
// semaphores.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "gemm_tc5.cuh"

namespace fvla {
namespace skinny {

using tc5::mbar_init;
using tc5::mbar_expect_tx;
using tc5::mbar_wait;
using tc5::tma_load_2d;
using tc5::smem_desc;

constexpr int TN = 128;          // N columns per CTA (MMA M)
constexpr int MAX_KB = 8;        // k-blocks of 64 per CTA
// Beyond 64 slots they go through a ring, and row groups may have twice as many: the down projection of a batch is one launch then instead of two of
// half of K each (eight episodes of 51 rows, 7.3 + 8.8 us end to end; forward 36.2 -> 35.5 ms, of one camera each 18.2 -> 17.5, five episodes 24.9 -> 24.35).
__host__ __device__ constexpr int max_kb(int tok) { return tok > 64 ? 2 * MAX_KB : MAX_KB; }
// TOK: token slots (MMA N): 32, 64, 96 or 128, of which the activation tile fills the rows there are, in eights (the MMAs read on into what
// lies behind; those columns are nobody's). Up to 64 slots every k-block of a CTA has a place in shared memory. With more, a k-block
// takes up to 32 KB and the exchange 48 or 64 KB, so only five to eight have one and the rest reuse the first ones' when their MMAs (and
// the readers of the sums of squares) are done.
constexpr int misc_bytes(int tok) { return tok * 4 + tok * 8 + (2 * max_kb(tok) + 2) * 8 + 32; }     // received sums, own sums, barriers, TMEM slot, flag
constexpr size_t smem_bytes(int tok, int x_rows, int slots) {
    return 1024 + (size_t)slots * (16384 + x_rows * 128) + tok * 512 + misc_bytes(tok);
}
constexpr int slots_of(int tok, int x_rows, int kblocks) {
    int n = kblocks;
    if (tok > 64)
        while (n > 1 && smem_bytes(tok, x_rows, n) > 232448) --n;
    return n;
}
static_assert(smem_bytes(64, 64, MAX_KB) <= 232448 && slots_of(128, 128, MAX_KB) == 5 && slots_of(96, 72, MAX_KB) == 7 && slots_of(128, 128, 2) == 2, "shared memory of one CTA");

enum Epi { EPI_QKV_ROPE = 0, EPI_RESIDUAL = 1, EPI_GEGLU = 2, EPI_BIAS = 3, EPI_RESIDUAL_SUMS = 4 };

struct SkinnyArgs {
    const void* x; int x_f32; int ldx;        // activations [M, K]
    const bf16* x_shadow;                     // optional bf16 copy of an fp32 x, kept current by its writers
    bf16* out_shadow;                         // optional bf16 copy of `out` to maintain (RESIDUAL / BIAS)
    int M, N, K;
    int groups;                               // independent row groups of M rows each, laid end to end (grid.z); 0 or 1 = one
    int kblocks;                              // 64-wide k-blocks per CTA (K / 64 / splits)
    int slots, x_rows;                        // of them in shared memory at a time; rows of an activation tile (a multiple of 8)
    int need_factor;                          // compute rsqrt(mean(x^2)+1e-6) per token
    // epilogue operands
    void* out; int out_f32; int ldo;          // RESIDUAL / BIAS / GEGLU destination
    const bf16* bias; int act;
    const bf16* rope; bf16* q; bf16* k; bf16* v; int heads, head_dim;
    int group_rows, kv_skip;                  // rows per sequence, and rows of a sequence's cache that are not written (0, 0: one sequence)
    uint32_t inv_group;                       // sequence of a row = row * inv_group >> 20 (rows < 128); 0 for one sequence
    bf16* factor_out;                         // optional bf16 copy of the factors
    float* row_sums; int sum_rows;            // RESIDUAL_SUMS: sums of squares of the rows as `out` holds them, per 32 columns, [columns / 128][sum_rows][4]
    int* status;
    uint32_t spin_limit;                       // polls before a wait gives up (0 = the default limit)
    uint32_t expect_extra_bytes;               // self-test only: bytes the owners wait for that no peer sends
    FVLA_DBG_MEMBER
};

// MMA: A = W tile (MN-major, 128 n x 16 k), B = x tile (K-major, 64 tokens x 16 k), D fp32 128x64.
__host__ __device__ constexpr uint32_t skinny_idesc(int tok) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (0u << 16) | ((uint32_t)(tok >> 3) << 17) |
           ((uint32_t)(TN >> 4) << 24);
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Shared memory map (offsets from a 1024-byte aligned base):
//   W      slots x 16 KB     [slot][atom(2)][64 k rows x 128 B]  (atom = 64 of the tile's 128 n)
//   X      slots x rows x 128 B  [slot][token][64 k]           (K-major, 128B swizzle)
//   RED    S x TS x 128 fp32 = TOK x 512 B   partials of the S ranks (the own one too), [src][4 tokens][n][4]
//   SSQ    S x TS fp32       partial sums of squares received, [src][token]
//   ssq_local TOK x 2 fp32, barriers, tmem slot, abort flag
__host__ __device__ constexpr int threads_of(int tok) { return tok == 32 ? 256 : 512; }

__device__ __forceinline__ void st_async4(uint32_t dst, uint32_t bar, float a, float b, float c, float d) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(dst), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async1(uint32_t dst, uint32_t bar, float a) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(dst), "f"(a), "r"(bar) : "memory");
}

template <int EPI, int TOK, int S>          // S: cluster size along K
__global__ void __launch_bounds__(threads_of(TOK), 1)
skinny_gemm_kernel(const SkinnyArgs p, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                   const __grid_constant__ CUtensorMap tmX) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    constexpr bool RESIDUAL = EPI == EPI_RESIDUAL || EPI == EPI_RESIDUAL_SUMS;
    constexpr int THREADS = threads_of(TOK), ISSUERS = TOK <= 64 ? 1 : 2;      // MMA-issuing threads, an accumulator each
    constexpr uint32_t RED_BYTES = TOK * 512, ACC_COLS = TOK == 96 ? 256 : ISSUERS * TOK;
    // The upper warps add up the rows' squares: the MMA issuers' warps come too late for it (gate/up: 1.6 us after the last MMA)
    constexpr int SSQ_WARPS = TOK == 96 ? 6 : THREADS / 64;
    constexpr int TS = TOK / S, COLS = EPI == EPI_GEGLU ? 64 : 128, ITEMS = TS / 4 * COLS, PRE = (ITEMS + THREADS - 1) / THREADS;      // owner: tokens, work items, per thread
    const int KB = p.kblocks, NS = p.slots;
    const uint32_t XB = p.x_rows * 128;
    const uint32_t w_bytes = NS * 16384u;
    const uint32_t sW = base, sX = sW + w_bytes;
    const uint32_t off_red = w_bytes + NS * XB;
    float* ssq_in = reinterpret_cast<float*>(gen + off_red + RED_BYTES);                   // [S][TS]
    float* ssq_local = reinterpret_cast<float*>(gen + off_red + RED_BYTES + TOK * 4);      // [TOK][2]
    const uint32_t off_bar = off_red + RED_BYTES + TOK * 12;
    const uint32_t bars = base + off_bar;                                        // a full barrier per k-block, done, incoming, a free barrier per slot
    constexpr int BARS = max_kb(TOK);
    const uint32_t done_bar = bars + BARS * 8, in_bar = bars + (BARS + 1) * 8, free_bars = bars + (BARS + 2) * 8;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + off_bar + (2 * BARS + 2) * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + off_bar + (2 * BARS + 2) * 8 + 8);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    FVLA_DBG_CTA(p, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
    FVLA_STAMP(0);
    const uint32_t rank = cluster_ctarank();                 // position along K within the cluster
    const int row0 = blockIdx.z * p.M;                       // first row of this CTA's row group in x / out
    const int tile = blockIdx.x;
    const int k0 = (int)rank * KB * 64;
    const int owners = (p.M + TS - 1) / TS;                  // ranks that own at least one real token
    const bool i_own = (int)rank < owners;

    // bf16 activations are fetched by TMA straight into the operand layout (rows past M read as
    // zero); fp32 activations are converted by the CTA further down.
    const bool x_by_tma = !p.x_f32 || p.x_shadow != nullptr;
    if (tid == 32) { tc5::prefetch_tensormap(&tmW); if (EPI == EPI_GEGLU) tc5::prefetch_tensormap(&tmW2); }
    if (tid == 64 && x_by_tma) tc5::prefetch_tensormap(&tmX);
    if (tid == 0) {
        mbar_init(done_bar, ISSUERS);                        // one commit from each issuing thread
        mbar_init(in_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (i_own)                                           // S - 1 peers send
            mbar_expect_tx(in_bar, (uint32_t)(S - 1) * ((uint32_t)(min(TS, p.M - (int)rank * TS) + 3) / 4 * 2048u + (p.need_factor ? TS * 4u : 0u)) + p.expect_extra_bytes);
    }
    auto request_w = [&](int kb, int slot) {
        mbar_expect_tx(bars + kb * 8, x_by_tma ? 16384 + XB : 16384);
        if (EPI == EPI_GEGLU) {
            tma_load_2d(sW + slot * 16384, &tmW, bars + kb * 8, tile * 64, k0 + kb * 64);          // gate columns
            tma_load_2d(sW + slot * 16384 + 8192, &tmW2, bars + kb * 8, tile * 64, k0 + kb * 64);  // up columns
        } else {
            tma_load_2d(sW + slot * 16384, &tmW, bars + kb * 8, tile * TN, k0 + kb * 64);
            tma_load_2d(sW + slot * 16384 + 8192, &tmW, bars + kb * 8, tile * TN + 64, k0 + kb * 64);
        }
    };
    // One lane per k-block sets up that block's barrier and requests its weights: all of this
    // CTA's share of W is in flight within a few hundred cycles of kernel start.
    if (lane == 0 && warp < KB) {
        const int kb = warp;
        mbar_init(bars + kb * 8, 1);
        if (TOK > 64) mbar_init(free_bars + kb * 8, 1 + (p.need_factor ? SSQ_WARPS : 0));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");      // both are signalled by the async proxy
        if (kb < NS) request_w(kb, kb);
    }
    __syncwarp();
    if (warp == 0) {
        tc5::tmem_alloc(base + off_bar + (2 * BARS + 2) * 8, ACC_COLS);
        tc5::tmem_relinquish();
    }
    // Programmatic dependent launch: everything above touched only weights and this CTA's own
    // shared memory, so it may run while the previous kernel in the stream is still finishing.
    // From here on activations written by that kernel are read, so wait for it; then let the
    // next kernel in the stream start its own prologue.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (x_by_tma && lane == 0 && warp < NS)
        tma_load_2d(sX + warp * XB, &tmX, bars + warp * 8, k0 + warp * 64, row0);
    // Tell the cluster this CTA is running (barriers initialised); peers wait for that before
    // sending anything into its shared memory.
    // (the fence after the barrier initialisation already published it cluster-wide, so a relaxed
    // arrive is enough; a releasing one would also wait for this thread's outstanding requests)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    // Epilogue operands that do not depend on the product (RoPE entries, residual values, bias) are
    // fetched now, so that their latency overlaps the weight stream instead of following the MMA.
    // Owner work items: (4 tokens of this rank's slice) x (column); after two lanes have swapped, a lane finishes two tokens
    // (ta, ta + 1) of two adjacent columns.
    // All index arithmetic is done here too: what follows the exchange is on the critical path of 16 warps.
    const int odd = lane & 1;
    const float inv_k = 1.0f / (float)p.K;
    uint4 pre[PRE];
    bf16* dst[PRE];                                           // QKV: Q, K or V
    uint32_t at[PRE][2];                                      // element offsets of the two tokens in the destination
    bool live[PRE][2], work[PRE];
#pragma unroll
    for (int j = 0; j < PRE; ++j) {
        pre[j] = make_uint4(0, 0, 0, 0);
        dst[j] = nullptr;
        const int item = tid + j * THREADS, c = item % COLS & ~1, n = tile * COLS + c, t4 = (int)rank * TS + item / COLS * 4, ta = t4 + odd * 2;
        work[j] = item < ITEMS && t4 < p.M;                   // uniform within a warp
        live[j][0] = work[j] && ta < p.M;
        live[j][1] = work[j] && ta + 1 < p.M;
        if (EPI == EPI_QKV_ROPE) {
            const int hd = p.head_dim, qd = p.heads * hd;
            const int seq0 = (int)((uint32_t)ta * p.inv_group >> 20), seq1 = (int)((uint32_t)(ta + 1) * p.inv_group >> 20);
            if (n < qd + hd) {
                const bf16* rp = p.rope + (n % hd);
                if (live[j][0]) pre[j].x = __ldg(reinterpret_cast<const uint32_t*>(rp + (size_t)(ta - seq0 * p.group_rows) * hd));
                if (live[j][1]) pre[j].z = __ldg(reinterpret_cast<const uint32_t*>(rp + (size_t)(ta + 1 - seq1 * p.group_rows) * hd));
            }
            if (n < qd) {
                dst[j] = p.q;
                at[j][0] = (uint32_t)(ta * qd + n); at[j][1] = at[j][0] + qd;
            } else {
                dst[j] = n < qd + hd ? p.k : p.v;
                const int col = n - qd - (n < qd + hd ? 0 : hd);
                at[j][0] = (uint32_t)((ta + seq0 * p.kv_skip) * hd + col); at[j][1] = (uint32_t)((ta + 1 + seq1 * p.kv_skip) * hd + col);
            }
        } else {
            at[j][0] = (uint32_t)((row0 + ta) * p.ldo + n); at[j][1] = at[j][0] + p.ldo;
            if (RESIDUAL && p.out_f32) {
                if (live[j][0]) { const uint2 a = *reinterpret_cast<const uint2*>(static_cast<const float*>(p.out) + at[j][0]); pre[j].x = a.x; pre[j].y = a.y; }
                if (live[j][1]) { const uint2 a = *reinterpret_cast<const uint2*>(static_cast<const float*>(p.out) + at[j][1]); pre[j].z = a.x; pre[j].w = a.y; }
            } else if (RESIDUAL) {
                const float2 a = unpack_bf16x2(live[j][0] ? *reinterpret_cast<const uint32_t*>(static_cast<const bf16*>(p.out) + at[j][0]) : 0u);
                const float2 b = unpack_bf16x2(live[j][1] ? *reinterpret_cast<const uint32_t*>(static_cast<const bf16*>(p.out) + at[j][1]) : 0u);
                pre[j] = make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
            } else if (EPI == EPI_BIAS) {
                const float2 b = unpack_bf16x2(__ldg(reinterpret_cast<const uint32_t*>(p.bias + n)));
                pre[j] = make_uint4(__float_as_uint(b.x), __float_as_uint(b.y), __float_as_uint(b.x), __float_as_uint(b.y));
            }
        }
    }

    FVLA_STAMP(1);
    // Activation slice -> bf16 K-major operand (manual 128B swizzle), plus partial sums of squares.
    // Each thread has four 32-byte loads in flight at a time.
    if (TOK == 64 && !x_by_tma) {
        const int chunks_per_row = KB * 8;                   // 16-byte (8 x bf16) chunks per token
        const int total = TOK * chunks_per_row;              // 512 (KB = 1) ... 4096 (KB = 8)
        for (int it0 = 0; it0 * THREADS < total; it0 += 4) {
            float4 ra[4], rb[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int idx = (it0 + u) * THREADS + tid;
                const int t = idx / chunks_per_row, c = idx % chunks_per_row;
                ra[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                rb[u] = ra[u];
                if (idx < total && t < p.M) {
                    const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + (size_t)(row0 + t) * p.ldx + k0 + c * 8);
                    ra[u] = src[0];
                    rb[u] = src[1];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int idx = (it0 + u) * THREADS + tid;
                if ((it0 + u) * THREADS < total) {           // uniform across the CTA
                    const int t = idx / chunks_per_row, c = idx % chunks_per_row;
                    const int kb = c >> 3, cc = c & 7;
                    uint4 packed = make_uint4(pack_bf16x2(ra[u].x, ra[u].y), pack_bf16x2(ra[u].z, ra[u].w),
                                              pack_bf16x2(rb[u].x, rb[u].y), pack_bf16x2(rb[u].z, rb[u].w));
                    *reinterpret_cast<uint4*>(gen + w_bytes + kb * 8192 + t * 128 + ((cc ^ (t & 7)) << 4)) = packed;
                    if (p.need_factor) {
                        float ss = ra[u].x * ra[u].x + ra[u].y * ra[u].y + ra[u].z * ra[u].z + ra[u].w * ra[u].w +
                                   rb[u].x * rb[u].x + rb[u].y * rb[u].y + rb[u].z * rb[u].z + rb[u].w * rb[u].w;
                        // chunks of one token sit in consecutive lanes: reduce over groups of min(32, chunks_per_row)
                        const int group = chunks_per_row < 32 ? chunks_per_row : 32;
                        for (int o = group >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                        if ((lane & (group - 1)) == 0) ssq_local[t * 2 + (c >> 5)] = ss;      // slot 1 only when KB = 8
                    }
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> visible to the MMA
    }
    tc5::tc_fence_before();
    __syncthreads();
    tc5::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every peer has initialised its barriers
    auto hand_out_ss = [&](int t, float ss) {          // a row's sum of squares over this CTA's K slice, to the row's owner
        const int r = t / TS, slot = (int)rank * TS + t % TS;
        if (r == (int)rank) ssq_in[slot] = ss;
        else if (r < owners) st_async1(map_to_cta(base + off_red + RED_BYTES + slot * 4u, (uint32_t)r), map_to_cta(in_bar, (uint32_t)r), ss);
    };
    FVLA_STAMP(2);

    // Up to 64 slots: one thread adds up all k-blocks in order in one accumulator, so that a product is a single fp32 sum over the CTA's
    // K slice from front to back, whatever issues it (decodes of several steps amplify a changed order of summation). Its warp
    // waits for all k-blocks at once, a lane each: they land within 0.1 us of one another, and waits in between take longer. MMAs
    // done after the X tile, at 51 rows: QKV 0.87 us, o 0.87, gate / up 1.9, down 1.3 (two threads with an accumulator each 0.92, 0.87, 2.4, 1.7).
    // Beyond 64 slots: two threads issue the k-blocks in turn, each into an accumulator of its own.
    constexpr uint32_t idesc = skinny_idesc(TOK);
    const uint64_t ad = smem_desc(sW, 8192, 1024), bd = smem_desc(sX, 16, 1024);
    auto issue_block = [&](int slot, uint32_t acc, bool first) {
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)
            tc5::umma_bf16(acc, ad + slot * (16384 >> 4) + k16 * (2048 >> 4), bd + slot * (XB >> 4) + k16 * (32 >> 4), idesc, !first || k16 > 0 ? 1u : 0u);
    };
    if (ISSUERS == 1 && __shfl_sync(0xffffffffu, warp, 0) == 0) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bars + min(lane, KB - 1) * 8, 0, abort_flag));
        __syncwarp();                                        // what the lanes saw is in order before the elected lane's MMAs
        tc5::tc_fence_after();
        if (tc5::elect_one()) {
#pragma unroll
            for (int kb = 0; kb < MAX_KB; ++kb)
                if (kb < KB && ok) issue_block(kb, tmem, kb == 0);
            tc5::umma_commit(done_bar);
        }
    }
    if (ISSUERS == 2 && warp < 2 && lane == 0) {
        for (int kb = warp, slot = warp; kb < KB; kb += 2) {
            if (!mbar_wait(bars + kb * 8, 0, abort_flag)) break;
            tc5::tc_fence_after();
            issue_block(slot, tmem + warp * TOK, kb < 2);
            if (kb + NS < KB) tc5::umma_commit(free_bars + kb * 8);
            slot += 2;
            if (slot >= NS) slot -= NS;
        }
        tc5::umma_commit(done_bar);
    }
    // The k-blocks that had no slot of their own: one lane asks for block kb + NS once block kb's slot is free, that is read
    // by its MMAs and by the warps below (neither this lane's nor the issuers': those would wait for themselves).
    if (TOK > 64 && warp == 2 && lane == 0)
        for (int kb = 0, slot = 0; kb + NS < KB; ++kb) {
            if (!mbar_wait(free_bars + kb * 8, 0, abort_flag)) break;
            request_w(kb + NS, slot);
            tma_load_2d(sX + slot * XB, &tmX, bars + (kb + NS) * 8, k0 + (kb + NS) * 64, row0);
            if (++slot == NS) slot = 0;
        }
    __syncwarp();
    if (x_by_tma && p.need_factor && warp >= THREADS / 32 - SSQ_WARPS) {
        // Sums of squares over this CTA's K slice, read back from the bf16 operand tile in shared
        // memory while the MMAs run (4 or 2 lanes per token).
        constexpr int LPT = SSQ_WARPS * 32 / TOK;            // lanes per token
        const int st = tid - (THREADS - SSQ_WARPS * 32), t = st / LPT, sub = st % LPT;
        float part[8 / LPT] = {};                            // one sum per 16-byte piece of the rows, added up pairwise below
        for (int kb = 0, slot = 0; kb < KB; ++kb) {
            mbar_wait(bars + kb * 8, 0, abort_flag);
#pragma unroll
            for (int h = 0; h < 8 / LPT; ++h) {
                const uint4 a = *reinterpret_cast<const uint4*>(gen + w_bytes + slot * XB + t * 128 + (sub + h * LPT) * 16);
                const float2 f0 = unpack_bf16x2(a.x), f1 = unpack_bf16x2(a.y), f2 = unpack_bf16x2(a.z), f3 = unpack_bf16x2(a.w);
                part[h] += f0.x * f0.x + f0.y * f0.y + f1.x * f1.x + f1.y * f1.y + f2.x * f2.x + f2.y * f2.y + f3.x * f3.x + f3.y * f3.y;
            }
            if (TOK > 64 && kb + NS < KB) {
                __syncwarp();
                if (lane == 0) tc5::mbar_arrive(free_bars + kb * 8);
            }
            if (++slot == NS) slot = 0;
        }
#pragma unroll
        for (int o = 1; o < LPT; o <<= 1)
#pragma unroll
            for (int h = 0; h < 8 / LPT; ++h) part[h] += __shfl_xor_sync(0xffffffffu, part[h], o);
#pragma unroll
        for (int n = 8 / LPT; n > 1; n /= 2)
#pragma unroll
            for (int h = 0; h < n / 2; ++h) part[h] = part[2 * h] + part[2 * h + 1];
        if (sub == 0) hand_out_ss(t, part[0]);
    }
    if (TOK == 64 && !x_by_tma && p.need_factor && tid < TOK)
        hand_out_ss(tid, tid < p.M ? ssq_local[tid * 2] + (KB == 8 ? ssq_local[tid * 2 + 1] : 0.f) : 0.f);
    mbar_wait(done_bar, 0, abort_flag);                // (after an expired wait the sums are garbage and the status says so)
    __syncwarp();
    tc5::tc_fence_after();
    FVLA_STAMP(3);
    // Hand the partial tile out: warp w reads TMEM lanes 32 (w & 3) .. + 32 (its columns) and tokens 16 (w >> 2) .. + 16 (and
    // + 64), and what a thread holds of four tokens goes as 16 bytes from registers to their owner's receive buffer
    // [src][4 tokens][column][4], which counts the bytes on its barrier; the own slice takes an ordinary store. (Staged in
    // shared memory and sent by bulk copies the exchange took 0.4 us longer.)
    const uint32_t red_mine = base + off_red + rank * (TS * 512u);
#pragma unroll
    for (int h = 0; h < (TOK * 8 + THREADS - 1) / THREADS; ++h) {
        const int q = warp & 3, g = (warp >> 2) + h * (THREADS / 128);
        if (TOK == 96 && g >= TOK / 16) break;
        float part[16];
        tc5::tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + g * 16, part);
        if (ISSUERS == 2 && KB > 1) {
            float second[16];
            tc5::tmem_ld16(tmem + TOK + ((uint32_t)(q * 32) << 16) + g * 16, second);
#pragma unroll
            for (int t = 0; t < 16; ++t) part[t] += second[t];
        }
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
            const int token = g * 16 + t, r = token / TS;
            if (token >= p.M) break;
            const uint32_t at = red_mine + (uint32_t)((token % TS) >> 2) * 2048u + (q * 32 + lane) * 16u;
            if (r == (int)rank) *reinterpret_cast<float4*>(gen + (at - base)) = make_float4(part[t], part[t + 1], part[t + 2], part[t + 3]);
            else st_async4(map_to_cta(at, (uint32_t)r), map_to_cta(in_bar, (uint32_t)r), part[t], part[t + 1], part[t + 2], part[t + 3]);
        }
    }
    tc5::tc_fence_before();
    __syncthreads();                                   // own slice and sums stored, accumulators read
    FVLA_STAMP(4);
    // Owner phase: this CTA finishes tokens [rank*TS, rank*TS + TS), summing partials in rank order.
    if (i_own) mbar_wait(in_bar, 0, abort_flag, p.spin_limit ? p.spin_limit : tc5::kSpinLimit);
    __syncwarp();
    FVLA_STAMP(5);
    // Nobody may leave while a peer can still send to it. Past this arrive nothing is outstanding towards this CTA, and the wait
    // at the end finds the peers here too.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    if (i_own) {
        const float* red = reinterpret_cast<const float*>(gen + off_red);
#pragma unroll
        for (int j = 0; j < PRE; ++j) {
            if (!work[j]) continue;
            const int item = tid + j * THREADS, group = item / COLS, c = item % COLS, tl = group * 4 + odd * 2;
            auto sum_sources = [&](int col, float2 (&t)[2]) {
                const float* src = red + (group * 128 + col) * 4;
                float4 in[S];                              // all sources requested before the first is used
#pragma unroll
                for (int s = 0; s < S; ++s) in[s] = *reinterpret_cast<const float4*>(src + s * TS * 128);
                float4 a = in[0];
#pragma unroll
                for (int s = 1; s < S; ++s) { a.x += in[s].x; a.y += in[s].y; a.z += in[s].z; a.w += in[s].w; }
                // swap with the lane of the neighbouring column: even lanes keep tokens 0, 1, odd lanes 2, 3
                const float r0 = __shfl_xor_sync(0xffffffffu, odd ? a.x : a.z, 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? a.y : a.w, 1);
                t[0] = odd ? make_float2(r0, a.z) : make_float2(a.x, r0);
                t[1] = odd ? make_float2(r1, a.w) : make_float2(a.y, r1);
            };
            float factor[2] = {1.f, 1.f};
            if (p.need_factor) {
                float2 ss = make_float2(0.f, 0.f);
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float2 q = *reinterpret_cast<const float2*>(ssq_in + s * TS + tl);
                    ss.x += q.x; ss.y += q.y;
                }
                factor[0] = rsqrtf(ss.x * inv_k + 1e-6f);
                factor[1] = rsqrtf(ss.y * inv_k + 1e-6f);
            }
            float2 v[2], up[2];
            float squares[2] = {0.f, 0.f};
            sum_sources(c, v);
            if (EPI == EPI_GEGLU) sum_sources(64 + c, up);        // columns 0..63 of the tile are gate columns, 64..127 the matching up columns
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (!live[j][i]) break;
                if (p.need_factor && p.factor_out && tile == 0 && c < 2) p.factor_out[(int)rank * TS + tl + i] = __float2bfloat16_rn(factor[i]);
                const uint32_t p0 = i == 0 ? pre[j].x : pre[j].z, p1 = i == 0 ? pre[j].y : pre[j].w;
                if (EPI == EPI_QKV_ROPE) {
                    float v0 = v[i].x * factor[i], v1 = v[i].y * factor[i];
                    if (dst[j] != p.v) {
                        const float2 cs = unpack_bf16x2(p0);
                        const float r0 = v0 * cs.x - v1 * cs.y, r1 = v1 * cs.x + v0 * cs.y;
                        v0 = r0; v1 = r1;
                    }
                    *reinterpret_cast<uint32_t*>(dst[j] + at[j][i]) = pack_bf16x2(v0, v1);
                } else if (EPI == EPI_GEGLU) {
                    const float f = factor[i];
                    *reinterpret_cast<uint32_t*>(static_cast<bf16*>(p.out) + at[j][i]) =
                        pack_bf16x2(gelu_f(v[i].x * f) * (up[i].x * f), gelu_f(v[i].y * f) * (up[i].y * f));
                } else {
                    // p0, p1 = bias (EPI_BIAS) or residual (EPI_RESIDUAL)
                    float v0 = v[i].x + __uint_as_float(p0), v1 = v[i].y + __uint_as_float(p1);
                    if (EPI == EPI_BIAS && p.act == 2) { v0 = silu_f(v0); v1 = silu_f(v1); }
                    const uint32_t word = pack_bf16x2(v0, v1);
                    if (p.out_shadow) *reinterpret_cast<uint32_t*>(p.out_shadow + at[j][i]) = word;
                    if (p.out_f32) *reinterpret_cast<float2*>(static_cast<float*>(p.out) + at[j][i]) = make_float2(v0, v1);
                    else *reinterpret_cast<uint32_t*>(static_cast<bf16*>(p.out) + at[j][i]) = word;
                    if (EPI == EPI_RESIDUAL_SUMS) {
                        const float2 w = p.out_f32 ? make_float2(v0, v1) : unpack_bf16x2(word);
                        squares[i] = w.x * w.x + w.y * w.y;
                    }
                }
            }
            if (EPI == EPI_RESIDUAL_SUMS) {      // a warp has 32 columns of four tokens, even lanes the first two
#pragma unroll
                for (int o = 2; o < 32; o <<= 1) {
                    squares[0] += __shfl_xor_sync(0xffffffffu, squares[0], o);
                    squares[1] += __shfl_xor_sync(0xffffffffu, squares[1], o);
                }
                const int part = (tile * TN + c) >> 5, row = row0 + (int)rank * TS + tl;
                float* to = p.row_sums + ((size_t)(part >> 2) * p.sum_rows + row) * 4 + (part & 3);
                if (lane < 2 && live[j][0]) to[0] = squares[0];
                if (lane < 2 && live[j][1]) to[4] = squares[1];
            }
        }
    }
    if (warp == 0) {
        __syncwarp();
        tc5::tc_fence_after();
        tc5::tmem_dealloc(tmem, ACC_COLS);
    }
    FVLA_STAMP(6);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    FVLA_STAMP(7);
    if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 2);
}

// ---- host side ---------------------------------------------------------------------------------
struct SkinnyPlan { int tok, splits, kblocks, tiles; bool ok; int slots, x_rows; size_t smem; };      // the last three by place_skinny

inline void place_skinny(SkinnyPlan& pl, int M, bool bf16_operand) {
    pl.x_rows = bf16_operand ? (M + 7) / 8 * 8 : pl.tok;      // (the in-kernel conversion of fp32 rows fills the whole tile)
    pl.slots = slots_of(pl.tok, pl.x_rows, pl.kblocks);
    pl.smem = smem_bytes(pl.tok, pl.x_rows, pl.slots);
}

// bf16_operand: rows as bf16 (the activation itself or its shadow).
inline SkinnyPlan plan_skinny(int M, int N, int K, bool geglu, bool bf16_operand, int groups = 1) {
    SkinnyPlan pl{};
    pl.ok = false;
    const int tile_n = geglu ? 64 : TN;
    if (M <= 0 || M > 128 || N % tile_n || K % 64) return pl;
    // The fewest token slots that hold the rows: measured per layer-step above. (The in-kernel conversion of fp32 rows exists for 64.)
    pl.tok = M <= 32 && bf16_operand ? 32 : (M <= 64 ? 64 : (M <= 96 ? 96 : 128));
    pl.tiles = N / tile_n;
    const int kb_total = K / 64;
    PlanChoice pinned;
    if (plan_lookup(M, N, K, geglu ? PLAN_SKINNY_DUAL : PLAN_SKINNY, &pinned)) {
        // a pinned cluster size: 1, 2, 4 or 8 CTAs along K, at most 8 k-blocks each
        const int s = pinned.splits;
        if (s < (pl.tok <= 64 ? 1 : 2) || s > 8 || (s & (s - 1)) || kb_total % s || kb_total / s > MAX_KB || ((kb_total / s) & (kb_total / s - 1))) return pl;
        pl.splits = s;
        pl.kblocks = kb_total / s;
        pl.ok = true;
        return pl;
    }
    // largest cluster (<= 8) that divides the k-blocks, keeps <= 8 k-blocks per CTA and stays near one wave
    int best = 0;
    for (int s = pl.tok <= 64 ? 1 : 2; s <= 8; s *= 2) {       // 8 = largest portable cluster; larger ones schedule in waves
        if (kb_total % s) continue;
        const int kb = kb_total / s;
        if (kb > MAX_KB || kb < 1 || (kb & (kb - 1))) continue;
        if (pl.tiles * s > 148 && best) break;
        best = s;
    }
    if (!best) return pl;
    if (groups > 1) {
        // Several row groups in one launch multiply the CTA count. Clusters are placed GPC by GPC: about 33
        // clusters of 4 or 15 of 8 are resident at once, so prefer the largest split whose clusters of all
        // groups are resident together (one wave) over the single-group choice.
        for (int s = best; s >= (pl.tok <= 64 ? 1 : 2); s /= 2) {
            const int kb = kb_total / s;
            if (kb_total % s || kb > max_kb(pl.tok)) break;
            const int resident = s >= 8 ? 15 * 8 : (s == 4 ? 33 * 4 : 148);
            if (pl.tiles * s * groups <= resident) { best = s; break; }
        }
    }
    pl.splits = best;
    pl.kblocks = kb_total / best;
    pl.ok = true;
    return pl;
}

// Whether the kernel takes a shape. More than 64 rows need the operand as bf16 rows (the activation itself or its shadow):
// the in-kernel conversion of fp32 rows exists for 64 token slots only.
// A shape of more than 64 rows with a plan of the general kernels (`general_kind`) pinned for it is theirs; -1: no such plan.
inline bool skinny_supports(int M, int N, int K, bool geglu, bool bf16_operand, int general_kind) {
    const SkinnyPlan pl = plan_skinny(M, N, K, geglu, bf16_operand);
    PlanChoice pinned;
    return pl.ok && (pl.tok <= 64 || (bf16_operand && !plan_lookup(M, N, K, general_kind, &pinned)));
}

template <int EPI, int TOK, int S>
inline int launch_skinny_cfg(SkinnyArgs a, const SkinnyPlan& pl, const void* W, const void* W2, int ldw, cudaStream_t st) {
    a.kblocks = pl.kblocks; a.slots = pl.slots; a.x_rows = pl.x_rows;
    const int groups = a.groups > 1 ? a.groups : 1;
    if (groups > 1 && (EPI == EPI_QKV_ROPE || a.need_factor || (a.x_f32 && a.x_shadow == nullptr))) {
        set_error("skinny gemm: row groups are only built for the bias / residual forms with a bf16 operand");
        return FVLA_ERR_UNSUPPORTED;
    }
    if (TOK != 64 && a.x_f32 && a.x_shadow == nullptr) { set_error("skinny gemm: fp32 rows without a bf16 copy take the 64-slot form only (%d slots)", TOK); return FVLA_ERR_UNSUPPORTED; }
    auto kern = skinny_gemm_kernel<EPI, TOK, S>;
    static PerDeviceFlag configured;
    if (!configured.get()) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return FVLA_ERR_LAUNCH; }
        configured.set();
    }
    CUtensorMap tmW, tmW2, tmX;
    int rc = tc5::make_map(&tmW, W, (uint64_t)a.N, (uint64_t)a.K, (uint64_t)ldw, 64, 64);
    if (rc) return rc;
    if (W2 == nullptr) tmW2 = tmW;                           // unused by the kernel in this case
    else rc = tc5::make_map(&tmW2, W2, (uint64_t)a.N, (uint64_t)a.K, (uint64_t)ldw, 64, 64);
    if (rc) return rc;
    if (a.x_f32 && a.x_shadow == nullptr) tmX = tmW;         // unused by the kernel in this case
    else rc = tc5::make_map(&tmX, a.x_f32 ? (const void*)a.x_shadow : a.x, (uint64_t)a.K, (uint64_t)a.M * groups, (uint64_t)a.ldx, 64, (uint32_t)pl.x_rows);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.tiles, pl.splits, groups);
    cfg.blockDim = dim3(threads_of(TOK), 1, 1);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = pl.splits;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a, tmW, tmW2, tmX);
    if (e != cudaSuccess) { set_error("skinny_gemm_kernel: %s", cudaGetErrorString(e)); return FVLA_ERR_LAUNCH; }
    return check_launch("skinny_gemm_kernel");
}

template <int EPI, int TOK>
inline int launch_skinny_tok(const SkinnyArgs& a, const SkinnyPlan& pl, const void* W, const void* W2, int ldw, cudaStream_t st) {
    switch (pl.splits) {
        case 1:
            if constexpr (TOK <= 64) return launch_skinny_cfg<EPI, TOK, 1>(a, pl, W, W2, ldw, st);
            else { set_error("skinny gemm: no cluster of one for %d rows", a.M); return FVLA_ERR_UNSUPPORTED; }
        case 2: return launch_skinny_cfg<EPI, TOK, 2>(a, pl, W, W2, ldw, st);
        case 4: return launch_skinny_cfg<EPI, TOK, 4>(a, pl, W, W2, ldw, st);
        default: return launch_skinny_cfg<EPI, TOK, 8>(a, pl, W, W2, ldw, st);
    }
}

template <int EPI>
inline int launch_skinny(const SkinnyArgs& a, const void* W, const void* W2, int ldw, cudaStream_t st) {
    const bool bf16_operand = !a.x_f32 || a.x_shadow != nullptr;
    SkinnyPlan pl = plan_skinny(a.M, a.N, a.K, EPI == EPI_GEGLU, bf16_operand, a.groups > 1 ? a.groups : 1);
    if (!pl.ok) { set_error("skinny gemm: shape %dx%dx%d not supported", a.M, a.N, a.K); return FVLA_ERR_UNSUPPORTED; }
    place_skinny(pl, a.M, bf16_operand);
    switch (pl.tok) {
        case 32: return launch_skinny_tok<EPI, 32>(a, pl, W, W2, ldw, st);
        case 64: return launch_skinny_tok<EPI, 64>(a, pl, W, W2, ldw, st);
        case 96: return launch_skinny_tok<EPI, 96>(a, pl, W, W2, ldw, st);
        default: return launch_skinny_tok<EPI, 128>(a, pl, W, W2, ldw, st);
    }
}

}  // namespace skinny
}  // namespace fvla
