// Streaming-softmax attention for the three attention shapes of Pi0.
//
//   * SigLIP: per (view, head), 256 queries x 256 keys, head_dim 72 (padded to 80 in shared
//     memory), Q/K/V interleaved in one packed (tokens, 3 * 1152) buffer.
//   * Prefix encoder: multi-query; the (token, head) axes collapse to one flat query axis of
//     S * 8 rows against one K/V head of S keys, head_dim 256, unmasked.
//   * Action-expert decoder: same flat multi-query form, 408 queries x (S + 51) keys, with the
//     Pi0 mask (the state token's 8 rows see keys j <= S only) and the keys split across CTAs
//     (flash-decoding); a second kernel merges the per-split partials by log-sum-exp.
//
// One CTA = 64 query rows, 4 warps of 16 rows; K/V stream through a 2-stage cp.async ring in
// 64-key blocks; scores and probabilities never leave registers.
#pragma once

#include "common.cuh"
#include "gemm_tc5.cuh"

namespace fvla {

struct AttnArgs {
    const bf16* q; const bf16* k; const bf16* v;
    bf16* out;                 // direct mode: (nq, o_stride) rows
    float* part_o;             // split mode: (splits, nq_pad, HD) fp32, normalised per split
    float* part_lse;           // split mode: (splits, nq_pad) log2-domain log-sum-exp
    int q_stride, k_stride, v_stride, o_stride;          // row strides in elements
    long long q_bs0, q_bs1, k_bs0, k_bs1, v_bs0, v_bs1, o_bs0, o_bs1;   // batch strides
    int batch_inner;           // blockIdx.y = b0 * batch_inner + b1
    int nq, nk, hd;            // rows, keys, real head dim
    int nq_pad;
    float scale_log2;          // softmax scale * log2(e)
    int mask_rows, mask_key_le;   // rows < mask_rows only see keys j <= mask_key_le
    int splits, keys_per_split;
};

// HD: padded head dim, multiple of 16. STAGES: K/V tiles in shared memory; 2 overlaps the next
// tile's load with this tile's math inside the CTA, 1 halves the footprint so that two CTAs share an SM
// and overlap each other instead.
template <int HD, int STAGES>
__global__ void __launch_bounds__(128) attention_kernel(const AttnArgs p) {
    constexpr int BQ = 64, BKV = 64;
    constexpr int PITCH = HD * 2 + 16;          // bytes; +16 keeps ldmatrix rows on distinct banks
    constexpr int CH = HD / 8;                  // 16-byte chunks per row
    constexpr int TILE = 64 * PITCH;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sQ = smem_u32(smem);
    const uint32_t sKV = sQ + TILE;             // stage s: K at sKV + s*2*TILE, V right after

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // the next kernel may be scheduled
    asm volatile("griddepcontrol.wait;" ::: "memory");      // no-op unless launched as a dependent
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q0 = blockIdx.x * BQ;
    const int b0 = blockIdx.y / p.batch_inner, b1 = blockIdx.y % p.batch_inner;
    const bf16* Q = p.q + b0 * p.q_bs0 + b1 * p.q_bs1;
    const bf16* K = p.k + b0 * p.k_bs0 + b1 * p.k_bs1;
    const bf16* V = p.v + b0 * p.v_bs0 + b1 * p.v_bs1;
    const int split = blockIdx.z;
    const int key_beg = split * p.keys_per_split;
    const int key_end = min(p.nk, key_beg + p.keys_per_split);
    const int nblocks = (key_end - key_beg + BKV - 1) / BKV;
    const int hd_chunks = (p.hd + 7) / 8;       // chunks holding real data (hd % 8 == 0)

    auto load_rows = [&](uint32_t dst, const bf16* src, int stride, int row0, int row_end) {
        for (int idx = tid; idx < 64 * CH; idx += 128) {
            int r = idx / CH, c = idx % CH;
            bool ok = (row0 + r) < row_end && c < hd_chunks;
            const bf16* s = ok ? src + (size_t)(row0 + r) * stride + c * 8 : src;
            cp_async16(dst + r * PITCH + c * 16, s, ok ? 16 : 0);
        }
    };

    load_rows(sQ, Q, p.q_stride, q0, p.nq);
    if (nblocks > 0) {
        load_rows(sKV, K, p.k_stride, key_beg, key_end);
        load_rows(sKV + TILE, V, p.v_stride, key_beg, key_end);
    }
    cp_async_commit();

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const int row_lo = q0 + warp * 16 + (lane >> 2);      // this thread's two rows: row_lo, row_lo + 8

    for (int jb = 0; jb < nblocks; ++jb) {
        const int stage = STAGES == 2 ? (jb & 1) : 0;
        if (STAGES == 2) {
            if (jb + 1 < nblocks) {
                const int kb = key_beg + (jb + 1) * BKV;
                load_rows(sKV + (stage ^ 1) * 2 * TILE, K, p.k_stride, kb, key_end);
                load_rows(sKV + (stage ^ 1) * 2 * TILE + TILE, V, p.v_stride, kb, key_end);
            }
            cp_async_commit();
            cp_async_wait<1>();
        } else {
            if (jb > 0) {                    // the barrier closing the previous iteration freed the tile
                const int kb = key_beg + jb * BKV;
                load_rows(sKV, K, p.k_stride, kb, key_end);
                load_rows(sKV + TILE, V, p.v_stride, kb, key_end);
                cp_async_commit();
            }
            cp_async_wait<0>();
        }
        __syncthreads();
        const uint32_t sK = sKV + stage * 2 * TILE, sV = sK + TILE;

        // S = Q K^T for this warp's 16 rows x 64 keys
        float s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
            uint32_t a[4];
            ldmatrix_x4(a, sQ + (warp * 16 + (lane & 15)) * PITCH + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
            for (int nj = 0; nj < 4; ++nj) {
                uint32_t b[4];
                int key = nj * 16 + (lane & 7) + (lane >> 4) * 8;
                ldmatrix_x4(b, sK + key * PITCH + (kk * 2 + ((lane >> 3) & 1)) * 16);
                mma_bf16_16816(s[2 * nj], a, b[0], b[1]);
                mma_bf16_16816(s[2 * nj + 1], a, b[2], b[3]);
            }
        }

        // scale, mask, online softmax (log2 domain)
        const int kbase = key_beg + jb * BKV;
        float m_new[2] = {m_run[0], m_run[1]};
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                int key = kbase + ni * 8 + (lane & 3) * 2 + (e & 1);
                int row = row_lo + (e >> 1) * 8;
                bool keep = key < key_end && (row >= p.mask_rows || key <= p.mask_key_le);
                float v = keep ? s[ni][e] * p.scale_log2 : -INFINITY;
                s[ni][e] = v;
                m_new[e >> 1] = fmaxf(m_new[e >> 1], v);
            }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            m_new[h] = fmaxf(m_new[h], __shfl_xor_sync(0xffffffffu, m_new[h], 1));
            m_new[h] = fmaxf(m_new[h], __shfl_xor_sync(0xffffffffu, m_new[h], 2));
        }
        float alpha[2], m_use[2], psum[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            m_use[h] = m_new[h] == -INFINITY ? 0.f : m_new[h];       // fully masked so far
            alpha[h] = exp2f(m_run[h] - m_use[h]);                   // m_run = -inf -> 0
            m_run[h] = m_new[h];
        }
#pragma unroll
        for (int ni = 0; ni < 8; ++ni)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float pv = exp2f(s[ni][e] - m_use[e >> 1]);
                s[ni][e] = pv;
                psum[e >> 1] += pv;
            }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            psum[h] += __shfl_xor_sync(0xffffffffu, psum[h], 1);
            psum[h] += __shfl_xor_sync(0xffffffffu, psum[h], 2);
            l_run[h] = l_run[h] * alpha[h] + psum[h];
        }
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) {
            o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
            o[i][2] *= alpha[1]; o[i][3] *= alpha[1];
        }

        // O += P V
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk) {
            uint32_t a[4];
            a[0] = pack_bf16x2(s[2 * kk][0], s[2 * kk][1]);
            a[1] = pack_bf16x2(s[2 * kk][2], s[2 * kk][3]);
            a[2] = pack_bf16x2(s[2 * kk + 1][0], s[2 * kk + 1][1]);
            a[3] = pack_bf16x2(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
            for (int dj = 0; dj < HD / 16; ++dj) {
                uint32_t b[4];
                int key = kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8;
                ldmatrix_x4_trans(b, sV + key * PITCH + (dj * 2 + (lane >> 4)) * 16);
                mma_bf16_16816(o[2 * dj], a, b[0], b[1]);
                mma_bf16_16816(o[2 * dj + 1], a, b[2], b[3]);
            }
        }
        __syncthreads();       // everyone is done with this stage before it is refilled
    }
    cp_async_wait<0>();

    float inv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) inv[h] = l_run[h] > 0.f ? 1.0f / l_run[h] : 0.f;

    if (p.part_o) {
        float* po = p.part_o + ((size_t)split * p.nq_pad) * HD;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int row = row_lo + h * 8;
            if (row < p.nq) {
#pragma unroll
                for (int i = 0; i < HD / 8; ++i) {
                    int d = i * 8 + (lane & 3) * 2;
                    *reinterpret_cast<float2*>(po + (size_t)row * HD + d) =
                        make_float2(o[i][2 * h] * inv[h], o[i][2 * h + 1] * inv[h]);
                }
                if ((lane & 3) == 0)
                    p.part_lse[(size_t)split * p.nq_pad + row] =
                        l_run[h] > 0.f ? m_run[h] + log2f(l_run[h]) : -INFINITY;
            }
        }
        return;
    }
    bf16* O = p.out + b0 * p.o_bs0 + b1 * p.o_bs1;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int row = row_lo + h * 8;
        if (row < p.nq) {
#pragma unroll
            for (int i = 0; i < HD / 8; ++i) {
                int d = i * 8 + (lane & 3) * 2;
                if (d < p.hd)
                    *reinterpret_cast<uint32_t*>(O + (size_t)row * p.o_stride + d) =
                        pack_bf16x2(o[i][2 * h] * inv[h], o[i][2 * h + 1] * inv[h]);
            }
        }
    }
}

// Merge flash-decoding partials: out[row] = sum_s w_s O_s / sum_s w_s, w_s = 2^(lse_s - max lse).
__global__ void __launch_bounds__(128) attention_combine_kernel(const float* __restrict__ part_o,
                                                                const float* __restrict__ part_lse,
                                                                bf16* __restrict__ out, int nq,
                                                                int nq_pad, int hd, int splits) {
    asm volatile("griddepcontrol.wait;" ::: "memory");      // no-op unless launched as a dependent
    const int row = blockIdx.x * 2 + (threadIdx.x >> 6);
    const int t = threadIdx.x & 63;
    if (row >= nq) return;
    float mx = -INFINITY;
    for (int s = 0; s < splits; ++s) mx = fmaxf(mx, part_lse[(size_t)s * nq_pad + row]);
    float wsum = 0.f;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < splits; ++s) {
        float l = part_lse[(size_t)s * nq_pad + row];
        float w = (l == -INFINITY) ? 0.f : exp2f(l - mx);
        wsum += w;
        if (w != 0.f && t * 4 < hd) {
            float4 v = *reinterpret_cast<const float4*>(part_o + ((size_t)s * nq_pad + row) * hd + t * 4);
            acc[0] += w * v.x; acc[1] += w * v.y; acc[2] += w * v.z; acc[3] += w * v.w;
        }
    }
    if (t * 4 < hd) {
        float inv = wsum > 0.f ? 1.0f / wsum : 0.f;
        uint2 pk = make_uint2(pack_bf16x2(acc[0] * inv, acc[1] * inv), pack_bf16x2(acc[2] * inv, acc[3] * inv));
        *reinterpret_cast<uint2*>(out + (size_t)row * hd + t * 4) = pk;
    }
}

template <int HD, int STAGES = 2>
inline int launch_attention(const AttnArgs& a, dim3 grid, cudaStream_t st) {
    constexpr int smem = (1 + 2 * STAGES) * 64 * (HD * 2 + 16);
    auto kern = attention_kernel<HD, STAGES>;
    static PerDeviceFlag configured;
    if (!configured.get()) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return FVLA_ERR_LAUNCH; }
        configured.set();
    }
    cudaError_t e = launch_pdl(kern, grid, dim3(128), smem, st, a);
    if (e != cudaSuccess) { set_error("attention_kernel: %s", cudaGetErrorString(e)); return FVLA_ERR_LAUNCH; }
    return check_launch("attention_kernel");
}


// ---------------------------------------------------------------------------------------------
// Decoder attention in one launch: a cluster of 4 to 11 CTAs has 32 flat query rows (4 tokens x 8 heads) and shares out
// the keys. Both products run on tcgen05 with the KEYS (then the head dimensions) as the 128-row operand and the query
// rows as N = 32:
//   S^T = K Q^T   one or two key tiles, accumulator lane = key, column = query row;
//   softmax       thread = one key x 16 rows; row maxima by a halving butterfly (16 shuffles for 16 rows), the
//                 32-key quadrants meet in shared memory; P goes to shared memory as the next operand;
//   O^T = V^T P^T two 128-dim tiles, accumulator lane = dim, column = query row.
// A thread's accumulator column then IS what an owner of 4 rows needs from it: normalised, it goes straight from registers to the
// owners' shared memory (st.async, 16 bytes = 4 rows of one dim), over the K tile, which nobody reads any more. Owners
// weight the parts by log-sum-exp in rank order and write bf16.
// One key tile (KT = 1): a CTA has a contiguous range of at most 128 keys, in two groups of 64 with a maximum, a sum and an accumulator
// of their own, merged before the exchange. Ranges, groups and the order of every sum are those of the warp-level kernel
// that this one replaced (two groups of warps, mma.sync), and mma.sync and tcgen05.mma add up the same bits, so the results are the
// same bits too: P is rounded to bf16 against its group's maximum, and ten Euler steps multiply any other rounding.
// Two key tiles (KT = 2), where that keeps more clusters resident: equal parts of the prefix and of the step's own keys, four groups.
// (With one maximum per CTA instead of per group fewer probabilities are exactly 1: 2.176e-3 from the 64-bit result at 65 tokens x 882
// unit-variance keys, 2.087e-3 with groups of 64, 2.080e-3 on 8 CTAs with one tile each.)
// Measured at 51 rows x 819 keys inside the decoder's chain: 6.1 us per launch, against 7.8 us for the warp-level form
// (mma.sync on 8 warps, halves staged in shared memory, bulk copies). What bounds it is a chain of
// latencies: dependency wait 0.9, Q 0.7, S^T 0.6, softmax and O^T 1.5, exchange 1.1 (28 KB per CTA; distributed shared memory
// moves 16 B/clk per SM when all SMs send), combine 0.5; DRAM and the tensor pipes idle.
// ---------------------------------------------------------------------------------------------
struct DecAttnArgs {
    const bf16* q; const bf16* k; const bf16* v; bf16* out;
    int nq, nk;
    // a batch of independent episodes (grid.z): element offsets between consecutive episodes' Q / out rows
    // and between their K / V caches; nq and nk are per episode
    long long q_episode_stride, kv_episode_stride;
    int episodes;
    float scale_log2;
    int mask_rows, mask_key_le;
    int prefix_keys;            // keys [0, prefix_keys) were not written by the preceding kernel
    // plan
    int splits;                 // cluster size
    int kp, nd;                 // KT = 1: keys per CTA, 0; KT = 2: prefix keys and own keys per CTA
    int pad;                    // rows of a CTA's K / V tile: kp + nd rounded up to 16
    int k_region;               // bytes of the K tile, or of the receive area that takes its place if that is larger
    int* status;
    FVLA_DBG_MEMBER
};

namespace decattn {
constexpr int HD = 256, BQ = 32, UNIT = 4, MIN_SPL = 4, MAX_SPL = 11, THREADS = 256;
// TMEM columns: O^T at 64 group + 32 (tile of 128 dims), behind them S^T at 64 tile + 32 (half of the dims)
constexpr int MAX_PAD = 208;                        // K + V tiles of 208 rows, Q / P and the rest just fit the SM
constexpr int QP_BYTES = 16384;                     // Q: 4 blocks of 64 dims x 32 rows; later P: up to 4 blocks of 64 keys x 32 rows
constexpr int UNIT_BYTES = HD * UNIT * 4;           // what one CTA sends for four rows
constexpr int OFF_PART = 64;                        // behind the barriers: row maxima and sums of one key tile
constexpr int OFF_STATS = OFF_PART + 1024;          // received log-sum-exps: [src][slot 2][row 4]
constexpr int MISC_BYTES = OFF_STATS + MAX_SPL * 32;
// KT = 1 only, behind the rest: per warp the weights of the two groups and 1 / sum, 32 rows each; fp32 probabilities, [row][key]
constexpr int FAC_BYTES = 8 * 384, E_PITCH = 136, E_BYTES = BQ * E_PITCH * 4;
__host__ __device__ constexpr int units_per_owner(int spl) { return (BQ / UNIT + spl - 1) / spl; }
inline int k_region_bytes(int spl, int pad) {
    const int recv = spl * units_per_owner(spl) * UNIT_BYTES;
    return pad * 512 > recv ? pad * 512 : recv;
}
inline int smem_bytes(int spl, int pad) { return 1024 + k_region_bytes(spl, pad) + pad * 512 + QP_BYTES + MISC_BYTES + (pad <= 128 ? FAC_BYTES + E_BYTES : 0); }

__host__ __device__ constexpr int block_threads(int kt) { return THREADS + 64 * kt; }      // and the warps that issue the MMAs
template <int KT> __device__ __forceinline__ void all_sync() { asm volatile("bar.sync 2, %0;" ::"n"(block_threads(KT)) : "memory"); }
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) { return tc5::mbar_wait(bar, parity, abort_flag); }
__device__ __forceinline__ uint32_t idesc(bool a_mn) { return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn ? 1u << 15 : 0u) | ((uint32_t)(BQ >> 3) << 17) | (8u << 24); }

// Reduce 16 values per lane over the 32 lanes of a warp: each step sends away the half of the values that the lane will not
// keep, so 16 rows take 16 shuffles. Afterwards lanes 2 k and 2 k + 1 hold row k.
template <typename Op>
__device__ __forceinline__ float butterfly16(float (&v)[16], int lane, Op op) {
#pragma unroll
    for (int half = 8; half >= 1; half >>= 1) {
        const bool up = lane & (2 * half);
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, 2 * half));
        }
    }
    return op(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1));
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float2 lds2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float lds1(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts1(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts4u(uint32_t a, const uint4& v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void sts_bf16(uint32_t a, float v) {
    asm volatile("st.shared.b16 [%0], %1;" ::"r"(a), "h"(__bfloat16_as_ushort(__float2bfloat16_rn(v))) : "memory");
}
}  // namespace decattn

__device__ __forceinline__ uint32_t dsm_map(uint32_t local_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
    return r;
}

template <int KT, int SPL>                                // key tiles of 128 per CTA, cluster size
__global__ void __launch_bounds__(decattn::block_threads(KT), 1)
decoder_attention_cluster_kernel(const __grid_constant__ DecAttnArgs p, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV) {
    using namespace decattn;
    constexpr int S_ISSUERS = 2 * KT, GROUPS = 2 * KT, S_COL = 64 * GROUPS, TMEM_COLS = 256 * KT;
    constexpr int RECV = SPL * units_per_owner(SPL) * UNIT_BYTES;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const uint32_t sK = (smem_u32(smem_raw) + 1023u) & ~1023u, sV = sK + p.k_region, sQ = sV + p.pad * 512, misc = sQ + QP_BYTES;
    uint8_t* gmisc = smem_raw + (misc - smem_u32(smem_raw));
    const uint32_t pre_bar = misc, in_bar = misc + 8, s_bar = misc + 16, o_bar = misc + 24;
    const uint32_t stats_in = misc + OFF_STATS, esum = misc + MISC_BYTES + FAC_BYTES;
    // Row maxima, then sums: [tile][row half][quadrant][16 rows] (sums of one tile: [group][row]); weights and 1 / sum per warp. Two tiles
    // leave no room for them; they lie in the K tile then, behind what the peers send, once the MMAs have read it.
    const uint32_t maxima = KT == 1 ? misc + OFF_PART : sK + RECV, sums = maxima + KT * 512;
    const uint32_t fac = (KT == 1 ? misc + MISC_BYTES : sums + KT * 512) + (threadIdx.x >> 5) * (GROUPS + 1) * BQ * 4;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gmisc + 32);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gmisc + 36);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    FVLA_DBG_CTA(p, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
    FVLA_STAMP(0);
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int q0 = blockIdx.x * BQ, rows_here = min(BQ, p.nq - q0), units = (rows_here + UNIT - 1) / UNIT;
    const float scale = p.scale_log2;
    const int pre_rows = min(p.prefix_keys, p.nk);
    const int key0 = (int)rank * p.kp, prefix_here = max(0, min(p.kp, pre_rows - key0));        // local keys [0, prefix_here): prefix
    const int new0 = KT == 1 ? max(0, key0 - pre_rows) : (int)rank * p.nd;                      // then new_here of the step's own
    const int new_here = max(0, min(KT == 1 ? p.kp - prefix_here : p.nd, p.nk - pre_rows - new0));
    const int owned = (int)rank < units ? 1 + ((int)rank + SPL < units ? 1 : 0) : 0;            // units rank, rank + SPL

    auto request_prefix = [&]() {
#pragma unroll
        for (int cb = 0; cb < HD / 64; ++cb) tc5::tma_load_3d(sK + cb * p.pad * 128, &tmK, pre_bar, cb * 64, key0, blockIdx.z);
#pragma unroll
        for (int cb = 0; cb < HD / 64; ++cb) tc5::tma_load_3d(sV + cb * p.pad * 128, &tmV, pre_bar, cb * 64, key0, blockIdx.z);
    };
    if (tid == 0) {
        tc5::mbar_init(pre_bar, 1);
        tc5::mbar_init(in_bar, 1);
        tc5::mbar_init(s_bar, S_ISSUERS);
        tc5::mbar_init(o_bar, 2);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (owned > 0) tc5::mbar_expect_tx(in_bar, (uint32_t)(owned * SPL) * (UNIT_BYTES + UNIT * 4));
        // The prefix rows of K and V arrive as one box of 64 dims x pad rows per block, through maps that END at the prefix:
        // the rows behind it, which the preceding kernel may still be writing, are not touched in memory and read as
        // zero. A batch, whose prefix rows the
        // preceding kernel may have written, only has them brought to L2 here and asks for them behind the dependency wait. (Rows past prefix_here hold the next CTA's keys; the own keys overwrite some, the rest is masked.)
        tc5::mbar_expect_tx(pre_bar, 2u * p.pad * 512u);
        if (p.episodes <= 1) request_prefix();
        else {
#pragma unroll
            for (int cb = 0; cb < HD / 64; ++cb) { tc5::tma_prefetch_3d(&tmK, cb * 64, key0, blockIdx.z); tc5::tma_prefetch_3d(&tmV, cb * 64, key0, blockIdx.z); }
        }
    }
    if (warp == 1) {
        tc5::tmem_alloc(misc + 32, TMEM_COLS);
        tc5::tmem_relinquish();
    }
    tc5::tc_fence_before();
    __syncthreads();
    tc5::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0 && p.episodes > 1) request_prefix();
    FVLA_STAMP(1);
    // What the preceding kernel wrote, Q and the own keys, comes through registers: plain 16-byte loads reach them sooner than
    // any bulk copy reaches shared memory. Both land in the swizzled operand layout (piece c of row r at c ^ (r & 7)).
    {
        const bf16* gq = p.q + (size_t)blockIdx.z * p.q_episode_stride + (size_t)q0 * HD;
        const size_t kv0 = (size_t)blockIdx.z * p.kv_episode_stride + (size_t)(pre_rows + new0) * HD;
        constexpr int QV = BQ * 32 / THREADS;
        uint4 qv[QV];
#pragma unroll
        for (int i = 0; i < QV; ++i) {
            const int idx = tid + i * THREADS;
            qv[i] = tid < THREADS && idx < rows_here * 32 ? *reinterpret_cast<const uint4*>(gq + (size_t)idx * 8) : make_uint4(0, 0, 0, 0);
        }
        constexpr int OWN = KT == 1 ? 8 : 4;                 // own keys, 8 rows per piece index; with KT = 1 one or two CTAs have them all
        uint4 kv[OWN], vv[OWN];
        const int total = new_here * 32;
        auto fetch_own = [&](int base) {
#pragma unroll
            for (int i = 0; i < OWN; ++i) {
                const int idx = base + tid + i * THREADS;
                if (tid < THREADS && idx < total) {
                    kv[i] = *reinterpret_cast<const uint4*>(p.k + kv0 + (size_t)idx * 8);
                    vv[i] = *reinterpret_cast<const uint4*>(p.v + kv0 + (size_t)idx * 8);
                }
            }
        };
        fetch_own(0);
#pragma unroll
        for (int i = 0; i < QV; ++i) {
            const int idx = tid + i * THREADS, r = idx >> 5, c = idx & 31;
            if (tid < THREADS) sts4u(sQ + (c >> 3) * (BQ * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4), qv[i]);
        }
        wait(pre_bar, 0, abort_flag);                        // the own rows go over what the boxes brought in
        for (int base = 0; base < total; base += OWN * THREADS) {
            if (base > 0) fetch_own(base);
#pragma unroll
            for (int i = 0; i < OWN; ++i) {
                const int idx = base + tid + i * THREADS, r = prefix_here + (idx >> 5), c = idx & 31;
                const uint32_t at = (c >> 3) * p.pad * 128 + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                if (tid < THREADS && idx < total) { sts4u(sK + at, kv[i]); sts4u(sV + at, vv[i]); }
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    FVLA_STAMP(2);
    // Issuing threads, in warps of their own behind the others: for S^T one per key tile and half of the head dimension (accumulators
    // added below), for O^T one per 128 dims. A thread needs 46 clk per MMA and more for the first, the tensor pipe 39; while two of the
    // softmax warps issued, their rows' sums came 500 clk after the others'. Per layer-step 24.94 -> 24.81 us at 51 rows, 22.94 -> 22.65 at 32,
    // 30.9 -> 30.5 at 65.
    const int issuer = __shfl_sync(0xffffffffu, warp, 0) - THREADS / 32;
    if (issuer >= 0) {
      if (tc5::elect_one()) {
        tc5::tc_fence_after();
        const int t = issuer >> 1, h = issuer & 1;
        const uint64_t a0 = tc5::smem_desc(sK + t * 128 * 128 + h * p.pad * 256, 16, 1024), b0 = tc5::smem_desc(sQ + h * (BQ * 256), 16, 1024);
#pragma unroll
        for (int cb = 0; cb < 2; ++cb)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                tc5::umma_bf16(tmem + S_COL + issuer * 32, a0 + cb * (p.pad * 8) + k * 2, b0 + cb * (BQ * 8) + k * 2, idesc(false), (cb | k) ? 1u : 0u);
        tc5::umma_commit(s_bar);
      }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
      all_sync<KT>();                                        // P is in place
      const uint64_t vd = tc5::smem_desc(sV + issuer * 2 * p.pad * 128, p.pad * 128, 1024), pd = tc5::smem_desc(sQ, 16, 1024);
      if (issuer < 2 && tc5::elect_one()) {
        tc5::tc_fence_after();
#pragma unroll
        for (int k = 0; k < (KT == 1 ? 8 : MAX_PAD / 16); ++k)
            if (k * 16 < p.pad)
                tc5::umma_bf16(tmem + (k >> 2) * 64 + issuer * 32, vd + k * 128, pd + (k >> 2) * (BQ * 8) + (k & 3) * 2, idesc(true),
                               k & 3 ? 1u : 0u);
        tc5::umma_commit(o_bar);
      }
      __syncwarp();
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
      all_sync<KT>();                                        // accumulators read
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      return;
    }
    wait(s_bar, 0, abort_flag);
    __syncwarp();
    tc5::tc_fence_after();
    // This CTA's MMAs have read its K tile: the peers may send into it (the matching wait stands before the first send). Relaxed:
    // no data is handed over, and a releasing arrive waits 0.4 us for the thread's earlier accesses.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    FVLA_STAMP(3);
    const int quad = warp & 3, half = warp >> 2;             // keys 32 quad .. + 31 of a tile, rows 16 half .. + 15
    {
        float v[KT][16], red[16];
#pragma unroll
        for (int t = 0; t < KT; ++t) {
            const uint32_t at = tmem + S_COL + t * 64 + half * 16 + ((uint32_t)(quad * 32) << 16);
            tc5::tmem_ld16(at, v[t]);
            tc5::tmem_ld16(at + 32, red);
            const int key = t * 128 + quad * 32 + lane;
            const bool see = key < prefix_here + new_here;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[t][i] = see ? (v[t][i] + red[i]) * scale : -INFINITY;
            // the state token's rows (the first of the sequence) see keys up to mask_key_le only
            if (q0 + half * 16 < p.mask_rows && key >= prefix_here && pre_rows + new0 + key - prefix_here > p.mask_key_le) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (q0 + half * 16 + i < p.mask_rows) v[t][i] = -INFINITY;
            }
        }
#pragma unroll
        for (int t = 0; t < KT; ++t) {
#pragma unroll
            for (int i = 0; i < 16; ++i) red[i] = v[t][i];
            const float m = butterfly16(red, lane, [](float a, float b) { return fmaxf(a, b); });
            if ((lane & 1) == 0) sts1(maxima + (((t * 2 + half) * 4 + quad) * 16 + (lane >> 1)) * 4, m);
        }
        compute_sync();
#pragma unroll
        for (int t = 0; t < KT; ++t) {
            const int key = t * 128 + quad * 32 + lane;
            // P over Q, whose readers are done; rows of a 64-key block are 128 bytes, 16-byte piece c of row r at c ^ (r & 7)
            const uint32_t at = maxima + ((t * 2 + half) * 64 + (quad >> 1) * 32) * 4;      // of the key's group, 0 where a row sees none of its keys
            const uint32_t dst = sQ + (key >> 6) * (BQ * 128) + half * 16 * 128 + (key & 7) * 2, c = ((key & 63) >> 3) << 4;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 a = lds4(at + i * 4), b = lds4(at + i * 4 + 64);
                const float mx[4] = {fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w)};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float e = exp2f(v[t][i + r] - (mx[r] == -INFINITY ? 0.f : mx[r]));
                    if (KT == 1) sts1(esum + ((half * 16 + i + r) * E_PITCH + key) * 4, e);
                    v[t][i + r] = e;
                }
            }
            if (key < p.pad) {
#pragma unroll
                for (int i = 0; i < 16; ++i) sts_bf16(dst + (c ^ ((i & 7) << 4)) + i * 128, v[t][i]);
            }
        }
        tc5::tc_fence_before();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        all_sync<KT>();                                      // the issuing warps go on with O^T
        if (KT == 1) {
            // Sum of a row over a group of 64 keys, four threads: each takes a pair of keys out of every eight, front to back.
            const int row = (warp >> 1) * 8 + (lane >> 2), group = warp & 1;
            const uint32_t at = esum + (row * E_PITCH + group * 64 + (lane & 3) * 2) * 4;
            float2 e[8];
#pragma unroll
            for (int n = 0; n < 8; ++n) e[n] = lds2(at + n * 32);
            float l = 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n) { l += e[n].x; l += e[n].y; }
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            if ((lane & 3) == 0) sts1(sums + (group * BQ + row) * 4, l);
        } else {
#pragma unroll
            for (int t = 0; t < KT; ++t) {
                const float l = butterfly16(v[t], lane, [](float a, float b) { return a + b; });
                if ((lane & 1) == 0) sts1(sums + (((t * 2 + half) * 4 + quad) * 16 + (lane >> 1)) * 4, l);
            }
        }
    }
    compute_sync();                                          // sums and maxima of all rows are in place
    // Every warp works out what its accumulator columns are multiplied with, lane = row: [group][row], then 1 / sum
    float f[2][BQ], fi[BQ], lse;                              // (the first two groups' in registers before the accumulators are there)
    auto factors = [&](int g, float (&out)[BQ]) {
#pragma unroll
        for (int i = 0; i < BQ; i += 4) {
            const float4 a = lds4(fac + (g * BQ + i) * 4);
            out[i] = a.x; out[i + 1] = a.y; out[i + 2] = a.z; out[i + 3] = a.w;
        }
    };
    {
        const int row = lane >> 4, i = lane & 15;
        float m[GROUPS], mn = -INFINITY, l = 0.f;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const uint32_t at = maxima + (((g >> 1) * 2 + row) * 64 + (g & 1) * 32 + i) * 4;
            m[g] = fmaxf(lds1(at), lds1(at + 64));
            mn = fmaxf(mn, m[g]);
        }
        const float mu = mn == -INFINITY ? 0.f : mn;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
            const uint32_t at = sums + (((g >> 1) * 2 + row) * 64 + (g & 1) * 32 + i) * 4;
            const float a = exp2f(m[g] - mu), lg = KT == 1 ? lds1(sums + (g * BQ + lane) * 4) : lds1(at) + lds1(at + 64);      // exp2(-inf) = 0
            l = g == 0 ? __fmul_rn(lg, a) : __fmaf_rn(lg, a, l);
            sts1(fac + (g * BQ + lane) * 4, a);
        }
        sts1(fac + (GROUPS * BQ + lane) * 4, l > 0.f ? 1.0f / l : 0.f);
        lse = l > 0.f ? mn + log2f(l) : -INFINITY;
        __syncwarp();
        factors(0, f[0]);
        factors(1, f[1]);
        factors(GROUPS, fi);
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 0 && lane < units * UNIT) {                  // row lane's log-sum-exp to its owner
        const int u = lane >> 2, owner = u % SPL, slot = u / SPL;
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];"
                     ::"r"(dsm_map(stats_in + rank * 32 + slot * 16 + (lane & 3) * 4, owner)), "f"(lse), "r"(dsm_map(in_bar, owner)) : "memory");
    }
    wait(o_bar, 0, abort_flag);
    __syncwarp();
    tc5::tc_fence_after();
    FVLA_STAMP(4);
    {
        float o[32];
        tc5::tmem_ld32(tmem + half * 32 + ((uint32_t)(quad * 32) << 16), o);                   // dim 128 half + 32 quad + lane
#pragma unroll
        for (int i = 0; i < BQ; ++i) o[i] = __fmul_rn(o[i], f[0][i]);      // (the rounding of each step is part of the result: no other contraction)
#pragma unroll
        for (int g = 1; g < GROUPS; ++g) {
            if (g * 64 >= p.pad) break;                      // a group without keys has no accumulator
            float og[32];
            tc5::tmem_ld32(tmem + g * 64 + half * 32 + ((uint32_t)(quad * 32) << 16), og);
            if (g > 1) factors(g, f[1]);
#pragma unroll
            for (int i = 0; i < BQ; ++i) o[i] = __fmaf_rn(og[i], f[1][i], o[i]);
        }
#pragma unroll
        for (int i = 0; i < BQ; ++i) o[i] *= fi[i];
        const uint32_t at = sK + rank * UNIT_BYTES + (half * 128 + quad * 32 + lane) * 16;
#pragma unroll
        for (int u = 0; u < BQ / UNIT; ++u) {
            if (u >= units) break;
            const int owner = u % SPL, slot = u / SPL;
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                         ::"r"(dsm_map(at + slot * SPL * UNIT_BYTES, owner)), "f"(o[4 * u]), "f"(o[4 * u + 1]), "f"(o[4 * u + 2]), "f"(o[4 * u + 3]),
                           "r"(dsm_map(in_bar, owner)) : "memory");
        }
    }
    tc5::tc_fence_before();
    if (owned > 0) wait(in_bar, 0, abort_flag);
    __syncwarp();
    FVLA_STAMP(5);
    // Nobody may leave while a peer can still send to it: after this arrive nothing is outstanding towards this CTA, so
    // the wait at the end costs nothing unless a peer is late.
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    for (int slot = 0; slot < owned; ++slot) {
        const int row0 = q0 + ((int)rank + slot * SPL) * UNIT;
        // log-sum-exp weights: lane = (source, row), a second one for sources 8 and up
        const int s0 = lane >> 2;
        const uint32_t st = stats_in + s0 * 32 + slot * 16 + (lane & 3) * 4;
        const bool have0 = SPL >= 8 || s0 < SPL, have1 = SPL > 8 && s0 + 8 < SPL;
        const float l0 = have0 ? lds1(st) : -INFINITY, l1 = have1 ? lds1(st + 256) : -INFINITY;
        float mx = fmaxf(l0, l1);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float w0 = l0 == -INFINITY ? 0.f : exp2f(l0 - mx), w1 = l1 == -INFINITY ? 0.f : exp2f(l1 - mx);
        float acc[UNIT] = {0.f, 0.f, 0.f, 0.f}, wsum[UNIT] = {0.f, 0.f, 0.f, 0.f};
        const uint32_t src = sK + slot * SPL * UNIT_BYTES + tid * 16;
        float4 in[SPL];                                       // all sources requested before the first is used
#pragma unroll
        for (int s = 0; s < SPL; ++s) in[s] = lds4(src + s * UNIT_BYTES);
#pragma unroll
        for (int s = 0; s < SPL; ++s) {
            const float a[UNIT] = {in[s].x, in[s].y, in[s].z, in[s].w};
#pragma unroll
            for (int r = 0; r < UNIT; ++r) {
                const float w = __shfl_sync(0xffffffffu, s < 8 ? w0 : w1, (s & 7) * 4 + r);
                wsum[r] += w;
                acc[r] = __fmaf_rn(w, a[r], acc[r]);
            }
        }
        const float ws = lane & 2 ? (lane & 1 ? wsum[3] : wsum[2]) : (lane & 1 ? wsum[1] : wsum[0]);
        const float inv = ws > 0.f ? 1.0f / ws : 0.f;
#pragma unroll
        for (int r = 0; r < UNIT; ++r) acc[r] *= __shfl_sync(0xffffffffu, inv, r);
        // two adjacent dims of two rows per lane, so that a store is a bf16 pair: even lanes rows 0 and 1, odd lanes 2 and 3
        const bool odd = lane & 1;
        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? acc[0] : acc[2], 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? acc[1] : acc[3], 1);
        const uint32_t v0 = odd ? pack_bf16x2(r0, acc[2]) : pack_bf16x2(acc[0], r0), v1 = odd ? pack_bf16x2(r1, acc[3]) : pack_bf16x2(acc[1], r1);
        const int row = row0 + (odd ? 2 : 0);
        bf16* out = p.out + (size_t)blockIdx.z * p.q_episode_stride + (size_t)row * HD + (tid & ~1);
        if (row < p.nq) *reinterpret_cast<uint32_t*>(out) = v0;
        if (row + 1 < p.nq) *reinterpret_cast<uint32_t*>(out + HD) = v1;
    }
    FVLA_STAMP(6);
    all_sync<KT>();
    if (warp == 1) {
        tc5::tc_fence_after();
        tc5::tmem_dealloc(tmem, TMEM_COLS);
    }
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    FVLA_STAMP(7);
    if (tid == 0 && *abort_flag && p.status) atomicExch(p.status, 3);
}

using DecAttnKernel = void (*)(const DecAttnArgs, const CUtensorMap, const CUtensorMap);
template <int KT>
inline DecAttnKernel decoder_attention_kernel(int spl) {
    static const DecAttnKernel table[] = {decoder_attention_cluster_kernel<KT, 4>, decoder_attention_cluster_kernel<KT, 5>, decoder_attention_cluster_kernel<KT, 6>,
                                          decoder_attention_cluster_kernel<KT, 7>, decoder_attention_cluster_kernel<KT, 8>, decoder_attention_cluster_kernel<KT, 9>,
                                          decoder_attention_cluster_kernel<KT, 10>, decoder_attention_cluster_kernel<KT, 11>};
    return table[spl - decattn::MIN_SPL];
}
inline bool configure_decoder_attention() {
    static PerDeviceFlag configured;
    if (configured.get()) return true;
    for (int i = 0; i < 2 * (decattn::MAX_SPL - decattn::MIN_SPL + 1); ++i) {
        const int spl = decattn::MIN_SPL + i / 2;
        const DecAttnKernel kern = i & 1 ? decoder_attention_kernel<2>(spl) : decoder_attention_kernel<1>(spl);
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);      // clusters of 9..11
        if (e != cudaSuccess) { set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e)); return false; }
    }
    configured.set();
    return true;
}

// Clusters of `spl` CTAs that the device holds at once with one CTA per SM (B200: 33 of 4, 26 of 5, 22 of 6, 15 of 7 to 9, 11 of
// 10, 7 of 11: SMs of a GPC that do not fill a cluster stay idle). Asked once per device and size.
inline int resident_attention_clusters(int spl) {
    static std::atomic<int> cached[kMaxDevices][decattn::MAX_SPL + 1];
    std::atomic<int>& c = cached[current_device()][spl];
    int n = c.load(std::memory_order_acquire);
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, spl); cfg.blockDim = dim3(decattn::block_threads(1)); cfg.dynamicSmemBytes = 168 * 1024;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = spl; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, decoder_attention_kernel<1>(spl), &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = 1; }
        c.store(n, std::memory_order_release);
    }
    return n;
}

// How the keys are shared out. One sequence of up to 64 tokens and 1 408 keys: ranges of 8 clusters' CTAs up to 1 024 keys and one
// CTA more per further 128, whatever is resident, so that the results of such a decode depend on nothing but its shape (and are the
// bits of the kernel before, see above). Else the cluster size, smallest first in every order of preference: all clusters of the
// launch resident together, with one key tile of at most 128 rows and 4 or 8 CTAs, so that the eight owners' shares come out even; then
// any size with one key tile; then with two (65 tokens x 882 keys: 33.2 us per layer-step with 5 CTAs, all 17 clusters resident, 37.8
// with 8, of which 15 are). Failing that the smallest that fits the SM at all. Returns whether all clusters are resident; 0 splits: the
// shape does not fit.
inline bool plan_decoder_attention(DecAttnArgs& a) {
    using namespace decattn;
    a.splits = 0;
    if (a.prefix_keys <= 0 || !configure_decoder_attention()) return false;
    const int clusters = ((a.nq + BQ - 1) / BQ) * (a.episodes > 1 ? a.episodes : 1), pre = a.prefix_keys < a.nk ? a.prefix_keys : a.nk;
    auto take = [&](int spl) {                               // false: more rows than the SM holds
        const int range = ((a.nk + spl - 1) / spl + 7) / 8 * 8;
        a.kp = range <= 128 ? range : (pre + spl - 1) / spl;
        a.nd = range <= 128 ? 0 : (a.nk - pre + spl - 1) / spl;
        a.pad = (a.kp + a.nd + 15) / 16 * 16;
        a.k_region = k_region_bytes(spl, a.pad);
        return a.pad <= MAX_PAD && smem_bytes(spl, a.pad) <= 232448;
    };
    const int ranges = (a.nk + 127) / 128 < 8 ? 8 : (a.nk + 127) / 128;
    if (a.episodes <= 1 && a.nq <= 512 && ranges <= MAX_SPL && take(ranges)) {
        a.splits = ranges;
        return clusters <= resident_attention_clusters(ranges);
    }
    for (int pass = 0; pass < 4; ++pass)
        for (int spl = MIN_SPL; spl <= MAX_SPL; ++spl) {
            if (pass == 0 && spl != 4 && spl != 8) continue;
            if (!take(spl) || (pass < 2 && a.pad > 128)) continue;
            if (pass < 3 && clusters > resident_attention_clusters(spl)) continue;
            a.splits = spl;
            return pass < 3;
        }
    return false;
}

inline int launch_decoder_attention_cluster(const DecAttnArgs& a, bool pdl, cudaStream_t st) {
    // K / V maps that end at the prefix (rows the preceding kernel may still be writing are never fetched by them)
    CUtensorMap tmK, tmV;
    const int seqs = a.episodes > 1 ? a.episodes : 1;
    const int pre_rows = a.prefix_keys < a.nk ? a.prefix_keys : a.nk;
    if (a.splits <= 0 || pre_rows <= 0) { set_error("decoder attention: %d keys (%d of the prefix) do not fit", a.nk, pre_rows); return FVLA_ERR_UNSUPPORTED; }
    int rc = tc5::make_map3d(&tmK, a.k, decattn::HD, (uint64_t)pre_rows, (uint64_t)seqs, decattn::HD, (uint64_t)a.kv_episode_stride, 64, (uint32_t)a.pad);
    if (rc) return rc;
    rc = tc5::make_map3d(&tmV, a.v, decattn::HD, (uint64_t)pre_rows, (uint64_t)seqs, decattn::HD, (uint64_t)a.kv_episode_stride, 64, (uint32_t)a.pad);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.nq + decattn::BQ - 1) / decattn::BQ, a.splits, seqs);
    cfg.blockDim = dim3(decattn::block_threads(a.pad > 128 ? 2 : 1), 1, 1);
    cfg.dynamicSmemBytes = decattn::smem_bytes(a.splits, a.pad);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = a.splits; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, a.pad > 128 ? decoder_attention_kernel<2>(a.splits) : decoder_attention_kernel<1>(a.splits), a, tmK, tmV);
    if (e != cudaSuccess) { set_error("decoder_attention_cluster_kernel: %s", cudaGetErrorString(e)); return FVLA_ERR_LAUNCH; }
    return check_launch("decoder_attention_cluster_kernel");
}

}  // namespace fvla
