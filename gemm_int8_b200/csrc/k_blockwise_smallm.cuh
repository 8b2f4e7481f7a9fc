// Blockwise-dequantised W8A8 GEMM for few tokens (M <= 16): the same chain as k_blockwise.cuh,
//   out[m,n] = bf16( sum_kb fp32(P[m,n,kb]) * (sa[m,kb] * sw[n/128,kb]) ),  kb ascending, one fused multiply-add per block,
// with the operands swapped as in k_smallm.cuh: 64 weight rows lie on the lanes of tensor memory and the tokens are its sixteen
// columns, so that a K block of 128 costs sixteen columns of promotion instead of a 128-row tile's worth.  Bound: HBM where
// the weights have many rows (16 x 8192 x 8192: 190 ns per K block and CTA, 5.5 TB/s over all), the serial path of a K block where
// they have few (16 x 4096 x 14336, 64 CTAs: 145 ns).
//
// Why 64 weight rows: 8192 columns make 128 tiles, one per SM, without a K split (the chain runs in the order of the K blocks, so
// partial sums cannot be added up; sending the exact partials to one CTA of a cluster, which runs the chain, was slower at every
// count of splits: 16 x 4096 x 4096 11.2 -> 13.6 us with two), and a tile lies inside one weight-scale block, so that its scale is one
// number per K block.  The MMAs are M = 128 all the same; their upper 64 rows read whatever lies behind the tile in shared
// memory and land in lanes 64..127, which nobody reads.
//
// Roles: a warp's lane quarter is warp % 4, so promotion warps are those with warp % 4 < 2 (8 columns each); warp 2 loads; warp 3,
// which allocates tensor memory, and warp 7 issue the MMAs of alternate stages (an MMA of any size takes some 60 cycles to
// issue).  A stage holds two K blocks and has its own 32 columns of tensor memory:
//   bar_full[s]   the TMA bytes of stage s.         Waiter: the stage's issuer; refilled only after bar_done[s].
//   bar_done[s]   the issuer's commit.              Waiters: the producer, whose refill the next completion needs, and the promotion
//                                                   warps, whose arrivals on bar_read[s] the next completion needs.
//   bar_read[s]   the promotion warps have loaded the partials.  Waiter: the stage's issuer, whose MMAs the next completion needs.
// Every wait is gated by its waiter's own next action, so parities cannot be missed; STAGES is even, so that a stage has one issuer.
//
// Measured, back to back, weights beyond L2, 64-wide tiles of k_blockwise.cuh -> this kernel (with the stages that the host takes), us:
// 16 x 8192 x 8192 18.8 -> 15.9 (six), 16 x 4096 x 4096 13.9 -> 8.3, 16 x 14336 x 4096 20.9 -> 13.7, 16 x 4096 x 14336 28.1 -> 21.3, 8 x 57344 x
// 8192 108 -> 82, 1 x 1024 x 4096 10.2 -> 7.6 (four), and from K = 16 on (16 x 57344 x 128 11.6 -> 10.2, 16 x 4096 x 16 5.9 -> 5.7).  On the way: sixteen columns a warp and scale products fetched from shared memory between the multiply-adds 17.5 at 16 x 8192 x 8192, the next
// stage's load not under this one's arithmetic 19.3.  With 32 tokens the same form is no better than the tiles (32 x 8192 x 8192 19.7 ->
// 20.4, 32 x 28672 x 4096 25.6 -> 41.0, 20 x 14336 x 4096 22.0 -> 22.3), so those keep them.
#pragma once

#include "k_blockwise.cuh"

namespace gi8 {

constexpr int kBwSmallTileN = 64;  // weight rows per CTA
constexpr int kBwSmallTokens = 16; // tokens per CTA

struct BlockwiseSmallMParams {
    uint16_t* out;        // bf16 [M, N], leading dimension ldo
    const float* sa;      // [M, KB], row stride ld_sa
    const float* sw;      // [ceil(N/128), KB], row stride ld_sw
    const uint16_t* bias; // bf16 [N] added to the rounded result, or null
    uint32_t* status;
    int64_t ldo, ld_sa, ld_sw;
    int M, N, K;
    int after_quant;      // launched as the programmatic dependent of the quantiser that writes x and sa (and of nothing else)
};

template <int STAGES_>
struct BlockwiseSmallM {
    static constexpr int MT = kBwSmallTokens;
    static constexpr int STAGES = STAGES_;
    static constexpr int GROUPS = MT / 8;                         // groups of eight columns: pairs of promotion warps
    static constexpr int THREADS = GROUPS * 128;
    static constexpr uint32_t BYTES_W = kBwSmallTileN * kBK;      // one K block of weights
    static constexpr uint32_t BYTES_X = MT * kBK;
    static constexpr uint32_t STAGE = 2 * (BYTES_W + BYTES_X);
    static constexpr uint32_t TMEM_COLS = 2 * STAGES * MT <= 128 ? 128 : 256;  // (two CTAs share an SM's)
    static_assert(2 * STAGES * MT <= 256 && STAGES % 2 == 0, "tensor memory; one issuer per stage");
    // (behind the stages: what the upper half of the last weight tile's MMAs reads)
    static constexpr uint32_t SMEM = STAGES * STAGE + BYTES_W + 1024;
};

template <int STAGES_>
__global__ void __launch_bounds__(BlockwiseSmallM<STAGES_>::THREADS)
blockwise_smallm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const BlockwiseSmallMParams p)
{
    using S = BlockwiseSmallM<STAGES_>;
    constexpr int STAGES = S::STAGES, MT = S::MT;
    constexpr uint32_t kIdesc = make_idesc_i8(128, MT, false);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

    __shared__ __align__(8) uint64_t bar_full[STAGES];
    __shared__ __align__(8) uint64_t bar_done[STAGES];
    __shared__ __align__(8) uint64_t bar_read[STAGES];
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile uint32_t abort_flag;
    __shared__ __align__(16) float t_s[S::GROUPS * 2][2][16];  // per promotion warp: scale products of a stage, two in turn

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int tile = blockIdx.x;
    const int num_kb = (p.K + kBK - 1) / kBK;
    const int num_st = (num_kb + 1) / 2;

    if (warp == 2) {
        if (elect_one()) {
            abort_flag = 0;
            for (int s = 0; s < STAGES; ++s) {
                mbar_init(&bar_full[s], 1);
                mbar_init(&bar_done[s], 1);
                mbar_init(&bar_read[s], S::GROUPS * 2);
            }
            fence_barrier_init();
            fence_proxy_async_smem();
            prefetch_tensormap(&map_w);
            prefetch_tensormap(&map_x);
        }
        __syncwarp();
    }
    if (warp == 3) {
        tmem_alloc(&tmem_base_slot, S::TMEM_COLS);
        tmem_relinquish_alloc_permit();
    }
    tcgen05_fence_before_sync();
    __syncthreads();
    tcgen05_fence_after_sync();
    const uint32_t tmem_base = tmem_base_slot;

    // Only the producer reads anything before the kernel in front has ended: the weights, behind a quantiser, which writes x and sa
    // and started this kernel after everything in front of it had ended.
    if (!(warp == 2 && p.after_quant)) pdl_wait();
    if (threadIdx.x == 96) pdl_launch_dependents();  // (a thread of warp 3, which has waited)

    if (warp == 2) {
        // ---------------------------------------------------------------------------------- TMA producer
        const uint64_t pol_w = l2_policy_evict_first();
        const uint64_t pol_x = l2_policy_evict_last();
        auto load_w = [&](int i, uint32_t s) {
            const int n = min(2, num_kb - 2 * i);
            mbar_arrive_expect_tx(&bar_full[s], n * (S::BYTES_W + S::BYTES_X));
            for (int j = 0; j < n; ++j)
                tma_load_2d_hint(smem + s * S::STAGE + j * S::BYTES_W, &map_w, &bar_full[s], (2 * i + j) * kBK, tile * kBwSmallTileN, pol_w);
        };
        auto load_x = [&](int i, uint32_t s) {
            const int n = min(2, num_kb - 2 * i);
            for (int j = 0; j < n; ++j)
                tma_load_2d_hint(smem + s * S::STAGE + 2 * S::BYTES_W + j * S::BYTES_X, &map_x, &bar_full[s], (2 * i + j) * kBK, 0, pol_x);
        };
        const int first = min(num_st, STAGES);
        if (elect_one())
            for (int i = 0; i < first; ++i) load_w(i, i);
        __syncwarp();
        if (p.after_quant) pdl_wait();
        if (elect_one())
            for (int i = 0; i < first; ++i) load_x(i, i);
        __syncwarp();
        int issued = first;
        for (uint32_t s = 0, ph = 0; issued < num_st; ++issued) {
            if (!warp_agrees(wait_or_abort(&bar_done[s], ph, &abort_flag), p.status, &abort_flag, ERR_TIMEOUT_PRODUCER)) break;
            if (elect_one()) {
                load_w(issued, s);
                load_x(issued, s);
            }
            __syncwarp();
            if (++s == STAGES) s = 0, ph ^= 1;
        }
        drain_stages<STAGES>(bar_full, bar_done, issued % STAGES, (issued / STAGES) & 1, min(issued, STAGES), p.status, &abort_flag);
    } else if (warp == 3 || warp == 7) {
        // ---------------------------------------------------------------------------------- MMA issuers
        // The MMAs of the two K blocks of a stage alternate: each accumulates onto the one before the last, not onto the last.
        const int me = warp == 3 ? 0 : 1;
        const uint32_t w_0 = smem_desc_lo(smem_u32(smem));
        uint32_t s = me, ph = 0;
        for (int i = me; i < num_st; i += 2) {
            const bool ready = wait_or_abort(&bar_full[s], ph, &abort_flag) && wait_or_abort(&bar_read[s], ph ^ 1, &abort_flag);
            if (!warp_agrees(ready, p.status, &abort_flag, ERR_TIMEOUT_MMA)) break;
            tcgen05_fence_after_sync();
            const bool two = 2 * i + 1 < num_kb;
            const uint32_t dw = w_0 + s * (S::STAGE / 16), dw1 = dw + S::BYTES_W / 16;
            const uint32_t dx = dw + 2 * S::BYTES_W / 16, dx1 = dx + S::BYTES_X / 16;
            const uint32_t d = tmem_base + s * (2 * MT);
            if (two) {
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < kBK / kUmmaK; ++k) {
                        umma_i8(d, smem_desc_k128_of(dw + 2 * k), smem_desc_k128_of(dx + 2 * k), kIdesc, k != 0);
                        umma_i8(d + MT, smem_desc_k128_of(dw1 + 2 * k), smem_desc_k128_of(dx1 + 2 * k), kIdesc, k != 0);
                    }
                    umma_commit(&bar_done[s]);
                }
            } else if (elect_one()) {
#pragma unroll
                for (int k = 0; k < kBK / kUmmaK; ++k) umma_i8(d, smem_desc_k128_of(dw + 2 * k), smem_desc_k128_of(dx + 2 * k), kIdesc, k != 0);
                umma_commit(&bar_done[s]);
            }
            __syncwarp();
            s += 2;
            if (s >= STAGES) s -= STAGES, ph ^= 1;
        }
    } else if ((warp & 3) < 2) {
        // ---------------------------------------------------------------------------------- promotion warps
        const int quarter = warp & 3;
        const int cg = warp >> 2;                    // tokens 8 cg .. 8 cg + 7
        const int n = tile * kBwSmallTileN + quarter * 32 + lane;
        const uint32_t tm_warp = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + cg * 8;
        // Scale products of a stage: lane l forms that of token 8 cg + l % 8 and K block l / 8 of the stage (the upper half-warp the
        // same once more); shared memory turns them into broadcast operands.  The loads run three stages ahead of their use.
        const float* sw_row = p.sw + static_cast<int64_t>(tile * kBwSmallTileN / 128) * p.ld_sw;
        const float* sa_row = p.sa + static_cast<int64_t>(min(cg * 8 + (lane & 7), p.M - 1)) * p.ld_sa;
        auto scale_kb = [&](int i) { return min(2 * i + ((lane >> 3) & 1), num_kb - 1); };
        float* const my_t = t_s[cg * 2 + quarter][0];
        const uint32_t t_addr = smem_u32(my_t);
        float a_q[2], w_q[2];
        my_t[lane & 15] = mul_in_place(ldg_in_place(sa_row + scale_kb(0)), ldg_in_place(sw_row + scale_kb(0)));
#pragma unroll
        for (int j = 0; j < 2; ++j) a_q[(j + 1) & 1] = ldg_in_place(sa_row + scale_kb(j + 1)), w_q[(j + 1) & 1] = ldg_in_place(sw_row + scale_kb(j + 1));
        uint64_t acc[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] = 0ull;
        uint32_t v[2][2][8];  // partials of a stage (two K blocks), two stages in turn
        uint32_t s = 0, ph = 0;
        // Waits for the partials of stage (s, ph) and starts their load.
        auto fetch = [&](uint32_t (&r)[2][8]) {
            if (!warp_agrees(wait_or_abort(&bar_done[s], ph, &abort_flag), p.status, &abort_flag, ERR_TIMEOUT_EPILOGUE)) return false;
            tcgen05_fence_after_sync();
#pragma unroll
            for (int j = 0; j < 2; ++j) tmem_ld_32x32b_x8(tm_warp + (s * 2 + j) * MT, r[j]);
            return true;
        };
        __syncwarp();  // the first scale products
        bool ok = fetch(v[0]);
        // Stage i, whose partials are on their way into v[q]: the next stage's load runs under this one's arithmetic, and all operands of
        // the arithmetic are in registers before it starts (the K blocks of a warp are one serial chain: every latency counts).
        auto stage = [&](int i, auto qc) {
            constexpr int q = decltype(qc)::value;
            uint64_t t[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(t[j][2 * c]), "=l"(t[j][2 * c + 1]) : "r"(t_addr + q * 64 + j * 32 + c * 16) : "memory");
            tmem_ld_wait();
            tcgen05_fence_before_sync();
            __syncwarp();
            mbar_arrive_elected_addr(smem_u32(&bar_read[s]));
            if (++s == STAGES) s = 0, ph ^= 1;
            if (i + 1 < num_st) {
                my_t[(q ^ 1) * 16 + (lane & 15)] = mul_in_place(a_q[q ^ 1], w_q[q ^ 1]);
                __syncwarp();
                a_q[q ^ 1] = ldg_in_place(sa_row + scale_kb(i + 3)), w_q[q ^ 1] = ldg_in_place(sw_row + scale_kb(i + 3));
                ok = fetch(v[q ^ 1]);
                if (!ok) return;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) promote_pair(acc[c], v[q][0][2 * c], v[q][0][2 * c + 1], t[0][c]);
            if (2 * i + 1 < num_kb) {
#pragma unroll
                for (int c = 0; c < 4; ++c) promote_pair(acc[c], v[q][1][2 * c], v[q][1][2 * c + 1], t[1][c]);
            }
        };
        for (int i = 0; i < num_st && ok; i += 2) {
            stage(i, std::integral_constant<int, 0>{});
            if (ok && i + 1 < num_st) stage(i + 1, std::integral_constant<int, 1>{});
        }
        if (n < p.N) {
            const uint16_t b = p.bias ? __ldg(p.bias + n) : uint16_t(0);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (cg * 8 + j < p.M) {
                    float lo, hi;
                    f32x2_split(acc[j / 2], lo, hi);
                    const uint16_t r = to_bf16_bits(j & 1 ? hi : lo);
                    p.out[static_cast<int64_t>(cg * 8 + j) * p.ldo + n] = p.bias ? add_bf16(r, b) : r;
                }
            }
        }
    }

    __syncwarp();
    tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == 3) {
        __syncwarp();
        tcgen05_fence_after_sync();
        tmem_dealloc(tmem_base, S::TMEM_COLS);
    }
}

}  // namespace gi8
