// Stage 1 of the block on the tensor cores for 64 hidden channels (h = 64; c = 64, the narrowest case of
// the reference's d_pair sweep, or c = 128, a projection to half the pair width): LayerNorm_in, pair mask
// and the two sigmoid-gated projections in one pass over z (reference.py:66-75), writing a and b as
// channel-major planes.
//
// Transposed like the other stage-1 kernels (D^T[channel][position], TMEM lane = output channel,
// epilogue thread = one channel and a run of positions -> swizzled staging box -> TMA store), but a
// side has only 64 output channels, and a tcgen05.mma wants M = 128: the LEFT and RIGHT weights are
// stacked into one A operand, [W_left ; W_right] for the projections and [W_left_gate ;
// W_right_gate] for the gates, so lanes 0..63 of the accumulators are the channels of a and lanes
// 64..127 those of b.  A tile is then 8 kSub UMMAs (K = 64 kSub) into 2 x 128 TMEM columns; the
// accumulators are double-buffered and the weight matrices stay in shared memory (halved once, exact in
// bf16, for the half-argument forms of the gate: the hardware tanh for c = 64; for c = 128, where the warp-MMA kernel
// had expf, the fp32 form, which keeps the bits of nearly shut gates.  It costs 1.8 us of a call at N = 512).
//
// What bounds it: HBM (c = 64: z once, a and b once).  LayerNorm and epilogue have the form of the CTA-pair
// kernel (tm1_pair_sm100.cuh): four lanes (c = 64) or eight (c = 128) per LayerNorm row with every value read once, and sixteen
// epilogue warps that store their own boxes, two tiles in flight, instead of one thread per row and two groups
// behind block-wide barriers.  Measured: c = 64, B = 2, N = 512: 1.35 us per tile and CTA on the timeline
// (48 KB of traffic: 5.3 TB/s over the chip), 2.1 us before; c = 128 (K = 128, 64 KB per tile): 2.4 us, paced by the
// LayerNorm of 128 rows x 128 channels (2.5 with the fp32 gates, from N = 448 30.5 -> 32.1 us).
//
// Persistent kernel, one CTA per SM, 832 threads, 128-position tiles:
//   warp 0        TMA producer: the weights once, then z tiles
//   warp 1        UMMA issuer
//   warps 2..9    LayerNorm (+ mask): two groups of four warps on alternate tiles, 32 rows per warp, in place
//                 in the swizzled tile; a masked position becomes a zero row
//   warps 10..25  epilogue, sixteen warps = (accumulator set, position half, TMEM lane quarter)
#pragma once

#include "tm1_common.cuh"

namespace trimul {

constexpr int kN1H = 64;                            // output channels of one side
constexpr int kN1Threads = 832;
constexpr int kN1LnWarps = 8;
constexpr int kN1EpiWarps = 16;
constexpr int kN1BoxBytes = 32 * 64 * 2;            // store box of one epilogue warp: 32 planes x 64 positions
constexpr int kN1LnBarrier = 2;        // 2, 3: the two LayerNorm groups
constexpr int kN1EpiBarrier = 4;       // 4, 5: the eight epilogue warps of accumulator set 0, 1

// kSub = number of 64-channel sub-tiles of a z row (c / 64)
template <int kSub> struct N1Layout {
    static constexpr int kXBytes = kSub * kT1SubTile;           // one z tile: [128 positions][c]
    static constexpr int kXStages = kSub == 1 ? 6 : 3;
    static constexpr int kWBytes = 2 * kSub * kT1SubTile;       // per K sub-tile: stacked proj operand; then the gates
    static constexpr int kOffX = kWBytes;
    static constexpr int kOffBox = kOffX + kXStages * kXBytes;
    static constexpr int kOffBars = kOffBox + kN1EpiWarps * kN1BoxBytes;
    static constexpr int kSmemBytes = kOffBars + 256;
    static_assert(kSmemBytes <= 232448, "narrow stage 1 shared memory exceeds the 227 KB a CTA may use");
    static_assert((6 + 3 * kXStages) * 8 + 8 <= 256, "barrier block too small");
};

template <int kSub>
__global__ void __launch_bounds__(kN1Threads, 1)
tm1_narrow_sm100_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmWl,
                        const __grid_constant__ CUtensorMap tmWlg, const __grid_constant__ CUtensorMap tmWr,
                        const __grid_constant__ CUtensorMap tmWrg, const __grid_constant__ CUtensorMap tmA,
                        const __grid_constant__ CUtensorMap tmB, const __grid_constant__ Tm1Params p) {
    using L = N1Layout<kSub>;
    constexpr int kXStages = L::kXStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0u) {
        if (threadIdx.x == 0) report_timeout(p.status, kStageIdTm1, 900);
        return;
    }
    uint8_t* sW = smem;                       // per K sub-tile [W_left ; W_right], then per K sub-tile the gates
    uint8_t* sX = smem + L::kOffX;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBars);
    uint64_t* w_full = bars;                          // weights landed
    uint64_t* w_ready = bars + 1;                     // weights halved (every worker thread)
    uint64_t* x_full = bars + 2;                      // [stages]
    uint64_t* xn_ready = x_full + kXStages;           // [stages] (4 arrivals: the group's warps)
    uint64_t* x_empty = xn_ready + kXStages;          // [stages]
    uint64_t* acc_full = x_empty + kXStages;          // [2]
    uint64_t* acc_empty = acc_full + 2;               // [2] (8 arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(w_full, 1);
        mbar_init(w_ready, kN1Threads - 64);
        for (int s = 0; s < kXStages; ++s) {
            mbar_init(&x_full[s], 1);
            mbar_init(&xn_ready[s], 4);
            mbar_init(&x_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], kN1EpiWarps / 2);
        }
        *abort_flag = 0;
        fence_mbarrier_init();
        tma_prefetch_desc(&tmZ);
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // Everything above touches no global memory; from here on the kernel reads what its
    // predecessor in the stream may have written.
    griddep_wait();
    griddep_launch_dependents();

    if (warp >= 2) {
        // every worker thread: halve its share of the weights once they have landed
        if (mbar_wait<true>(w_full, 0, abort_flag, p.status, kStageIdTm1, 150)) {
            halve_bf16_smem(sW, L::kWBytes, threadIdx.x - 64, kN1Threads - 64);
            fence_proxy_async_smem();
        }
        mbar_arrive(w_ready);
        __syncwarp();
    }

    const int stride = gridDim.x;
    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            mbar_arrive_expect_tx(w_full, L::kWBytes);
            // box = [64 rows][64 k] = 8 KB: left matrix into rows 0..63, right matrix into rows 64..127
            for (int ks = 0; ks < kSub; ++ks) {
                uint8_t* wp = sW + ks * kT1SubTile;
                uint8_t* wg = sW + (kSub + ks) * kT1SubTile;
                tma_load_2d(wp, &tmWl, w_full, ks * 64, 0);
                tma_load_2d(wp + 8192, &tmWr, w_full, ks * 64, 0);
                tma_load_2d(wg, &tmWlg, w_full, ks * 64, 0);
                tma_load_2d(wg + 8192, &tmWrg, w_full, ks * 64, 0);
            }
            uint32_t it = 0;
            Tm1Cursor cur;
            cur.init(p, blockIdx.x);
            for (int tile = blockIdx.x; tile < p.total_tiles; tile += stride, ++it, cur.next(p, 0)) {
                const int s = it % kXStages;
                const uint32_t ph = (it / kXStages) & 1u;
                if (!mbar_wait<true>(&x_empty[s], ph ^ 1u, abort_flag, p.status, kStageIdTm1, 100 + s)) break;
                TRIMUL_STAMP(0, it, 0);
                mbar_arrive_expect_tx(&x_full[s], L::kXBytes);
                const int col = p.incoming ? cur.f : cur.t0();
                const int row = p.incoming ? cur.t0() : cur.f;
                for (int ks = 0; ks < kSub; ++ks)
                    tma_load_4d(sX + s * L::kXBytes + ks * kT1SubTile, &tmZ, &x_full[s], ks * 64, col, row, cur.b);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ UMMA issuer
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_bf16(128, kT1P);
            bool ok = mbar_wait<true>(w_ready, 0, abort_flag, p.status, kStageIdTm1, 200);
            tcgen05_fence_after();
            const uint32_t wp = smem_u32(sW), wg = smem_u32(sW + kSub * kT1SubTile);
            uint32_t it = 0;
            for (int tile = blockIdx.x; ok && tile < p.total_tiles; tile += stride, ++it) {
                const int s = it % kXStages;
                const uint32_t ph = (it / kXStages) & 1u;
                const int acc = it & 1;
                if (!mbar_wait<true>(&acc_empty[acc], ((it >> 1) & 1u) ^ 1u, abort_flag, p.status, kStageIdTm1, 220 + acc))
                    break;
                TRIMUL_STAMP(1, it, 0);
                if (!mbar_wait<true>(&xn_ready[s], ph, abort_flag, p.status, kStageIdTm1, 210 + s)) break;
                tcgen05_fence_after();
                TRIMUL_STAMP(1, it, 1);
                const uint32_t xs = smem_u32(sX + s * L::kXBytes);
                const uint32_t d_p = tmem_base + acc * 256, d_g = d_p + 128;
#pragma unroll
                for (int kk = 0; kk < 4 * kSub; ++kk) {
                    const uint32_t sub = (kk >> 2) * kT1SubTile;
                    const uint64_t kofs = (kk & 3) * kDescKStep;
                    const uint64_t db = umma_smem_desc_sw128(xs + sub) + kofs;
                    umma_bf16_ss(d_p, umma_smem_desc_sw128(wp + sub) + kofs, db, idesc, kk != 0);
                    umma_bf16_ss(d_g, umma_smem_desc_sw128(wg + sub) + kofs, db, idesc, kk != 0);
                }
                umma_commit(&x_empty[s]);
                umma_commit(&acc_full[acc]);
                TRIMUL_STAMP(1, it, 2);
            }
        }
        __syncwarp();
    } else if (warp < 2 + kN1LnWarps) {
        // ------------------------------------------------------------------ LayerNorm (+ mask)
        // warp lw of group lg owns rows [32 lw, 32 lw + 32) of every second tile; four lanes per row of 64 channels
        // (a tile of the group in 1.3 us, 2.5 us with eight lanes), eight per row of 128
        const int lg = (warp - 2) >> 2;
        const int lw = (warp - 2) & 3;
        constexpr int kRows = kSub == 1 ? 8 : 4;       // rows per step of a warp
        const int rr = lane / (32 / kRows);
        f32x2 gb[16];
        if constexpr (kSub == 1) ln_load_affine_quad(gb, p.gamma, p.beta, lane);
        else ln_load_affine<kSub>(gb, p.gamma, p.beta, lane);
        const int first = blockIdx.x + lg * stride;
        uint32_t it = lg;
        Tm1Cursor cur;
        cur.init(p, first);
        // pair mask: lane l looks up position 32 lw + l one tile ahead, a ballot hands the bits out
        bool keep_next = true;
        if (p.mask_kind != 0 && first < p.total_tiles) keep_next = tm1_keep(p, cur.b, cur.f, cur.t0() + 32 * lw + lane);
        for (int tile = first; tile < p.total_tiles; tile += 2 * stride, it += 2) {
            const int s = it % kXStages;
            const uint32_t ph = (it / kXStages) & 1u;
            const bool keep = keep_next;
            cur.next(p, 1);
            if (p.mask_kind != 0 && tile + 2 * stride < p.total_tiles)
                keep_next = tm1_keep(p, cur.b, cur.f, cur.t0() + 32 * lw + lane);
            if (!group_wait<true>(&x_full[s], ph, lw == 0 && lane == 0, kN1LnBarrier + lg, 128, abort_flag, p.status,
                                  kStageIdTm1, 300 + s))
                break;
            uint32_t zero_bits = 0u;
            if (p.mask_kind != 0) {
                const uint32_t drop = ~__ballot_sync(0xffffffffu, keep);
#pragma unroll
                for (int i = 0; i < 32 / kRows; ++i) zero_bits |= ((drop >> (kRows * i + rr)) & 1u) << i;
            }
            if (lw == 0 && lane == 0) TRIMUL_STAMP(2, it, 0);
            if constexpr (kSub == 1) ln_rows64_warp<4>(sX + s * L::kXBytes, 32 * lw, lane, gb, p.eps, zero_bits);
            else ln_rows_warp<8, kSub>(sX + s * L::kXBytes, kT1SubTile, 32 * lw, lane, gb, p.eps, zero_bits);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&xn_ready[s]);
            if (lw == 0 && lane == 0) TRIMUL_STAMP(2, it, 1);
        }
    } else {
        // ------------------------------------------------------------------ epilogue, sixteen warps
        // Warp = (accumulator set eb, position half, TMEM lane quarter q): 32 planes x 64 positions of every
        // second tile into its own store box; quarters 0, 1 are channels of a, quarters 2, 3 of b.
        const int ew = warp - 10;
        const uint32_t eb = (uint32_t)ew >> 3;
        const int half = (ew >> 2) & 1;
        const int q = warp & 3;
        uint8_t* box = smem + L::kOffBox + ew * kN1BoxBytes;
        const bool left = q < 2;
        const CUtensorMap* om = left ? &tmA : &tmB;
        const int rc = left ? p.a_row_chunk : p.b_row_chunk;
        const int cc = left ? p.a_col_chunk : p.b_col_chunk;
        const uint32_t t_p = tmem_base + eb * 256 + half * 64 + ((uint32_t)(q * 32) << 16);
        uint32_t it = eb;
        Tm1Cursor cur;
        const int first = blockIdx.x + (int)eb * stride;
        cur.init(p, first);
        for (int tile = first; tile < p.total_tiles; tile += 2 * stride, it += 2, cur.next(p, 1)) {
            if (lane == 0) tma_store_wait_read<0>();   // this warp's previous store has read the box
            if (!group_wait<true>(&acc_full[eb], (it >> 1) & 1u, (ew & 7) == 0 && lane == 0, kN1EpiBarrier + (int)eb, 256,
                                  abort_flag, p.status, kStageIdTm1, 400 + (int)eb))
                break;
            tcgen05_fence_after();
            if ((ew & 7) == 0 && lane == 0) TRIMUL_STAMP(3, it, 0);
            auto emit8 = [&](int c8, const uint32_t (&rp)[8], const uint32_t (&rg)[8]) {
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    o[e] = gate_halves_bf16<kSub == 2>(f2_pack(__uint_as_float(rp[2 * e]), __uint_as_float(rp[2 * e + 1])),
                                                       f2_pack(__uint_as_float(rg[2 * e]), __uint_as_float(rg[2 * e + 1])));
                const int chunk = c8 ^ (lane & 7);
                *reinterpret_cast<uint4*>(box + lane * 128 + (chunk << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            };
            uint32_t rpA[8], rgA[8], rpB[8], rgB[8];
            tmem_ld_32x8(t_p, rpA);
            tmem_ld_32x8(t_p + 128, rgA);
#pragma unroll 1
            for (int c8 = 0; c8 < 8; c8 += 2) {
                tmem_ld_wait();
                tmem_ld_32x8(t_p + (c8 + 1) * 8, rpB);
                tmem_ld_32x8(t_p + 128 + (c8 + 1) * 8, rgB);
                emit8(c8, rpA, rgA);
                tmem_ld_wait();
                if (c8 + 2 < 8) {
                    tmem_ld_32x8(t_p + (c8 + 2) * 8, rpA);
                    tmem_ld_32x8(t_p + 128 + (c8 + 2) * 8, rgA);
                } else {
                    // every TMEM read of this warp's share has completed
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[eb]);
                    if ((ew & 7) == 0 && lane == 0) TRIMUL_STAMP(3, it, 1);
                }
                emit8(c8 + 1, rpB, rgB);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                const int col0 = cur.t0() + half * 64;
                if (col0 < p.n_run) {
                    tma_store_4d(om, box, col0 % cc, cur.f % rc, cur.b * kN1H + (q & 1) * 32, col0 / cc + cur.f / rc);
                    tma_store_commit();
                }
                if ((ew & 7) == 0) TRIMUL_STAMP(3, it, 2);
            }
        }
        if (lane == 0) tma_store_wait_all<0>();
        __syncwarp();
    }

    if (*abort_flag != 0) {
        for (int i = 0; i < 256; ++i) __nanosleep(1000);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace trimul
