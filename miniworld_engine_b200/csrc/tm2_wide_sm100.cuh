// Stage 3 of the block on the tensor cores for c = h = 256 (reference.py:76-83):
// out = sigmoid(Wg . LN_in(z)) * (Wo . LN_out(tri)) [* drop_scale] [+ residual].
//
// Both LayerNorms are folded into the projections as in tm2_fold_sm100.cuh: the tensor cores multiply
// the RAW z and tri tiles by W * gamma / 2, mean and rstd of every position enter in the epilogue as
// one FMA per value.  Nothing is normalised in place, so the operands can stream through shared
// memory in 64-channel SLICES, and that is what makes room for the weights: the two 256 x 256 matrices
// (256 KB) are resident, one half in each CTA of a PAIR (tcgen05 cta_group::2, M = 256 positions, N = 256
// output channels: A is read from the CTA that owns the 128 positions, B half from each CTA).
// A slice is read once from memory and used by four UMMAs of 256 x 256 x 16.
//
// What bounds it: HBM in principle (z, tri and out once: 192 KB per tile and CTA, 4.4 us at the copy rate); in
// fact the two accumulators fill the 512 TMEM columns, so a tile's UMMAs (2.1 us) and its epilogue
// alternate, and only the loads run ahead (four slices).  Measured: 8.7 us per tile on the timeline (epilogue 4.2,
// UMMAs 3.7, of which 1.6 are the latency of the second four slices), 13.8 with streamed weights, both LayerNorms in
// place and one tile at a time; B = 2, N = 512 with the residual: 383 -> 270 us in the step, N = 384: 106 -> 95.
//
// Persistent kernel, CTA pairs, 640 threads per CTA, 128-position tiles (z row r, columns j0..j0+127); CTA k of a
// pair works on tile 2 i + k of the list, whatever row that lies in:
//   warp 0        TMA producer: this CTA's weight halves once; per tile four z slices [128 positions][64 channels],
//                 then four tri slices [64 channel rows][128 positions], through a ring of four
//   warp 1        UMMA issuer (leader CTA): gate += z slice . Wg'^T (K-major), proj += tri slice . Wo'^T (MN-major, used
//                 as the contraction wrote it)
//   warp 2        tells the leader that a slice of this CTA has landed
//   warp 3        idle
//   warps 4..7    statistics: of the z slices one thread per position, of the tri slices 8 positions x 8 channel
//                 rows per thread and a halving butterfly over the 8 lanes that share the positions
//   warps 8..19   epilogue: warp = (TMEM lane quarter, third of the eight 32-channel pieces): TMEM -> statistics ->
//                 gate -> (* scale) (+ residual) -> bf16 -> the warp's own [32 positions][32 channels] box -> TMA store
// Before the first tile warps 4..19 fold gamma and 1/2 into the weights, Wg while Wo is still on its way, while the tile's z
// slices arrive; the per-channel (rowsum, bias) pairs are written to both CTAs.  With one tile per CTA that start is a third
// of the stage: with eight folding warps and z slices requested only after the fold the block took 1.5 us longer (N = 64
// 40.1 -> 38.6 us without the residual, 40.6 -> 39.0 with it; N = 256 117.1 -> 114.7 and 121.2 -> 117.8).
//
// mbarriers (full, empty, acc_full, stat in each CTA; ready and acc_empty used in the leader only):
//   full[s]       this CTA's slice landed        ready[s]      2 arrivals: both CTAs' slices landed
//   empty[s]      5 arrivals: the pair's UMMAs that read the slot retired, four statistics warps done
//   acc_full      the tile's UMMAs retired       acc_empty     24 arrivals: every epilogue warp of both CTAs
//   stat[2]       4 arrivals: statistics of the tile written (two tiles' worth of buffers)
#pragma once

#include "tm2_sm100.cuh"

namespace trimul {

constexpr int kW2C = 256;
constexpr int kW2Threads = 640;
constexpr int kW2Slots = 4;
constexpr int kW2SlotBytes = kT2SubTile;            // 16 KB
constexpr int kW2EpiWarps = 12;
constexpr int kW2BoxBytes = 32 * 32 * 2;
constexpr int kW2WSub = 128 * 128;                  // [128 output channels][64 k] of a weight half
constexpr int kW2OffSlots = 8 * kW2WSub;            // Wg: 4 K slices, Wo: 4 K slices
constexpr int kW2OffBox = kW2OffSlots + kW2Slots * kW2SlotBytes;
constexpr int kW2OffConst = kW2OffBox + kW2EpiWarps * kW2BoxBytes;  // [2 matrices][128 channel pairs] (s0, s1, b0, b1)
constexpr int kW2OffStat = kW2OffConst + 2 * 128 * 16;              // [2 tiles][128 positions] (r_in, t_in, r_out, t_out)
constexpr int kW2OffBars = kW2OffStat + 2 * 128 * 16;
constexpr int kW2SmemBytes = kW2OffBars + 256;
constexpr int kW2StatBarrier = 2;
constexpr int kW2EpiBarrier = 3;
static_assert(kW2SmemBytes <= 232448, "wide stage 3 shared memory exceeds the 227 KB a CTA may use");

struct Tm2WideParams {
    Tm2Params base;
    const __nv_bfloat16* residual;     // [B, rows, N, 256] or null
    const __nv_bfloat16* drop_scale;   // [B, 1, N, 256] or null
};

__device__ __forceinline__ void st_cluster_f32(uint32_t cluster_addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(cluster_addr), "f"(v) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kW2Threads, 1)
tm2_wide_sm100_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmWg,
                      const __grid_constant__ CUtensorMap tmWo, const __grid_constant__ CUtensorMap tmOut,
                      const __grid_constant__ CUtensorMap tmTri, const __grid_constant__ Tm2WideParams wp) {
    const Tm2Params& p = wp.base;
    extern __shared__ __align__(1024) uint8_t smem[];
    if ((smem_u32(smem) & 1023u) != 0u) {
        // both CTAs of a pair see the same offset, so both leave here and nobody waits for the other
        if (threadIdx.x == 0) report_timeout(p.status, kStageIdTm2, 900);
        return;
    }
    uint8_t* sW = smem;
    uint8_t* sSlot = smem + kW2OffSlots;
    float4* sConst = reinterpret_cast<float4*>(smem + kW2OffConst);
    float4* sStat = reinterpret_cast<float4*>(smem + kW2OffStat);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kW2OffBars);
    uint64_t* w_full = bars;                  // [2] Wg, Wo half landed
    uint64_t* full = bars + 2;                // [slots]
    uint64_t* ready = full + kW2Slots;        // [slots] leader
    uint64_t* empty = ready + kW2Slots;       // [slots]
    uint64_t* acc_full = empty + kW2Slots;
    uint64_t* acc_empty = acc_full + 1;       // leader
    uint64_t* stat = acc_empty + 1;           // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stat + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    static_assert((6 + 3 * kW2Slots) * 8 + 8 <= 256, "barrier block too small");

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();     // 0 = leader
    const bool is_leader = rank == 0;

    if (threadIdx.x == 0) {
        mbar_init(&w_full[0], 1);
        mbar_init(&w_full[1], 1);
        for (int s = 0; s < kW2Slots; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&ready[s], 2);
            mbar_init(&empty[s], 5);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * kW2EpiWarps);
        mbar_init(&stat[0], 4);
        mbar_init(&stat[1], 4);
        *abort_flag = 0;
        fence_mbarrier_init();
        tma_prefetch_desc(&tmZ);
        tma_prefetch_desc(&tmTri);
        tma_prefetch_desc(&tmOut);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();          // both CTAs' barriers are initialised before anyone signals the peer
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // set-up done without touching global memory: now wait for the producer of tri (and of z)
    griddep_wait();
    griddep_launch_dependents();

    // this CTA's tiles: 2 * pair + rank; an odd last one is worked on twice and stored once
    const int cluster_id = blockIdx.x >> 1;
    const int num_clusters = gridDim.x >> 1;
    const int total_pairs = (p.total_tiles + 1) / 2;
    auto place = [&](int pt, int& b, int& r, int& j0) {
        const int tile = min(2 * pt + (int)rank, p.total_tiles - 1);
        j0 = (tile % p.tiles_per_row) * kT2P;
        const int br = tile / p.tiles_per_row;
        r = br % p.rows;
        b = br / p.rows;
    };

    // slice u of this CTA (slice j of its tile) into slot u % kW2Slots
    auto load_slice = [&](uint32_t u, int j, int b, int r, int j0) {
        const int s = u % kW2Slots;
        mbar_arrive_expect_tx(&full[s], kW2SlotBytes);
        uint8_t* dst = sSlot + s * kW2SlotBytes;
        if (j < 4) {
            tma_load_4d(dst, &tmZ, &full[s], j * 64, j0, r, b);
        } else {
            // tri planes viewed as (column, row, plane, chunk): 64 columns x 64 planes per box
            const int plane = b * kW2C + (j - 4) * 64;
            tma_load_4d(dst, &tmTri, &full[s], j0, r, plane, 0);
            tma_load_4d(dst + kW2SlotBytes / 2, &tmTri, &full[s], j0 + 64, r, plane, 0);
        }
    };
    if (warp == 0 && lane == 0) {
        mbar_arrive_expect_tx(&w_full[0], 4 * kW2WSub);
        for (int ks = 0; ks < 4; ++ks) tma_load_2d(sW + ks * kW2WSub, &tmWg, &w_full[0], ks * 64, (int)rank * 128);
        mbar_arrive_expect_tx(&w_full[1], 4 * kW2WSub);
        for (int ks = 0; ks < 4; ++ks) tma_load_2d(sW + (4 + ks) * kW2WSub, &tmWo, &w_full[1], ks * 64, (int)rank * 128);
        // the first tile's z slices fill the empty ring while the weights are folded
        int b, r, j0;
        place(cluster_id, b, r, j0);
        for (int j = 0; j < kW2Slots; ++j) load_slice(j, j, b, r, j0);
    }
    __syncwarp();
    if (warp >= 4) {
        // two threads per row: matrix m (0: Wg with LN_in, 1: Wo with LN_out), row n of this CTA's half, half of the K slices
        // (16 rows and both K halves in a warp: eight lanes of a quarter warp on eight rows of one K slice)
        const int w = warp - 4, m = w >> 3, n = 16 * (w & 7) + (lane & 15), kh = lane >> 4;
        float s_ = 0.f, b_ = 0.f;
        const bool landed = mbar_wait<true>(&w_full[m], 0, abort_flag, p.status, kStageIdTm2, 1150);
        if (landed) {
            fold_row_smem(sW + (4 * m + 2 * kh) * kW2WSub, kW2WSub, n, (m == 0 ? p.gamma_in : p.gamma_out) + 128 * kh,
                          (m == 0 ? p.beta_in : p.beta_out) + 128 * kh, 2, s_, b_);
            fence_proxy_async_smem();      // folded weights -> visible to the UMMA (async proxy)
        }
        __syncwarp();
        s_ += __shfl_xor_sync(0xffffffffu, s_, 16);
        b_ += __shfl_xor_sync(0xffffffffu, b_, 16);
        if (landed) {                      // K half kh writes the pair's sums to CTA kh
            const int ch = (int)rank * 128 + n;
            const uint32_t a = map_to_cta(smem_u32(reinterpret_cast<float*>(&sConst[m * 128 + (ch >> 1)]) + (ch & 1)), (uint32_t)kh);
            st_cluster_f32(a, s_);
            st_cluster_f32(a + 8, b_);
        }
    }
    __syncwarp();
    cluster_sync_all();          // weights folded and constants written in both CTAs

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            uint32_t u = kW2Slots;         // slices 0 .. 3 of the first tile are on their way
            bool ok = true;
            for (int pt = cluster_id; ok && pt < total_pairs; pt += num_clusters) {
                int b, r, j0;
                place(pt, b, r, j0);
                for (int j = pt == cluster_id ? kW2Slots : 0; j < 8; ++j, ++u) {
                    const int s = u % kW2Slots;
                    if (!mbar_wait<true>(&empty[s], ((u / kW2Slots) & 1u) ^ 1u, abort_flag, p.status, kStageIdTm2, 1100 + s)) {
                        ok = false;
                        break;
                    }
                    load_slice(u, j, b, r, j0);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------------ UMMA issuer (leader)
        if (lane == 0 && is_leader) {
            constexpr uint32_t idesc = umma_idesc_bf16(256, 256);
            constexpr uint32_t idesc_mn = umma_idesc_bf16(256, 256, 1, 0);   // A (tri) is MN-major
            uint32_t u = 0, it = 0;
            bool ok = true;
            const uint32_t wg = smem_u32(sW), wo = smem_u32(sW + 4 * kW2WSub);
            for (int pt = cluster_id; ok && pt < total_pairs; pt += num_clusters, ++it) {
                if (!mbar_wait<true>(acc_empty, (it & 1u) ^ 1u, abort_flag, p.status, kStageIdTm2, 1210)) break;
                TRIMUL_STAMP(1, it, 0);
                for (int j = 0; j < 8; ++j, ++u) {
                    const int s = u % kW2Slots;
                    if (!mbar_wait<true>(&ready[s], (u / kW2Slots) & 1u, abort_flag, p.status, kStageIdTm2, 1220 + s)) {
                        ok = false;
                        break;
                    }
                    tcgen05_fence_after();
                    if (j == 4) TRIMUL_STAMP(1, it, 1);
                    const uint32_t sl = smem_u32(sSlot + s * kW2SlotBytes);
                    const uint64_t db = umma_smem_desc_sw128((j < 4 ? wg : wo) + (j & 3) * kW2WSub);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint32_t acc = ((j & 3) | kk) != 0 ? 1u : 0u;
                        if (j < 4)
                            umma_bf16_ss_pair(tmem_base, umma_smem_desc_sw128(sl) + kk * kDescKStep, db + kk * kDescKStep,
                                              idesc, acc);
                        else
                            // slice rows are channels (K), 128 bytes = 64 positions per row, the second 64 positions
                            // 8 KB further; a K step of 16 is two 8-row groups = 2048 B
                            umma_bf16_ss_pair(tmem_base + 256,
                                              umma_smem_desc_mn_sw128(sl + kk * 2048, kW2SlotBytes / 2, 1024),
                                              db + kk * kDescKStep, idesc_mn, acc);
                    }
                    umma_commit_pair(&empty[s]);
                }
                if (ok) umma_commit_pair(acc_full);
                TRIMUL_STAMP(1, it, 2);
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ------------------------------------------------------------------ slice landed -> leader
        if (lane == 0) {
            uint32_t u = 0;
            bool ok = true;
            for (int pt = cluster_id; ok && pt < total_pairs; pt += num_clusters)
                for (int j = 0; j < 8; ++j, ++u) {
                    const int s = u % kW2Slots;
                    if (!mbar_wait<true>(&full[s], (u / kW2Slots) & 1u, abort_flag, p.status, kStageIdTm2, 1250 + s)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_remote(map_to_cta(smem_u32(&ready[s]), 0));
                }
        }
        __syncwarp();
    } else if (warp == 3) {
        // idle
    } else if (warp < 8) {
        // ------------------------------------------------------------------ statistics
        const int tid = threadIdx.x - 128;             // 0..127: position (z), and what the butterfly leaves it with (tri)
        const bool poller = tid == 0;
        // tri: position chunk cq (positions 8 cq .. 8 cq + 7), channel rows rs, rs + 8, ... of a slice; all of them
        // have r & 7 == rs, so its 16 bytes sit at the same offset in every row
        const int rs = lane & 7;
        const int cq = 4 * (warp - 4) + (lane >> 3);
        const uint32_t col_off = (uint32_t)(cq >> 3) * (kW2SlotBytes / 2) + ((((uint32_t)cq & 7u) ^ (uint32_t)rs) << 4);
        const uint32_t zsw = (uint32_t)(tid & 7);
        constexpr float kInvC = 1.0f / (float)kW2C;
        uint32_t u = 0, it = 0;
        bool alive = true;
        for (int pt = cluster_id; alive && pt < total_pairs; pt += num_clusters, ++it) {
            // ---- z: one thread per position, sums shifted by the position's channel 0
            float shift = 0.f;
            f32x2 nshift = 0ull;
            f32x2 s1[4] = {0ull, 0ull, 0ull, 0ull}, s2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 1
            for (int j = 0; j < 4; ++j, ++u) {
                const int s = u % kW2Slots;
                if (!group_wait<true>(&full[s], (u / kW2Slots) & 1u, poller, kW2StatBarrier, 128, abort_flag, p.status,
                                      kStageIdTm2, 1300 + s)) {
                    alive = false;
                    break;
                }
                const uint8_t* rowp = sSlot + s * kW2SlotBytes + tid * 128;
                if (j == 0) {
                    shift = bf16_lo(*reinterpret_cast<const uint32_t*>(rowp + (zsw << 4)));
                    nshift = f2_pack(-shift, -shift);
                }
#pragma unroll 4
                for (int k = 0; k < 8; ++k) {
                    const uint4 v = *reinterpret_cast<const uint4*>(rowp + ((((uint32_t)k) ^ zsw) << 4));
                    const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const f32x2 d = f2_add(f2_from_bf16x2(w4[e]), nshift);
                        s1[e] = f2_add(s1[e], d);
                        s2[e] = f2_fma(d, d, s2[e]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);
            }
            if (!alive) break;
            {
                const float m1 = f2_hsum(f2_add(f2_add(s1[0], s1[1]), f2_add(s1[2], s1[3]))) * kInvC;
                const float q1 = f2_hsum(f2_add(f2_add(s2[0], s2[1]), f2_add(s2[2], s2[3])));
                const float rstd = rsqrtf(fmaxf(fmaf(-m1, m1, q1 * kInvC), 0.f) + p.eps_in);
                *reinterpret_cast<float2*>(&sStat[(it & 1u) * 128 + tid]) = make_float2(rstd, -(shift + m1) * rstd);
            }
            // ---- tri
            uint32_t sh[4] = {0u, 0u, 0u, 0u};
            f32x2 nsh[4] = {0ull, 0ull, 0ull, 0ull}, a[4] = {0ull, 0ull, 0ull, 0ull}, qq[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 1
            for (int j = 0; j < 4; ++j, ++u) {
                const int s = u % kW2Slots;
                if (!group_wait<true>(&full[s], (u / kW2Slots) & 1u, poller, kW2StatBarrier, 128, abort_flag, p.status,
                                      kStageIdTm2, 1310 + s)) {
                    alive = false;
                    break;
                }
                const uint8_t* base = sSlot + s * kW2SlotBytes + col_off + rs * 128;
                if (j == 0) {
                    // common shift of each position: its channel 0 (row 0, held by the rs == 0 lane)
                    const uint4 v0 = *reinterpret_cast<const uint4*>(base);
                    sh[0] = __shfl_sync(0xffffffffu, v0.x, lane & 24);
                    sh[1] = __shfl_sync(0xffffffffu, v0.y, lane & 24);
                    sh[2] = __shfl_sync(0xffffffffu, v0.z, lane & 24);
                    sh[3] = __shfl_sync(0xffffffffu, v0.w, lane & 24);
#pragma unroll
                    for (int w = 0; w < 4; ++w) nsh[w] = f2_pack(-bf16_lo(sh[w]), -bf16_hi(sh[w]));
                }
#pragma unroll 4
                for (int m = 0; m < 8; ++m) {
                    const uint4 v = *reinterpret_cast<const uint4*>(base + m * 1024);
                    const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const f32x2 d = f2_add(f2_from_bf16x2(w4[w]), nsh[w]);
                        a[w] = f2_add(a[w], d);
                        qq[w] = f2_fma(d, d, qq[w]);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);
            }
            if (!alive) break;
            float t1[8], t2[8];
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                f2_unpack(a[w], t1[2 * w], t1[2 * w + 1]);
                f2_unpack(qq[w], t2[2 * w], t2[2 * w + 1]);
            }
            // halving butterfly: after the three steps lane rs holds the complete sums of position rs of the chunk
#pragma unroll
            for (int half = 4; half >= 1; half >>= 1) {
                const bool up = (rs & half) != 0;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const float send1 = up ? t1[i] : t1[i + half], keep1 = up ? t1[i + half] : t1[i];
                    const float send2 = up ? t2[i] : t2[i + half], keep2 = up ? t2[i + half] : t2[i];
                    t1[i] = keep1 + __shfl_xor_sync(0xffffffffu, send1, half);
                    t2[i] = keep2 + __shfl_xor_sync(0xffffffffu, send2, half);
                }
            }
            const uint32_t shw = (rs >> 1) == 0 ? sh[0] : (rs >> 1) == 1 ? sh[1] : (rs >> 1) == 2 ? sh[2] : sh[3];
            const float tshift = (rs & 1) ? bf16_hi(shw) : bf16_lo(shw);
            const float m1 = t1[0] * kInvC;
            const float rstd = rsqrtf(fmaxf(fmaf(-m1, m1, t2[0] * kInvC), 0.f) + p.eps_out);
            // position 8 cq + rs == tid
            *(reinterpret_cast<float2*>(&sStat[(it & 1u) * 128 + tid]) + 1) = make_float2(rstd, -(tshift + m1) * rstd);
            __syncwarp();
            if (lane == 0) mbar_arrive(&stat[it & 1u]);
        }
    } else {
        // ------------------------------------------------------------------ epilogue
        const int ew = warp - 8;
        const int grp = ew >> 2;                       // pieces grp, grp + 3, grp + 6 of the eight
        const int q = warp & 3;
        const int row = q * 32 + lane;                 // position inside the tile == TMEM lane
        const bool poller = ew == 0 && lane == 0;
        uint8_t* box = smem + kW2OffBox + ew * kW2BoxBytes;
        uint8_t* box_row = box + lane * 64;
        const uint32_t bsw = ((uint32_t)lane >> 1) & 3u;              // 64-byte swizzle of the store box
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
        const ulonglong2* cG = reinterpret_cast<const ulonglong2*>(sConst);
        const ulonglong2* cO = cG + 128;
        uint32_t it = 0;
        for (int pt = cluster_id; pt < total_pairs; pt += num_clusters, ++it) {
            int b, r, j0;
            place(pt, b, r, j0);
            const bool in_range = j0 + row < p.N;
            const __nv_bfloat16* scale = wp.drop_scale != nullptr && in_range
                ? wp.drop_scale + ((size_t)b * p.N + j0 + row) * kW2C : nullptr;
            // A piece's residual goes through the warp's store box: four lanes read the 64 bytes of a position (one
            // position per thread would touch 32 lines per load, which kept the load/store pipe busy for 2 us per tile),
            // fetched one piece ahead, the first one while the UMMAs run.
            uint4 rn[4];
            const int rrow = lane >> 2;               // positions rrow, rrow + 8, ... of the warp's 32
            auto fetch_res = [&](int piece) {
                if (wp.residual == nullptr || piece >= 8) return;
                const __nv_bfloat16* src = wp.residual + (((size_t)b * p.rows + r) * p.N + j0 + q * 32 + rrow) * kW2C +
                                           piece * 32 + (lane & 3) * 8;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    rn[k] = j0 + q * 32 + rrow + 8 * k < p.N ? __ldg(reinterpret_cast<const uint4*>(src + (size_t)k * 8 * kW2C))
                                                            : make_uint4(0u, 0u, 0u, 0u);
            };
            fetch_res(grp);
            bool ok = true;
            if (poller)
                ok = mbar_wait<true>(&stat[it & 1u], (it >> 1) & 1u, abort_flag, p.status, kStageIdTm2, 1410) &&
                     mbar_wait<true>(acc_full, it & 1u, abort_flag, p.status, kStageIdTm2, 1400);
            if (!named_barrier_all(kW2EpiBarrier, kW2EpiWarps * 32, ok)) break;
            tcgen05_fence_after();
            if (ew == 0 && lane == 0) TRIMUL_STAMP(3, it, 0);
            const float4 st = sStat[(it & 1u) * 128 + row];
            const f32x2 rin = f2_pack(st.x, st.x), tin = f2_pack(st.y, st.y);
            const f32x2 rout = f2_pack(st.z, st.z), tout = f2_pack(st.w, st.w);
            const bool store = 2 * pt + (int)rank < p.total_tiles && j0 + q * 32 < p.N;
#pragma unroll 1
            for (int piece = grp; piece < 8; piece += 3) {
                const int ch0 = piece * 32;
                uint32_t rgA[8], rpA[8], rgB[8], rpB[8];
                tmem_ld_32x8(t_row + ch0, rgA);
                tmem_ld_32x8(t_row + 256 + ch0, rpA);
                if (lane == 0) tma_store_wait_read<0>();   // this warp's previous store has read the box
                __syncwarp();
                if (wp.residual != nullptr) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)           // rows rrow + 8 k: (row >> 1) & 3 == (rrow >> 1) & 3
                        *reinterpret_cast<uint4*>(box + (rrow + 8 * k) * 64 +
                                                  ((((uint32_t)lane & 3u) ^ (((uint32_t)rrow >> 1) & 3u)) << 4)) = rn[k];
                    __syncwarp();
                    fetch_res(piece + 3);
                }
                auto emit8 = [&](int c8, const uint32_t (&rg)[8], const uint32_t (&rp)[8]) {
                    uint32_t o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int pair = ch0 / 2 + c8 * 4 + k;
                        const ulonglong2 kg = cG[pair], ko = cO[pair];     // the channel pair's constants
                        const f32x2 hg = f2_fma(f2_pack(__uint_as_float(rg[2 * k]), __uint_as_float(rg[2 * k + 1])), rin,
                                                f2_fma(tin, kg.x, kg.y));
                        const f32x2 ho = f2_fma(f2_pack(__uint_as_float(rp[2 * k]), __uint_as_float(rp[2 * k + 1])), rout,
                                                f2_fma(tout, ko.x, ko.y));
                        float g0, g1;
                        f2_unpack(hg, g0, g1);
                        o[k] = f2_to_bf16x2(f2_fma(ho, f2_pack(tanh_fast(g0), tanh_fast(g1)), ho));
                    }
                    if (scale != nullptr) {   // the scale multiplies the rounded block output, like `out * scale`
                        const uint4 dv = __ldg(reinterpret_cast<const uint4*>(scale + ch0) + c8);
                        const uint32_t dw[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = f2_to_bf16x2(f2_mul(f2_from_bf16x2(o[k]), f2_from_bf16x2(dw[k])));
                    }
                    uint4* dst = reinterpret_cast<uint4*>(box_row + (((uint32_t)c8 ^ bsw) << 4));
                    if (wp.residual != nullptr) {     // the reference rounds the block output to bf16 before `out + pair`
                        const uint4 rv = *dst;
                        const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            o[k] = f2_to_bf16x2(f2_add(f2_from_bf16x2(o[k]), f2_from_bf16x2(rw[k])));
                    }
                    *dst = make_uint4(o[0], o[1], o[2], o[3]);
                };
#pragma unroll
                for (int c8 = 0; c8 < 4; c8 += 2) {
                    tmem_ld_wait();
                    tmem_ld_32x8(t_row + ch0 + (c8 + 1) * 8, rgB);
                    tmem_ld_32x8(t_row + 256 + ch0 + (c8 + 1) * 8, rpB);
                    emit8(c8, rgA, rpA);
                    tmem_ld_wait();
                    if (c8 + 2 < 4) {
                        tmem_ld_32x8(t_row + ch0 + (c8 + 2) * 8, rgA);
                        tmem_ld_32x8(t_row + 256 + ch0 + (c8 + 2) * 8, rpA);
                    } else if (piece + 3 >= 8) {
                        // every TMEM read of this warp's share of the accumulators has completed
                        tcgen05_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(acc_empty), 0));
                        if (ew == 0 && lane == 0) TRIMUL_STAMP(3, it, 1);
                    }
                    emit8(c8 + 1, rgB, rpB);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0 && store) {
                    tma_store_4d(&tmOut, box, ch0, j0 + q * 32, r, b);
                    tma_store_commit();
                }
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
    cluster_sync_all();          // the peer may still be reading this CTA's shared memory / barriers
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

}  // namespace trimul
