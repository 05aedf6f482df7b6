// W8A8 GEMM for more than 64 rows (gk == K) on CTA pairs with the operands exchanged.  The weight rows are the MMA's M operand (256 of
// them, 128 per CTA and tensor-memory lane set), the activation rows its N: a row tile is any multiple of 32 up to 256, the sizes
// that an int8 MMA of a CTA pair has.
// A CTA of a pair reads and is sent half of the activation tile, a third less than a 128 x 256 tile needs on one CTA.  ncu, 34816 x 5120
// at 2,048 rows against w8a8_tile_kernel: tensor pipe 93.6 % of the active cycles (76.7), shared-memory banks 24 % for reads and for
// writes (29), 217.6 us (250.7).  A stage takes 2.06 cycles per activation row (its MMAs alone 2), 355 + nt / 4 where that is more, and
// the drain of a pair's last tile 42 cycles per row: the bound of small products (5120 x 5120 at 500 rows, tiles of 192: 16,200 cycles
// of stages, 8,100 of drain).
// Barriers as in w8a8_pair_kernel: `full` and `tempty` in the leader, `empty` and `tfull` in both CTAs.  No multicast.
#pragma once
#include "w8a8_gemm.cuh"

namespace w8a8 {

constexpr int TP_MAX = 256;                                       // activation rows of a tile
constexpr int TP_STAGES = 6;
constexpr int TP_STAGE_BYTES = BM * BK + TP_MAX / 2 * BK;         // per CTA: 128 weight rows, half of the activation rows
constexpr int TP_SMEM = TP_STAGES * TP_STAGE_BYTES + 1024 + (int)sizeof(Aux) + 2 * TP_MAX * 4;
constexpr int TP_THREADS = 64 + 8 * 32;

// REGS (residual add): read, one rounded add, write, 16 rows requested ahead - before the products are there, for the first ones.
// Otherwise a reduction at the memory side, for which nothing waits, but which flushes values below 2^-126.
template <int EPI, bool REGS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1)
w8a8_tpair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a, const float* __restrict__ a_s,
                  const float* __restrict__ w_s, void* __restrict__ out, long ldo, const int* __restrict__ n_rows, int M, int N,
                  int K, int nt, int flags) {
    const int n_fastest = flags & 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = align1024(smem_raw);
    Aux* aux = (Aux*)(smem + TP_STAGES * TP_STAGE_BYTES);
    float* sa_stash = (float*)(aux + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;

    int live = *n_rows;
    live = live < M ? live : M;
    const int num_m = (live + nt - 1) / nt, num_n = (N + 2 * BM - 1) / (2 * BM);
    const int num_tiles = num_m * num_n, KB = (K + BK - 1) / BK;
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    auto tile_m = [&](int t) { return (n_fastest ? t / num_n : t % num_m) * nt; };
    auto tile_n = [&](int t) { return (n_fastest ? t % num_n : t / num_m) * 2 * BM; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < TP_STAGES; ++s) {
            mbar_init(smem_u32(&aux->full[s]), 1);                // used in the leader only
            mbar_init(smem_u32(&aux->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&aux->tfull[b]), 1);
            mbar_init(smem_u32(&aux->tempty[b]), 16);             // used in the leader only: 8 warps of each CTA
        }
        aux->abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(&aux->tmem_base), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                            // both CTAs' barriers exist before any remote use
    tc_fence_after();
    const uint32_t tmem_base = aux->tmem_base;
    volatile int* abort_flag = &aux->abort_flag;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer (one thread per CTA)
        if (lane == 0) {
            tma_prefetch_desc(&tm_a);
            tma_prefetch_desc(&tm_w);
            const uint32_t tx = (uint32_t)(2 * (BM + nt / 2) * BK);              // both CTAs' bytes
            int stage = 0;
            uint32_t phase = 0;
            bool ok = !(flags & 2);                              // failure injection from the host: nothing is requested
            for (int t = pair; t < num_tiles && ok; t += npairs) {
                const int m0 = tile_m(t) + (int)rank * (nt / 2), n0 = tile_n(t) + (int)rank * BM;
                for (int kb = 0; kb < KB; ++kb) {
                    if (!mbar_wait(smem_u32(&aux->empty[stage]), phase ^ 1, abort_flag, 0x1900 + stage)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = map_to_cta(smem_u32(&aux->full[stage]), 0);
                    if (leader) mbar_expect_tx(smem_u32(&aux->full[stage]), tx);
                    uint8_t* st = smem + stage * TP_STAGE_BYTES;
                    tma_load_2d_pair(smem_u32(st), &tm_w, kb * BK, n0, bar);
                    tma_load_2d_pair(smem_u32(st + BM * BK), &tm_a, kb * BK, m0, bar);
                    if (++stage == TP_STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {
                unsigned long long t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 2000000ull) {
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (the leader's one thread)
        if (leader && elect_one()) {
            const uint32_t idesc = umma_idesc_i8(2 * BM, nt);
            int stage = 0, buf = 0;
            uint32_t phase = 0, bphase = 0;
            bool ok = true, ready = false;
            for (int t = pair; t < num_tiles && ok; t += npairs) {
                if (!mbar_wait(smem_u32(&aux->tempty[buf]), bphase ^ 1, abort_flag, 0x1A00 + buf)) break;
                tc_fence_after();
                const uint32_t d = tmem_base + buf * TP_MAX;
                for (int kb = 0; kb < KB; ++kb) {
                    if (!ready && !mbar_wait(smem_u32(&aux->full[stage]), phase, abort_flag, 0x1B00 + stage)) {
                        ok = false;
                        break;
                    }
                    const int nstage = stage + 1 == TP_STAGES ? 0 : stage + 1;
                    const uint32_t nphase = nstage == 0 ? phase ^ 1 : phase;
                    ready = mbar_peek(smem_u32(&aux->full[nstage]), nphase);      // asked now, answered while this stage is issued
                    tc_fence_after();
                    uint8_t* st = smem + stage * TP_STAGE_BYTES;
                    const uint64_t wd = umma_desc_k128(smem_u32(st));
                    const uint64_t xd = umma_desc_k128(smem_u32(st + BM * BK));
#pragma unroll
                    for (int k = 0; k < BK / 32; ++k)
                        umma_i8_pair(d, umma_desc_advance(wd, k * 32), umma_desc_advance(xd, k * 32), idesc, (kb | k) ? 1u : 0u);
                    const uint32_t eb = smem_u32(&aux->empty[stage]);
                    tc_commit_pair(eb);                           // this CTA's producer may refill the stage ...
                    tc_commit_pair(map_to_cta(eb, 1));            // ... and the peer's
                    stage = nstage;
                    phase = nphase;
                }
                if (!ok) break;
                const uint32_t fb = smem_u32(&aux->tfull[buf]);
                tc_commit_pair(fb);
                tc_commit_pair(map_to_cta(fb, 1));
                buf ^= 1;
                if (buf == 0) bphase ^= 1;
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: 8 warps, two per lane quarter, half of the
        // columns each; a lane holds one output column, so a warp's store of a row is 32 neighbouring columns
        const int q = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
        int buf = 0;
        uint32_t bphase = 0;
        for (int t = pair; t < num_tiles; t += npairs) {
            const int m0 = tile_m(t), n = tile_n(t) + (int)rank * BM + q * 32 + lane;
            float* sab = sa_stash + buf * TP_MAX;
            for (int i = et; i < nt; i += 256) sab[i] = m0 + i < live ? a_s[m0 + i] : 0.0f;
            const float sw = n < N ? w_s[n] : 0.0f;
            const int c1 = (half + 1) * (nt / 2);                        // nt / 2: a multiple of 16
            float h0[16], h1[16];
            auto fetch = [&](int c0, float (&h)[16]) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c0 < c1 && m0 + c0 + j < live && n < N) h[j] = __ldcg((const float*)out + (long)(m0 + c0 + j) * ldo + n);
            };
            if (REGS) fetch(half * (nt / 2), h0);
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (!mbar_wait(smem_u32(&aux->tfull[buf]), bphase, abort_flag, 0x1C00 + buf)) break;
            tc_fence_after();
            const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * TP_MAX;
            auto rows8 = [&](int c0, const float* h) {
                uint32_t r[8];
                tmem_ld8(lane_addr + c0, r);
                const float4 s0 = *(const float4*)(sab + c0), s1 = *(const float4*)(sab + c0 + 4);
                const float sa[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                tmem_ld_wait();
                if (n < N) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (m0 + c0 + j >= live) continue;
                        const float v = scale2((int)r[j], sa[j], sw);
                        const long at = (long)(m0 + c0 + j) * ldo + n;
                        if (EPI == EPI_ADD && REGS) ((float*)out)[at] = __fadd_rn(h[j], v);
                        else if (EPI == EPI_ADD) atomicAdd((float*)out + at, v);
                        else ((__nv_bfloat16*)out)[at] = __float2bfloat16_rn(v);
                    }
                }
            };
            if (REGS) {
#pragma unroll 1
                for (int c0 = half * (nt / 2); c0 < c1 && m0 + c0 < live; c0 += 32) {
                    fetch(c0 + 16, h1);
                    rows8(c0, h0);
                    rows8(c0 + 8, h0 + 8);
                    fetch(c0 + 32, h0);
                    if (c0 + 16 < c1) {
                        rows8(c0 + 16, h1);
                        rows8(c0 + 24, h1 + 8);
                    }
                }
            } else {
#pragma unroll 1
                for (int c0 = half * (nt / 2); c0 < c1 && m0 + c0 < live; c0 += 8) rows8(c0, nullptr);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&aux->tempty[buf]), 0));
            buf ^= 1;
            if (buf == 0) bphase ^= 1;
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                            // no CTA leaves while its peer may still signal it
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

}  // namespace w8a8
