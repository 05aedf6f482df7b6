// MXFP4 for a decode batch (up to 64 activation rows): the operands of mxfp4_gemm_kernel exchanged.  The weight tile (128 rows)
// is the MMA's M operand, so a tensor-memory lane holds an output column, and the activation rows, rounded up to 16, are its
// N: an MMA takes a fraction of the 64 cycles that 128 x 128 take, no activation row is padding in shared memory beyond
// the next 16, and a CTA needs few columns and stages, so two share an SM.  One accumulator over all of K in ascending
// order, as in the other kernels: the same bits.
// What bound the 128 x 128 kernel here was its issuing thread: nine asynchronous instructions and a barrier test per 256 inputs
// took it about 1,100 cycles, and 40 tiles of 68 such blocks are a chain.  Issued by an elected thread, with the test of the next
// block's barrier asked before this block's instructions, a block takes about 500; what is left is that chain.
// The activation scales are read as the quantizer wrote them (row-major) and placed in the tensor core's order by a warp
// of their own: no launch in front of the GEMM.
// `parts` CTAs share a 128-row weight tile when the tiles alone would leave SMs idle: each brings its 128 / parts rows to their
// places in the operand (the other lanes multiply whatever is there and are not read).
// One launch with the scales' tiling, us, 128 x 128 kernel -> this one: 7168 x 5120 16 rows 15.4 -> 8.5, 64 rows 17.9 -> 11.0;
// 5120 x 5120 16.1 -> 8.9, 18.0 -> 10.8; 34816 x 5120 31.2 -> 17.9, 28.4 -> 20.6; 5120 x 17408 36.4 -> 20.2, 38.1 -> 22.5.
#pragma once
#include "mma_sync.cuh"
#include "mxfp4_gemm.cuh"

namespace mxfp4 {

constexpr int FEW_ROWS = 64;
constexpr int FEW_X_BYTES = FEW_ROWS * KB_BYTES;
constexpr int FEW_STAGE_BYTES = A_BYTES + FEW_X_BYTES + 2 * SF_BYTES;    // weights | activations | weight scales | activation scales
constexpr int FEW_AHEAD = 2;                                             // activation scales requested this many stages ahead
template <int ST>
constexpr int few_smem() { return ST * FEW_STAGE_BYTES + 1024 + 256; }

struct FewArgs {
    const uint8_t* as;      // activation scales [M, K/32]
    const uint8_t* sfw;     // tiled weight scales
    void* out;
    long ldo;
    int M, N, K, epi, xbox, parts;
};

template <int ST>
__global__ void __launch_bounds__(224)
mxfp4_few_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const FewArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    AuxM* aux = (AuxM*)(smem + ST * FEW_STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KB = p.K / 256, KA = p.K / 128;
    const int nt = blockIdx.x / p.parts, rows = 128 / p.parts, r0 = (blockIdx.x % p.parts) * rows;   // this CTA's rows of the tile
    const int cols = (p.M + 15) & ~15;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(smem_u32(&aux->full[s]), 2);                        // the copies' bytes, the activation scales
            mbar_init(smem_u32(&aux->empty[s]), 1);
        }
        mbar_init(smem_u32(&aux->tfull[0]), 1);
        aux->abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&aux->tmem_base), 128);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = aux->tmem_base;
    volatile int* abort_flag = &aux->abort_flag;

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            const uint32_t tx = (uint32_t)(rows * KB_BYTES + p.xbox * KB_BYTES + SF_BYTES);
            for (int kb = 0; kb < KB; ++kb) {
                if (!mbar_wait(smem_u32(&aux->empty[stage]), phase ^ 1, abort_flag, 0x1800 + stage)) {
                    ok = false;
                    break;
                }
                const uint32_t bar = smem_u32(&aux->full[stage]);
                mbar_expect_tx(bar, tx);
                const uint32_t st = smem_u32(smem + stage * FEW_STAGE_BYTES);
                tma_load_2d(st + r0 * KB_BYTES, &tm_w, kb * KB_BYTES, nt * 128 + r0, bar);
                bulk_load(st + A_BYTES + FEW_X_BYTES, p.sfw + ((long)nt * KA + kb * 2) * 512, SF_BYTES, bar);
                tma_load_2d(st + A_BYTES, &tm_x, kb * KB_BYTES, 0, bar);
                if (++stage == ST) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (!ok) {                                                   // let armed copies land before the CTA can exit
                unsigned long long t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 2000000ull) {
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ready = false, ok = true;
            const uint32_t d = tmem_base;
            for (int kb = 0; kb < KB; ++kb) {
                if (!ready && !mbar_wait(smem_u32(&aux->full[stage]), phase, abort_flag, 0x1810 + stage)) {
                    ok = false;
                    break;
                }
                const int nstage = stage + 1 == ST ? 0 : stage + 1;
                const uint32_t nphase = nstage == 0 ? phase ^ 1 : phase;
                ready = mbar_peek(smem_u32(&aux->full[nstage]), nphase); // asked now, answered while this block is issued
                tc_fence_after();
                const uint32_t st = smem_u32(smem + stage * FEW_STAGE_BYTES);
                const uint32_t sf = st + A_BYTES + FEW_X_BYTES;
                const uint32_t sfw_t = tmem_base + FEW_ROWS + (kb & 1) * 16, sfx_t = sfw_t + 8;
                tmem_cp_sf(sfw_t, sf);
                tmem_cp_sf(sfx_t, sf + SF_BYTES);
                tmem_cp_sf(sfw_t + 4, sf + 512);
                tmem_cp_sf(sfx_t + 4, sf + SF_BYTES + 512);
                const uint64_t ad = umma_desc_k128(st), bd = umma_desc_k128(st + A_BYTES);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t sf_id = (k & 1) * 2;
                    umma_mxf4(d, umma_desc_advance(ad, k * 32), umma_desc_advance(bd, k * 32), idesc_mxf4(128, cols, sf_id, sf_id),
                              sfw_t + (k >> 1) * 4, sfx_t + (k >> 1) * 4, (kb | k) ? 1u : 0u);
                }
                tc_commit(smem_u32(&aux->empty[stage]));
                stage = nstage;
                phase = nphase;
            }
            if (ok) tc_commit(smem_u32(&aux->tfull[0]));
        }
    } else if (warp == 2) {
        // activation scales: four neighbouring scales of a row are one word of a 512-byte block (32 x 16 bytes)
        for (int kb = 0; kb < KB + FEW_AHEAD; ++kb) {
            if (kb < KB) {
                const int stage = kb % ST;
                if (!mbar_wait(smem_u32(&aux->empty[stage]), ((kb / ST) & 1) ^ 1, abort_flag, 0x1820 + stage)) break;
                const uint32_t dst = smem_u32(smem + stage * FEW_STAGE_BYTES) + A_BYTES + FEW_X_BYTES + SF_BYTES;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = (lane >> 1) + 16 * i, ka = lane & 1;
                    if (r < p.M) cp_async4(dst + ka * 512 + (r & 31) * 16 + (r >> 5) * 4, p.as + (long)r * (p.K >> 5) + kb * 8 + ka * 4);
                }
            }
            cp_async_commit();
            if (kb >= FEW_AHEAD) {
                cp_async_wait<FEW_AHEAD>();
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&aux->full[(kb - FEW_AHEAD) % ST]));
            }
        }
        cp_async_wait<0>();
    } else {
        const int q = warp & 3;
        const int n = nt * 128 + q * 32 + lane;
        const bool mine = q * 32 >= r0 && q * 32 < r0 + rows;
        if (mine && mbar_wait(smem_u32(&aux->tfull[0]), 0, abort_flag, 0x1830)) {
            tc_fence_after();
            const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < p.M; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(lane_addr + c0, r);
                tmem_ld_wait();
                if (n < p.N) {
                    if (p.epi == 0) {
                        __nv_bfloat16* o = (__nv_bfloat16*)p.out + n;
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c0 + j < p.M) o[(long)(c0 + j) * p.ldo] = __float2bfloat16_rn(__uint_as_float(r[j]));
                    } else {
                        float* o = (float*)p.out + n;
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c0 + j < p.M) v[j] = __ldcg(o + (long)(c0 + j) * p.ldo);
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c0 + j < p.M) o[(long)(c0 + j) * p.ldo] = __fadd_rn(v[j], __uint_as_float(r[j]));
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 128);
}

}  // namespace mxfp4
