// W4A8 for a decode batch: up to a few dozen activation rows against Q4_K / Q6_K weights with mma.sync
// (mma_sync.cuh says why not tcgen05 here).  The arithmetic is that of the other W4A8 kernels (w4a8_gemm.cuh): exact integers inside a
// 256-input super-block, one fp32 step per super-block, super-blocks in order - the same bits for every shape.
//
// A warp takes 16 * NT weight rows (the MMA's M) x 8 * MT activation rows (its N) of ONE super-block at a time:
//   Q4_K  a 32-input sub-block is one m16n8k32 per tile; a packed 32-bit word's low nibbles are operand register 0 and
//         its high nibbles register 2 (inputs t and t + 16 share a byte), so unpacking is an AND and a shift; the sums
//         are scaled by the 6-bit sub-block scale and added in int32 (4 IMADs: as long as the MMA itself);
//         the mins term is two k16 MMAs per super-block (mins against the low and the high parts of the group sums);
//   Q6_K  a 16-input sub-block is one m16n8k16, scaled by its int8 scale.
// The super-block's term t_b = d * float(acc) [- dmin * float(mins)] goes to shared memory; the CTA's WK warp groups
// work on WK consecutive super-blocks, and the threads then run the chain y = fma(a_b, t_b, y) over them in order,
// one round later (two term buffers, one barrier per round).  So K is split over warps without a change of bits, and
// a 5120-row Q4_K projection is 320 CTAs of 16 rows (Q6_K: 80 to 160 of 64 or 32).
// Operands come through a ring of ST rounds by cp.async (16 bytes a lane, rows of 128 bytes whole), XOR-swizzled so
// that every ldmatrix is free of bank conflicts; the WN warps of a super-block share its activations.
//
// What bounds it: instruction issue, with too few warps to fill the slots (ncu, Q4_K at 12 rows: 34816 x 5120 54 % of them, DRAM
// 45 %, two CTAs of four warps per SM, fixed latencies the first stall; 6144 x 5120 45 %, the ring's copies the first stall).
// Measured, one launch with weights from HBM, before (tcgen05 with the sums through tensor memory; dp4a up to eight rows)
// and after:
//   Q4_K  6144 x 5120   8 rows 18.2 ->  7.1 us   12 rows 17.2 ->  9.1    32 rows 21.9 -> 15.4
//         34816 x 5120  8 rows 37.3 -> 21.4      12 rows 42.4 -> 27.6    32 rows 81.6 -> 46.4
//   Q6_K  5120 x 17408  8 rows 45.0 -> 24.0      12 rows 72.5 -> 33.5    32 rows 142.5 -> 56.9
#pragma once
#include "mma_sync.cuh"
#include "w4a8_gemm.cuh"

namespace w4a8 {

template <int KIND, int MT_, int NT_, int WN_, int WK_, int ST_>
struct MmaCfg {
    static constexpr int MT = MT_, NT = NT_, WN = WN_, WK = WK_, ST = ST_;
    static constexpr int MP = 8 * MT, WROWS = 16 * NT, ROWS = WROWS * WN, THREADS = 32 * WN * WK;
    static constexpr int WB = KIND == KIND_Q4K ? 128 : 256;              // weight bytes per row and super-block
    static constexpr int SCB = KIND == KIND_Q4K ? 8 : 16;                // sub-block scale bytes
    static constexpr int OFF_X = ROWS * WB;
    static constexpr int OFF_SC = OFF_X + MP * 256;
    static constexpr int OFF_MN = OFF_SC + ROWS * SCB;
    static constexpr int OFF_D = OFF_MN + (KIND == KIND_Q4K ? ROWS * 8 : 0);
    static constexpr int OFF_DM = OFF_D + ROWS * 4;
    static constexpr int OFF_XS = OFF_DM + (KIND == KIND_Q4K ? ROWS * 4 : 0);
    static constexpr int SB_BYTES = OFF_XS + (KIND == KIND_Q4K ? MP * 16 : 0);   // one super-block of one round
    static constexpr int TS = ROWS + 4;                                  // row stride of the term buffer in floats
    static constexpr int OFF_TERMS = ST * WK * SB_BYTES;
    static constexpr int OFF_A = OFF_TERMS + 2 * WK * MP * TS * 4;
    static constexpr int SMEM = OFF_A + (ST + 1) * WK * MP * 4;          // the chain reads a round's scales a round later
    static constexpr int E = ROWS * MP / THREADS;                        // chain elements per thread
    static_assert(E * THREADS == ROWS * MP && SB_BYTES % 16 == 0, "whole elements per thread");
};

// Byte i of w, sign-extended (one byte permute: the upper result bytes replicate the byte's sign).
__device__ __forceinline__ int byte_signed(uint32_t w, int i) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "r"(0x8880 + 0x1111 * i));
    return (int)r;
}

template <int KIND, int MT, int NT, int WN, int WK, int ST>
__global__ void __launch_bounds__(32 * WN * WK)
w4a8_mma_kernel(const GemvArgs p) {
    using C = MmaCfg<KIND, MT, NT, WN, WK, ST>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wn = warp % WN, wk = warp / WN;
    const int g = lane >> 2, t4 = lane & 3;
    int live = *p.n_rows;
    live = live < p.M ? live : p.M;
    const int mblocks = (p.M + C::MP - 1) / C::MP;                       // the row blocks of a weight tile are neighbours: L2
    const int m0 = (int)(blockIdx.x % mblocks) * C::MP;
    if (m0 >= live) return;
    const long n0 = (long)(blockIdx.x / mblocks) * C::ROWS;
    const int NSB = p.K / 256;
    const int R = (NSB + WK - 1) / WK;

    // ---- copies of this warp's group for the next round into ring slot `slot`; rows past N or M are left as they are (an
    // output depends on its own weight row and activation row only, and theirs are not stored)
    const long wrow0 = n0 + wn * C::WROWS;
    const int nrows = p.N - wrow0 > C::WROWS ? C::WROWS : (int)(p.N - wrow0);   // this warp's weight rows (may be <= 0)
    const int mrows = p.M - m0;
    constexpr int CPR = C::WB / 16, WR = 32 / CPR;                       // chunks per weight row, rows per copy instruction
    const long wpitch = (long)(p.K / 256) * C::WB, wstep = wpitch * WR;
    const int wr = lane / CPR, wc = lane % CPR;
    const uint8_t* wsrc = p.wq + (wrow0 + wr) * wpitch + (long)wk * C::WB + wc * 16;
    const uint32_t wdst = (wn * C::WROWS + wr) * C::WB + (((wc & 7) ^ wr) | (wc & 8)) * 16;
    const int xm = wn * 2 + (lane >> 4), xc = lane & 15;                 // rows xm, xm + 2 WN, ...
    const int8_t* xsrc = p.xq + (long)(m0 + xm) * p.K + (long)wk * 256 + xc * 16;
    const long xstep = (long)p.K * (2 * WN);
    const uint32_t xdst = C::OFF_X + xm * 256 + (((xc & 7) ^ (xm & 7)) | (xc & 8)) * 16;
    // scales: 16-byte pieces of the warp's rows (N is a multiple of four: a piece is all inside or all outside)
    constexpr int SCN = KIND == KIND_Q4K ? 24 * NT : 20 * NT, SCI = (SCN + 31) / 32;
    const uint8_t* ssrc[SCI];
    long sstep[SCI];
    uint32_t sdst[SCI];
    bool sok[SCI];
#pragma unroll
    for (int i = 0; i < SCI; ++i) {
        const int id = lane + 32 * i;
        if (KIND == KIND_Q4K) {
            const int kind = id / (8 * NT), j = id - kind * 8 * NT;      // 0 sc, 1 mn, 2 d | dm
            const int q = j >= 4 * NT, row = kind < 2 ? 2 * j : 4 * (j - q * 4 * NT);
            sok[i] = id < SCN && row < nrows;
            sstep[i] = (long)p.N * (kind < 2 ? 8 : 4);
            ssrc[i] = (kind < 2 ? (kind ? p.mn : p.sc) + (wrow0 + row) * 8
                                : (const uint8_t*)((q ? p.dm : p.d) + wrow0 + row)) + wk * sstep[i];
            sdst[i] = kind < 2 ? (kind ? C::OFF_MN : C::OFF_SC) + (wn * C::WROWS + row) * 8
                               : (q ? C::OFF_DM : C::OFF_D) + (wn * C::WROWS + row) * 4;
        } else {
            const int kind = id >= 16 * NT, row = kind ? 4 * (id - 16 * NT) : id;
            sok[i] = id < SCN && row < nrows;
            sstep[i] = (long)p.N * (kind ? 4 : 16);
            ssrc[i] = (kind ? (const uint8_t*)(p.d + wrow0 + row) : p.sc + (wrow0 + row) * 16) + wk * sstep[i];
            sdst[i] = kind ? C::OFF_D + (wn * C::WROWS + row) * 4 : C::OFF_SC + (wn * C::WROWS + row) * 16;
        }
    }
    constexpr int AI = (C::MP + 32 * WN - 1) / (32 * WN);
    const int am = wn * 32 + lane;                                       // activation row of this lane's scale and sums
    const float* asrc = p.a + (long)wk * p.Ma + m0 + am;
    const int8_t* gsrc = p.xs + ((long)wk * p.Ma + m0 + am) * 16;
    int bl = wk, slot = 0, aslot = 0;                                    // super-block, ring slot and scale slot of the next load
    auto load = [&]() {
        if (bl < NSB) {
            const uint32_t sb = sbase + (slot * WK + wk) * C::SB_BYTES;
#pragma unroll
            for (int i = 0; i < C::WROWS / WR; ++i)
                if (wr + i * WR < nrows) cp_async16(sb + (wdst ^ (((i * WR) & 7) << 4)) + i * (WR * C::WB), wsrc + i * wstep);
#pragma unroll
            for (int i = 0; i < (C::MP + 2 * WN - 1) / (2 * WN); ++i) {
                const int m = xm + i * 2 * WN;
                if (m < mrows && m < C::MP)
                    cp_async16(sb + (xdst ^ (((i * 2 * WN) & 7) << 4)) + i * (2 * WN * 256), xsrc + i * xstep);
            }
#pragma unroll
            for (int i = 0; i < SCI; ++i)
                if (sok[i]) cp_async16(sb + sdst[i], ssrc[i]);
#pragma unroll
            for (int i = 0; i < AI; ++i) {
                const int m = am + i * 32 * WN;
                if (m < C::MP && m < mrows) {
                    if (KIND == KIND_Q4K) cp_async16(sb + C::OFF_XS + m * 16, gsrc + i * 32 * WN * 16);
                    cp_async4(sbase + C::OFF_A + ((aslot * WK + wk) * C::MP + m) * 4, asrc + i * 32 * WN);
                }
            }
            wsrc += WK * C::WB;
            xsrc += WK * 256;
#pragma unroll
            for (int i = 0; i < SCI; ++i) ssrc[i] += WK * sstep[i];
            asrc += (long)WK * p.Ma;
            gsrc += (long)WK * p.Ma * 16;
        }
        bl += WK;
        if (++slot == ST) slot = 0;
        if (++aslot == ST + 1) aslot = 0;
        cp_async_commit();
    };

    float y[C::E];
#pragma unroll
    for (int e = 0; e < C::E; ++e) y[e] = 0.0f;
    float* terms = (float*)(smem + C::OFF_TERMS);
    // ---- the chain over round r's super-blocks: element e of a thread is (n, m) = (id % ROWS, id / ROWS)
    auto chain = [&](int r) {
        const float* tb = terms + (r & 1) * (WK * C::MP * C::TS);
        const float* as = (const float*)(smem + C::OFF_A) + (r % (ST + 1)) * (WK * C::MP);
#pragma unroll
        for (int kk = 0; kk < WK; ++kk) {
            if (r * WK + kk < NSB) {
#pragma unroll
                for (int e = 0; e < C::E; ++e) {
                    const int id = threadIdx.x + e * C::THREADS, n = id % C::ROWS, m = id / C::ROWS;
                    y[e] = __fmaf_rn(as[kk * C::MP + m], tb[(kk * C::MP + m) * C::TS + n], y[e]);
                }
            }
        }
    };

#pragma unroll
    for (int s = 0; s < ST - 1; ++s) load();
    for (int r = 0; r < R; ++r) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (r > 0) chain(r - 1);
        load();
        if (r * WK + wk < NSB) {
            const uint32_t sb = sbase + ((r % ST) * WK + wk) * C::SB_BYTES;
            const uint8_t* sp = smem + ((r % ST) * WK + wk) * C::SB_BYTES;
            const int lr = lane & 7, lm = lane >> 3;                     // ldmatrix: row and matrix this lane names
            int acc[NT][MT][4];
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < MT; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[i][j][c] = 0;
            float tt[NT][MT][4];
            if (KIND == KIND_Q4K) {
                uint2 sc[NT][2];
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        sc[i][h] = *(const uint2*)(sp + C::OFF_SC + (wn * C::WROWS + i * 16 + h * 8 + g) * 8);
#pragma unroll
                for (int jp = 0; jp < 4; ++jp) {                         // two sub-blocks of 32 inputs
                    uint32_t w[NT][4];                                   // rows g, g + 8 of sub-block 2 jp, then of 2 jp + 1
#pragma unroll
                    for (int i = 0; i < NT; ++i)
                        ldmatrix_x4(w[i], sb + (wn * C::WROWS + i * 16 + (lm & 1) * 8 + lr) * 128 +
                                              (((2 * jp + (lm >> 1)) ^ lr) << 4));
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        uint32_t x[4];                                   // 16-byte chunks 4 jp .. 4 jp + 3 of row j * 8 + g
                        const int c = 4 * jp + lm;
                        ldmatrix_x4(x, sb + C::OFF_X + (j * 8 + lr) * 256 + ((((c & 7) ^ lr) | (c & 8)) << 4));
#pragma unroll
                        for (int s = 0; s < 2; ++s)
#pragma unroll
                            for (int i = 0; i < NT; ++i) {
                                const uint32_t wa = w[i][2 * s], wb = w[i][2 * s + 1];
                                int d[4];
                                mma_s8_k32(d, wa & 0x0F0F0F0Fu, wb & 0x0F0F0F0Fu, (wa >> 4) & 0x0F0F0F0Fu,
                                           (wb >> 4) & 0x0F0F0F0Fu, x[2 * s], x[2 * s + 1], 0);
                                const int q = 2 * jp + s;
                                const int s0 = (int)__byte_perm(q < 4 ? sc[i][0].x : sc[i][0].y, 0, 0x4440 + (q & 3));
                                const int s1 = (int)__byte_perm(q < 4 ? sc[i][1].x : sc[i][1].y, 0, 0x4440 + (q & 3));
                                acc[i][j][0] += s0 * d[0];
                                acc[i][j][1] += s0 * d[1];
                                acc[i][j][2] += s1 * d[2];
                                acc[i][j][3] += s1 * d[3];
                            }
                    }
                }
                // mins against the group sums: k = 0..7 of a k16 step (operand words of threads 0 and 1 of a quad)
                const uint32_t keep = t4 < 2 ? 0xffffffffu : 0u;
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const int r0 = wn * C::WROWS + i * 16 + g;
                    const uint32_t ma = *(const uint32_t*)(sp + C::OFF_MN + r0 * 8 + (t4 & 1) * 4) & keep;
                    const uint32_t mb = *(const uint32_t*)(sp + C::OFF_MN + (r0 + 8) * 8 + (t4 & 1) * 4) & keep;
                    const float d0 = *(const float*)(sp + C::OFF_D + r0 * 4), d1 = *(const float*)(sp + C::OFF_D + r0 * 4 + 32);
                    const float e0 = -*(const float*)(sp + C::OFF_DM + r0 * 4), e1 = -*(const float*)(sp + C::OFF_DM + r0 * 4 + 32);
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        const uint8_t* xs = sp + C::OFF_XS + (j * 8 + g) * 16 + (t4 & 1) * 4;
                        int lo[4], hi[4];
                        mma_s8_k16(lo, ma, mb, *(const uint32_t*)xs);
                        mma_s8_k16(hi, ma, mb, *(const uint32_t*)(xs + 8));
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float v = __fmul_rn(c < 2 ? d0 : d1, __int2float_rn(acc[i][j][c]));
                            tt[i][j][c] = __fmaf_rn(c < 2 ? e0 : e1, __int2float_rn(lo[c] + 64 * hi[c]), v);
                        }
                    }
                }
            } else {
#pragma unroll
                for (int jq = 0; jq < 4; ++jq) {                         // four sub-blocks of 16 inputs
                    uint32_t w[NT][2][4];
                    uint32_t sc[NT][2];
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        const int r0 = wn * C::WROWS + i * 16;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int c = 4 * jq + 2 * u + (lm >> 1);
                            ldmatrix_x4(w[i][u], sb + (r0 + (lm & 1) * 8 + lr) * 256 + ((((c & 7) ^ lr) | (c & 8)) << 4));
                        }
                        sc[i][0] = *(const uint32_t*)(sp + C::OFF_SC + (r0 + g) * 16 + 4 * jq);
                        sc[i][1] = *(const uint32_t*)(sp + C::OFF_SC + (r0 + 8 + g) * 16 + 4 * jq);
                    }
#pragma unroll
                    for (int j = 0; j < MT; ++j) {
                        uint32_t x[4];
                        const int c = 4 * jq + lm;
                        ldmatrix_x4(x, sb + C::OFF_X + (j * 8 + lr) * 256 + ((((c & 7) ^ lr) | (c & 8)) << 4));
#pragma unroll
                        for (int s = 0; s < 4; ++s)
#pragma unroll
                            for (int i = 0; i < NT; ++i) {
                                int d[4];
                                mma_s8_k16(d, w[i][s >> 1][2 * (s & 1)], w[i][s >> 1][2 * (s & 1) + 1], x[s]);
                                const int s0 = byte_signed(sc[i][0], s), s1 = byte_signed(sc[i][1], s);
                                acc[i][j][0] += s0 * d[0];
                                acc[i][j][1] += s0 * d[1];
                                acc[i][j][2] += s1 * d[2];
                                acc[i][j][3] += s1 * d[3];
                            }
                    }
                }
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    const int r0 = wn * C::WROWS + i * 16 + g;
                    const float d0 = *(const float*)(sp + C::OFF_D + r0 * 4), d1 = *(const float*)(sp + C::OFF_D + r0 * 4 + 32);
#pragma unroll
                    for (int j = 0; j < MT; ++j)
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            tt[i][j][c] = __fmul_rn(c < 2 ? d0 : d1, __int2float_rn(acc[i][j][c]));
                }
            }
            float* tb = terms + ((r & 1) * WK + wk) * (C::MP * C::TS);
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < MT; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        tb[(j * 8 + 2 * t4 + (c & 1)) * C::TS + wn * C::WROWS + i * 16 + (c >> 1) * 8 + g] = tt[i][j][c];
        }
    }
    __syncthreads();
    chain(R - 1);
#pragma unroll
    for (int e = 0; e < C::E; ++e) {
        const int id = threadIdx.x + e * C::THREADS, m = m0 + id / C::ROWS;
        const long n = n0 + id % C::ROWS;
        if (n < p.N && m < live) {
            if (p.epi == 0) ((__nv_bfloat16*)p.out)[(long)m * p.ldo + n] = __float2bfloat16_rn(y[e]);
            else {
                float* o = (float*)p.out + (long)m * p.ldo + n;
                *o = __fadd_rn(*o, y[e]);
            }
        }
    }
}

}  // namespace w4a8
