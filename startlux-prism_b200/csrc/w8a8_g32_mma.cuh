// W8A8 with one scale per 32 inputs on both operands with mma.sync (mma_sync.cuh says why not tcgen05 here):
// out[m, n] = sum over groups g, in ascending order, of mul_rn(mul_rn(float(sum_g), a_s[m, g]), w_s[n, g])
// (kernels/w8a8.py:31-98 with GK = 32); for the vocabulary head, whose reference kernel leaves the roundings to its
// compiler (kernels/decode.py:157), acc = fma_rn(mul_rn(float(sum_g), a_s), w_s, acc).
//
// A group is one m16n8k32 per 16 weight rows x 8 activation rows, and its int32 sums appear in the registers of the warp
// that owns the output elements' fp32 chain.  The MMA's accumulator input is the bit pattern of 1.5 * 2^23, so that the
// sums (below 2^19) come out as floats biased by that constant: no conversion.  Per tile and group that leaves six packed
// fp32 instructions and four scalar adds (the head: six packed ones) beside one MMA: 16 (12) cycles of the fp32 pipe
// against 8 of the tensor pipe.  A warp takes 16 * NT weight rows x 8 * MT activation rows over the whole of K (the chain is
// serial), a CTA WN x WM such warps on one ring of ST stages of KQ * 128 bytes of K, filled by cp.async and XOR-swizzled for
// ldmatrix; the activation scales are staged as row pairs, so that one 16-byte read serves two groups of NT tiles.
// What bounds it: at NT = 1 with many rows shared-memory reads (ncu of a first version: 67 % of the wavefronts), hence NT = 2; there
// the chain's fp32 pipe at many rows (500 rows: 55 % busy, issue slots 52 %, shared memory 49 %), at 48 rows the latencies of
// the chain with two warps per scheduler (fp32 pipe 41 %, DRAM 34 %), and below 17 rows those of one warp per scheduler.
// Measured against the tcgen05 kernel that ran all of these before (us, one launch):
//   5120 x 5120   8 rows 12.8 -> 11.0   16 rows 14.6 -> 12.5   64 rows 29.5 -> 25.6   256 rows 84.6 -> 56.6
//   7168 x 5120   500 rows 189 -> 141   1000 rows 337 -> 258;   34816 x 5120   256 rows 421 -> 317
//   head, 248320 x 5120   16 rows 245 -> 225   30 rows 366 -> 282   48 rows 626 -> 379   64 rows 697 -> 512
#pragma once
#include "mma_sync.cuh"
#include "w8a8_g32.cuh"

namespace w8a8 {

template <int MT_, int NT_, int WN_, int WM_, int KQ_, int ST_>
struct G32Mma {
    static constexpr int MT = MT_, NT = NT_, WN = WN_, WM = WM_, KQ = KQ_, ST = ST_;
    static constexpr int ROWS = 16 * NT * WN, MP = 8 * MT, MC = MP * WM, THREADS = 32 * WN * WM;
    static constexpr int OFF_X = ROWS * 128, OFF_SW = OFF_X + MC * 128, OFF_SA = OFF_SW + ROWS * 16;
    static constexpr int SUB = OFF_SA + MC * 16;                  // one 128-byte piece of K with its scales
    static constexpr int SMEM = ST * KQ * SUB;
};

template <int MT, int NT, int WN, int WM, int KQ, int ST, bool FUSE>
__global__ void __launch_bounds__(32 * WN * WM)
w8a8_g32_mma_kernel(const int8_t* __restrict__ a, const int8_t* __restrict__ w, const SwapArgs p) {
    using C = G32Mma<MT, NT, WN, WM, KQ, ST>;
    constexpr int T = C::THREADS;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int wn = warp % WN, wm = warp / WN;
    const int g = lane >> 2, t4 = lane & 3, lr = lane & 7, lm = lane >> 3;
    if (p.pdl) pdl_trigger();
    int live = *p.n_rows;
    live = live < p.M ? live : p.M;
    const int mblocks = (p.M + C::MC - 1) / C::MC;                // the row blocks of a weight tile are neighbours: L2
    const int m0 = (int)(blockIdx.x % mblocks) * C::MC;
    if (m0 >= live) return;
    const long n0 = (long)(blockIdx.x / mblocks) * C::ROWS;
    const int KC = p.K / 128, G = p.K / 32;
    const int nrows = p.N - n0 < C::ROWS ? (int)(p.N - n0) : C::ROWS, mrows = p.M - m0;

    // ---- this thread's share of a 128-byte piece of K: 16-byte chunks of weight and activation rows (rows past N or M are
    // left as they are: an output depends on its own two rows only, and theirs are not stored), scales
    constexpr int STEP = T / 8;                                   // rows per copy instruction of the CTA
    const int r0 = tid >> 3, c0 = tid & 7;
    const uint32_t d0 = r0 * 128 + ((c0 ^ (r0 & 7)) << 4);
    const int8_t* wsrc = w + (n0 + r0) * p.K + c0 * 16;
    const int8_t* xsrc = a + (long)(m0 + r0) * p.K + c0 * 16;
    const float* swsrc = p.w_s + (n0 + tid) * G;
    const float* sasrc = p.a_s + (long)(m0 + (tid >> 2)) * G + (tid & 3);
    auto load_w = [&](int kc, uint32_t sb) {
#pragma unroll
        for (int i = 0; i < C::ROWS / STEP; ++i)
            if (r0 + i * STEP < nrows)
                cp_async16(sb + (d0 ^ (((i * STEP) & 7) << 4)) + i * STEP * 128, wsrc + (long)i * STEP * p.K + kc * 128);
    };
    auto load_x = [&](int kc, uint32_t sb) {                      // activations and both operands' scales
#pragma unroll
        for (int i = 0; i < (C::ROWS + T - 1) / T; ++i)
            if (tid + i * T < nrows) cp_async16(sb + C::OFF_SW + (tid + i * T) * 16, swsrc + (long)i * T * G + kc * 4);
#pragma unroll
        for (int i = 0; i < (C::MC + STEP - 1) / STEP; ++i) {
            const int m = r0 + i * STEP;
            if (m < C::MC && m < mrows)
                cp_async16(sb + C::OFF_X + (d0 ^ (((i * STEP) & 7) << 4)) + i * STEP * 128, xsrc + (long)i * STEP * p.K + kc * 128);
        }
#pragma unroll
        for (int i = 0; i < (C::MC * 4 + T - 1) / T; ++i) {       // activation scales as row pairs: [MC / 2][4 groups][2]
            const int m = (tid >> 2) + i * (T / 4);
            if (m < C::MC && m < mrows)
                cp_async4(sb + C::OFF_SA + (m >> 1) * 32 + (tid & 3) * 8 + (m & 1) * 4, sasrc + (long)i * (T / 4) * G + kc * 4);
        }
    };

    f32x2 acc[NT][MT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j) acc[i][j][0] = acc[i][j][1] = pack2(0.0f, 0.0f);
    const f32x2 unbias = pack2(-12582912.0f, -12582912.0f);
    const int R = (KC + KQ - 1) / KQ;

    // a programmatic dependent requests its first int8 weights, and nothing else, before it waits for the kernel before it:
    // that one may write the activations and the scales of either operand
#pragma unroll
    for (int s = 0; s < ST - 1; ++s)
#pragma unroll
        for (int q = 0; q < KQ; ++q)
            if (s * KQ + q < KC) load_w(s * KQ + q, sbase + (s * KQ + q) * C::SUB);
    if (p.pdl) pdl_wait();
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
#pragma unroll
        for (int q = 0; q < KQ; ++q)
            if (s * KQ + q < KC) load_x(s * KQ + q, sbase + (s * KQ + q) * C::SUB);
        cp_async_commit();
    }
    int slot = 0, fill = ST - 1;
    for (int r = 0; r < R; ++r) {
        cp_async_wait<ST - 2>();
        __syncthreads();
#pragma unroll
        for (int q = 0; q < KQ; ++q) {
            const int kc = (r + ST - 1) * KQ + q;
            if (kc < KC) {
                load_w(kc, sbase + (fill * KQ + q) * C::SUB);
                load_x(kc, sbase + (fill * KQ + q) * C::SUB);
            }
        }
        cp_async_commit();
        if (++fill == ST) fill = 0;
#pragma unroll
        for (int q = 0; q < KQ; ++q) {
            if (r * KQ + q >= KC) break;
            const uint32_t sb = sbase + (slot * KQ + q) * C::SUB;
            const uint8_t* sp = smem + (slot * KQ + q) * C::SUB;
            const int wrow = wn * 16 * NT;
            float sw[NT][2][4];
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float4 v = *(const float4*)(sp + C::OFF_SW + (wrow + i * 16 + e * 8 + g) * 16);
                    sw[i][e][0] = v.x, sw[i][e][1] = v.y, sw[i][e][2] = v.z, sw[i][e][3] = v.w;
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) {                         // two groups at a time
                uint32_t wr[NT][2][4];
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        ldmatrix_x4(wr[i][u], sb + (wrow + i * 16 + (lm & 1) * 8 + lr) * 128 +
                                                  (((4 * h + 2 * u + (lm >> 1)) ^ lr) << 4));
#pragma unroll
                for (int j = 0; j < MT; ++j) {
                    uint32_t x[4];
                    ldmatrix_x4(x, sb + C::OFF_X + (wm * C::MP + j * 8 + lr) * 128 + (((4 * h + lm) ^ lr) << 4));
                    const float4 s4 = *(const float4*)(sp + C::OFF_SA + ((wm * C::MP + j * 8) / 2 + t4) * 32 + h * 16);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const f32x2 sa = u ? pack2(s4.z, s4.w) : pack2(s4.x, s4.y);
#pragma unroll
                        for (int i = 0; i < NT; ++i) {
                            int d[4];
                            mma_s8_k32(d, wr[i][u][0], wr[i][u][1], wr[i][u][2], wr[i][u][3], x[2 * u], x[2 * u + 1], 0x4B400000);
                            const float wa = sw[i][0][2 * h + u], wb = sw[i][1][2 * h + u];
                            const f32x2 f0 = mul2(add2(pack2(__int_as_float(d[0]), __int_as_float(d[1])), unbias), sa);
                            const f32x2 f1 = mul2(add2(pack2(__int_as_float(d[2]), __int_as_float(d[3])), unbias), sa);
                            f32x2(&c)[2] = acc[i][j];
                            if (FUSE) {
                                c[0] = fma2(f0, pack2(wa, wa), c[0]);
                                c[1] = fma2(f1, pack2(wb, wb), c[1]);
                            } else {
                                // scalar adds: the assembler contracts a packed multiply and a packed add into one fma
                                const float2 p0 = unpack2(mul2(f0, pack2(wa, wa))), p1 = unpack2(mul2(f1, pack2(wb, wb)));
                                const float2 a0 = unpack2(c[0]), a1 = unpack2(c[1]);
                                c[0] = pack2(__fadd_rn(a0.x, p0.x), __fadd_rn(a0.y, p0.y));
                                c[1] = pack2(__fadd_rn(a1.x, p1.x), __fadd_rn(a1.y, p1.y));
                            }
                        }
                    }
                }
            }
        }
        if (++slot == ST) slot = 0;
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < MT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int rl = wn * 16 * NT + i * 16 + h * 8 + g;
                const float2 v = unpack2(acc[i][j][h]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int m = m0 + wm * C::MP + j * 8 + 2 * t4 + e;
                    if (rl < nrows && m < live) {
                        const long at = (long)m * p.ldo + n0 + rl;
                        const float f = e ? v.y : v.x;
                        if (p.epi == EPI_BF16) ((__nv_bfloat16*)p.out)[at] = __float2bfloat16_rn(f);
                        else if (p.epi == EPI_F32) ((float*)p.out)[at] = f;
                        else ((float*)p.out)[at] = __fadd_rn(((float*)p.out)[at], f);
                    }
                }
            }
}

}  // namespace w8a8
