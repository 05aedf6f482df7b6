// W4A8 GEMM on llama.cpp k-quant weights (Q4_K, Q6_K) with int8 activations scaled per 256 inputs, on the sm_100a
// tensor cores.  Arithmetic of the reference (kernels/w4a8.py:14-24), per 256-input super-block b in increasing b:
//   Q4_K  acc  = sum_g sc[n, g] * (xq . q)_g          mins = sum_g mn[n, g] * S[m, g]            (int32, exact)
//         t = d[n, b] * float(acc); t = fma(-dmin[n, b], float(mins), t); y = fma(a[m, b], t, y)
//   Q6_K  acc  = sum_h sc[n, h] * (xq . q)_h (16-input sub-blocks);  y = fma(a[m, b], d[n, b] * float(acc), y)
// then bf16(y) or out + y.
//
// The tensor core cannot scale per sub-block, so the integer scale is folded into the weights, as two int8 planes whose
// weighted sum is exact (the scheme of the reference's Hopper kernel, csrc/w4a8_wgmma.cu:4-16, 201-217):
//   Q4_K  sc = s0 + 8 s1 (3 bits each):   plane0 = s0 * q, plane1 = s1 * q  (0..105)                  acc = P0 + 8 P1
//   Q6_K  p = sc * q (13 bits signed):    plane0 = low byte of p as int8, plane1 = (p - plane0) >> 8  acc = P0 + 256 P1
// The expanded planes are the MMA's A operand and live in TENSOR memory: the threads that expand them write them with
// tcgen05.st, and shared memory carries the packed weights and the activations only.
// Q4_K's mins are one fp16 MMA of K = 16 per super-block: A = the 6-bit mins twice, B = the low and 64 x the high parts of the
// activation group sums.  Every product and partial sum is a whole number below 2^21: exact in its fp32 accumulator, which
// is float(mins) as it stands.
//
// One persistent CTA per SM, tiles of 128 weight rows (tensor-memory lanes) x up to HMAX units of NBU activation rows
// (accumulator columns); two accumulator sets alternate over the units, so the MMAs of one unit run while the
// epilogue warps drain the other, and the weights are expanded once for both units of a tile.
// Warps: 0 TMA producer, 1 MMA issuer, EXPW expanders, EPIW epilogue warps, both a quarter of them per tensor-memory lane quarter.
#pragma once
#include <cuda_fp16.h>

#include "mma_sync.cuh"

namespace w4a8 {

constexpr int KIND_Q4K = 0, KIND_Q6K = 1;
constexpr int TS_BM = 128;

template <int KIND>
struct TsCfg {
    static constexpr int NBU = 64, HMAX = 2;
    static constexpr bool Q4 = KIND == KIND_Q4K;
    static constexpr int XU_BYTES = 2 * NBU * 128;                       // one unit's activations: two 128-byte K halves
    static constexpr int WQ_BYTES = Q4 ? TS_BM * 128 : TS_BM * 256;
    static constexpr int XS_BYTES = Q4 ? HMAX * NBU * 16 : 0;
    static constexpr int SC_BYTES = Q4 ? TS_BM * 8 : TS_BM * 16;
    static constexpr int MN_BYTES = Q4 ? TS_BM * 8 : 0;
    static constexpr int OFF_WQ = HMAX * XU_BYTES;
    static constexpr int OFF_XS = OFF_WQ + WQ_BYTES;
    static constexpr int OFF_SC = OFF_XS + XS_BYTES;
    static constexpr int OFF_MN = OFF_SC + SC_BYTES;
    static constexpr int STAGE_BYTES = (OFF_MN + MN_BYTES + 1023) / 1024 * 1024;
    static constexpr int STAGES = 3;
    // four expander and eight epilogue warps: 128 registers a thread.  With eight and sixteen the expanders wait for most of their time
    // and the accumulators are read no sooner (34816 x 5120 at 2,048 rows 944 -> 1,148 us).
    static constexpr int EXPW = 4, EPIW = 8, CG = EPIW / 4;              // CG: column groups of a unit
    static_assert(16 % (8 * CG) == 0, "a warp's share of 16 rows is read eight columns at a time");
    static constexpr int EXP0 = 2, EPI0 = EXP0 + EXPW;
    static constexpr int THREADS = (EPI0 + EPIW) * 32;
    static constexpr int SETC = (Q4 ? 3 : 2) * NBU;                      // columns of an accumulator set: P0 | P1 (| mins)
    static constexpr int A_COL = 2 * SETC;                               // the expanded planes: ring of 64-column halves of a
    static constexpr int RING = A_COL + 256 <= 512 ? 4 : 2;              //   super-block (128 inputs of both planes each)
    static constexpr int MB = Q4 ? TS_BM * 32 : 0;                       // mins operand (fp16)
    static constexpr int SB16 = Q4 ? HMAX * NBU * 32 : 0;                // group sums (fp16)
    static constexpr int OFF_MB = STAGES * STAGE_BYTES;
    static constexpr int OFF_SUM = OFF_MB + 2 * MB;
    static constexpr int OFF_RING = OFF_SUM + 2 * SB16;                  // per epilogue warp: ring of scales,
    static constexpr int SLOTS = 4;                      //   32 d | 32 dmin | HMAX x AW a
    static constexpr int AW = NBU / CG;                                  // columns of a unit per epilogue warp
    static constexpr int SLOT_F = 64 + HMAX * AW;
    static constexpr int OFF_AUX = OFF_RING + EPIW * SLOTS * SLOT_F * 4;
    static constexpr int SMEM = OFF_AUX + 512 + 1024;
};

struct TsAux {
    uint64_t full[6], empty[6];
    uint64_t afull[4], aempty[4];
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
    int abort_flag;
};

struct TsMaps {
    CUtensorMap x, wq, xs, sc, mn;
};

struct TsArgs {
    const float* a;                    // activation scales fp32 [K/256, Ma]
    const float *d, *dm;               // weight scales fp32 [K/256, N]
    void* out;
    long ldo;
    const int* n_rows;
    int M, N, K, Ma, epi, xbox;        // xbox: activation rows of one TMA box (the unit, or fewer for fewer rows)
};

// K-major operand without swizzle: 8-row x 16-byte core matrices, `sbo` bytes between 8-row groups, `lbo` bytes
// between the two 16-byte K chunks of a 32-byte step.
__device__ __forceinline__ uint64_t umma_desc_plain(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ uint32_t swz(int row, int chunk) { return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4)); }

__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        : : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
            "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
            "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
            "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        : : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
            "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]^T, int8; and the fp16 product of two shared-memory operands.
__device__ __forceinline__ void umma_i8_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        : : "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        : : "r"(d), "l"(a), "l"(b), "r"(idesc) : "memory");
}
// fp16 A and B, fp32 accumulator
__device__ __forceinline__ uint32_t umma_idesc_f16(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Four signed bytes -> four halves, times `scale` (1 or 64): v + 128 under the exponent of 1024, minus 1152, all exact.
__device__ __forceinline__ uint2 halves_s8(uint32_t w, unsigned short scale) {
    w ^= 0x80808080u;
    const __half2 k = __half2half2(__ushort_as_half(0x6480)), s = __half2half2(__ushort_as_half(scale));
    const uint32_t lo = __byte_perm(w, 0x64646464u, 0x5140), hi = __byte_perm(w, 0x64646464u, 0x7362);
    const __half2 a = __hmul2(__hsub2(*(const __half2*)&lo, k), s), b = __hmul2(__hsub2(*(const __half2*)&hi, k), s);
    return make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}

// Q4_K: 32 packed inputs (low nibbles = inputs 0..15, high nibbles = 16..31) times the 6-bit sub-block scale s0 + 8 s1:
// r[0..7] plane 0, r[8..15] plane 1.  A byte holds at most 15 * 7 = 105: one 32-bit multiply scales four values.
__device__ __forceinline__ void ts_expand_q4(uint32_t* r, uint4 w, uint32_t sc) {
    const uint32_t s0 = sc & 7, s1 = sc >> 3;
    const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t lo = v[i] & 0x0F0F0F0Fu, hi = (v[i] >> 4) & 0x0F0F0F0Fu;
        r[i] = lo * s0;
        r[4 + i] = hi * s0;
        r[8 + i] = lo * s1;
        r[12 + i] = hi * s1;
    }
}

// Q6_K: four int8 values q (-32..31) of one sub-block -> the planes of p = sc * q.  u = q + 32 is unsigned; two of them
// sit in 16-bit fields and one multiply-add gives both p + 128 (kc holds 128 - 32 sc twice, and 0x8000 on the lower field
// so that it never borrows from the upper one).  The low byte is plane 0 + 128, the high byte plane 1 (the
// lower field's with its top bit flipped by the 0x8000): two byte gathers and two exclusive ors.
__device__ __forceinline__ void ts_split_q6(uint32_t w, uint32_t sc, uint32_t kc, uint32_t& lo, uint32_t& hi) {
    const uint32_t ue = (w ^ 0x00200020u) & 0x003F003Fu;
    const uint32_t uo = ((w >> 8) ^ 0x00200020u) & 0x003F003Fu;
    const uint32_t re = ue * sc + kc, ro = uo * sc + kc;
    lo = __byte_perm(re, ro, 0x6240) ^ 0x80808080u;
    hi = __byte_perm(re, ro, 0x7351) ^ 0x00008080u;
}

template <int KIND>
__global__ void __launch_bounds__(TsCfg<KIND>::THREADS, 1)
w4a8_ts_kernel(const __grid_constant__ TsMaps maps, const TsArgs p) {
    using C = TsCfg<KIND>;
    constexpr bool Q4 = C::Q4;
    constexpr int NBU = C::NBU, HMAX = C::HMAX;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    TsAux* aux = (TsAux*)(smem + C::OFF_AUX);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    int live = *p.n_rows;
    live = live < p.M ? live : p.M;
    const int num_m = live > 0 ? (live + NBU * HMAX - 1) / (NBU * HMAX) : 0;
    const int tiles = num_m * ((p.N + TS_BM - 1) / TS_BM);
    if ((int)blockIdx.x >= tiles) return;
    const int NSB = p.K / 256;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&aux->full[s]), 1);
            mbar_init(smem_u32(&aux->empty[s]), 1 + C::EXPW);            // MMA commit, expander warps
        }
        for (int i = 0; i < C::RING; ++i) {
            mbar_init(smem_u32(&aux->afull[i]), 4);                      // one expander warp of each lane quarter
            mbar_init(smem_u32(&aux->aempty[i]), 1);
        }
        for (int e = 0; e < 2; ++e) {
            mbar_init(smem_u32(&aux->acc_full[e]), 1);
            mbar_init(smem_u32(&aux->acc_empty[e]), C::EPIW);
        }
        aux->abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&aux->tmem_base), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = aux->tmem_base;
    volatile int* abort_flag = &aux->abort_flag;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const int m0 = (t % num_m) * (NBU * HMAX), n0 = (t / num_m) * TS_BM;
                const int hn = live - m0 > NBU ? 2 : 1;
                const uint32_t tx = (uint32_t)(hn * 256 * p.xbox + C::WQ_BYTES + (Q4 ? hn * NBU * 16 : 0) + C::SC_BYTES + C::MN_BYTES);
                for (int b = 0; b < NSB; ++b) {
                    if (!mbar_wait(smem_u32(&aux->empty[stage]), phase ^ 1, abort_flag, 0xA00 + stage)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&aux->full[stage]);
                    mbar_expect_tx(bar, tx);
                    const uint32_t st = smem_u32(smem + stage * C::STAGE_BYTES);
                    if (Q4) {
                        tma_load_2d(st + C::OFF_WQ, &maps.wq, b * 128, n0, bar);
                        tma_load_2d(st + C::OFF_SC, &maps.sc, n0 * 2, b, bar);
                        tma_load_2d(st + C::OFF_MN, &maps.mn, n0 * 2, b, bar);
                    } else {
                        tma_load_2d(st + C::OFF_WQ, &maps.wq, b * 256, n0, bar);
                        tma_load_2d(st + C::OFF_WQ + TS_BM * 128, &maps.wq, b * 256 + 128, n0, bar);
                        tma_load_2d(st + C::OFF_SC, &maps.sc, n0 * 4, b, bar);
                        tma_load_2d(st + C::OFF_SC + 1024, &maps.sc, n0 * 4 + 256, b, bar);
                    }
                    for (int h = 0; h < hn; ++h) {
                        const uint32_t xd = st + h * C::XU_BYTES;
                        tma_load_2d(xd, &maps.x, b * 256, m0 + h * NBU, bar);
                        tma_load_2d(xd + NBU * 128, &maps.x, b * 256 + 128, m0 + h * NBU, bar);
                        if (Q4) tma_load_2d(st + C::OFF_XS + h * NBU * 16, &maps.xs, (m0 + h * NBU) * 4, b, bar);
                    }
                    if (++stage == C::STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {                                       // let armed copies land before the CTA can exit
                unsigned long long t0 = global_timer_ns();
                while (global_timer_ns() - t0 < 2000000ull) {
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        // A barrier test takes about 200 cycles to answer: each is asked (without waiting) before
        // the MMAs of the half before, and waited for only where the answer was no.  The stage's own barrier is
        // not tested: the expanders passed it before they handed over the first half.
        if (elect_one()) {
            int stage = 0;
            unsigned sb = 0, u = 0;
            bool ok = true, ra = false, rc = false;                      // the coming half's operand, the coming unit's set
            auto slot_of = [&](unsigned b, int half) { return C::RING == 4 ? (int)(b & 1) * 2 + half : half; };
            auto aphase = [&](unsigned b) { return (C::RING == 4 ? b >> 1 : b) & 1; };
            auto full_a = [&](unsigned b, int half) { return smem_u32(&aux->afull[slot_of(b, half)]); };
            auto free_c = [&](unsigned v) { return smem_u32(&aux->acc_empty[v & 1]); };
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                const int m0 = (t % num_m) * (NBU * HMAX);
                const int hn = live - m0 > NBU ? 2 : 1;
                for (int b = 0; b < NSB && ok; ++b, ++sb) {
                    const uint32_t st = smem_u32(smem + stage * C::STAGE_BYTES);
                    const uint32_t st_empty = smem_u32(&aux->empty[stage]);
                    if (++stage == C::STAGES) stage = 0;
                    const uint32_t mins_a = smem_u32(smem + C::OFF_MB + (sb & 1) * C::MB);
                    const uint32_t mins_b = smem_u32(smem + C::OFF_SUM + (sb & 1) * C::SB16);
#pragma unroll
                    for (int h = 0; h < HMAX; ++h) {
                        if (h >= hn) break;
                        int cols = live - m0 - h * NBU;
                        cols = cols < NBU ? (cols + 15) & ~15 : NBU;
                        const uint32_t idesc = umma_idesc_i8(TS_BM, cols);
                        const uint32_t e = u & 1, d = tmem_base + e * C::SETC;
                        const bool last = h == hn - 1;
                        if (!rc && !mbar_wait(free_c(u), ((u >> 1) & 1) ^ 1, abort_flag, 0xB20 + e)) ok = false;
                        ++u;
#pragma unroll
                        for (int half = 0; half < 2; ++half) {
                            if (h == 0 && !ra && !mbar_wait(full_a(sb, half), aphase(sb), abort_flag, 0xB10 + half)) ok = false;
                            if (!ok) break;
                            // ask for what the next half and the next unit need
                            if (h == 0 && half == 0) ra = mbar_peek(full_a(sb, 1), aphase(sb));
                            if (half == 1) {
                                if (last) ra = mbar_peek(full_a(sb + 1, 0), aphase(sb + 1));
                                rc = mbar_peek(free_c(u), ((u >> 1) & 1) ^ 1);
                            }
                            tc_fence_after();
                            const int slot = slot_of(sb, half);
                            const uint32_t ac = tmem_base + C::A_COL + slot * 64;
                            const uint64_t xd = umma_desc_k128(st + h * C::XU_BYTES + half * (NBU * 128));
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint64_t bd = umma_desc_advance(xd, k * 32);
                                umma_i8_ts(d, ac + k * 16, bd, idesc, (half | k) ? 1u : 0u);
                                umma_i8_ts(d + NBU, ac + k * 16 + 8, bd, idesc, (half | k) ? 1u : 0u);
                            }
                            if (Q4 && half == 1)
                                umma_f16(d + 2 * NBU, umma_desc_plain(mins_a, TS_BM * 16, 128),
                                         umma_desc_plain(mins_b + h * (NBU * 32), NBU * 16, 128), umma_idesc_f16(TS_BM, cols));
                            if (last) tc_commit(smem_u32(&aux->aempty[slot]));
                        }
                        if (!ok) break;
                        if (last) tc_commit(st_empty);
                        tc_commit(smem_u32(&aux->acc_full[e]));
                    }
                }
            }
        }
    } else if (warp < C::EPI0) {
        // ------------------------------------------------------------------ expanders: packed weights -> int8 planes
        const int n = (warp & 3) * 32 + lane;                            // weight row in the tile
        const uint32_t a_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + C::A_COL;
        int stage = 0;
        uint32_t phase = 0;
        unsigned sb = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            const int m0 = (t % num_m) * (NBU * HMAX);
            const int hn = live - m0 > NBU ? 2 : 1;
            for (int b = 0; b < NSB; ++b, ++sb) {
                if (!mbar_wait(smem_u32(&aux->full[stage]), phase, abort_flag, 0xC00 + stage)) {
                    ok = false;
                    break;
                }
                const uint8_t* st = smem + stage * C::STAGE_BYTES;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int slot = C::RING == 4 ? (int)(sb & 1) * 2 + half : half;
                    uint32_t scw[2];                                         // this half's scales
                    if (Q4) {
                        scw[0] = *(const uint32_t*)(st + C::OFF_SC + n * 8 + half * 4);
                        scw[1] = 0;
                    } else {
                        const uint2 v = *(const uint2*)(st + C::OFF_SC + n * 16 + half * 8);
                        scw[0] = v.x;
                        scw[1] = v.y;
                    }
                    constexpr int STEP = Q4 ? 2 : 1;                         // 32-input steps per store: registers
#pragma unroll
                    for (int c = 0; c < 4; c += STEP) {
                        uint32_t r[16 * STEP];
#pragma unroll
                        for (int e = 0; e < STEP; ++e) {
                            if (Q4) {
                                ts_expand_q4(r + 16 * e, *(const uint4*)(st + C::OFF_WQ + swz(n, half * 4 + c + e)), (scw[0] >> (8 * (c + e))) & 0xff);
                            } else {
                                const uint32_t s2 = scw[c >> 1] >> (16 * (c & 1));
#pragma unroll
                                for (int k = 0; k < 2; ++k) {                // 16 inputs each
                                    const uint32_t sc = (uint32_t)(int)(int8_t)(s2 >> (8 * k));
                                    const uint32_t kc = (((128u - 32u * sc) & 0xffffu) << 16) + (0x8080u - 32u * sc);
                                    const uint4 w = *(const uint4*)(st + C::OFF_WQ + half * (TS_BM * 128) + swz(n, c * 2 + k));
                                    uint32_t* o = r + k * 4;
                                    ts_split_q6(w.x, sc, kc, o[0], o[8]);
                                    ts_split_q6(w.y, sc, kc, o[1], o[9]);
                                    ts_split_q6(w.z, sc, kc, o[2], o[10]);
                                    ts_split_q6(w.w, sc, kc, o[3], o[11]);
                                }
                            }
                        }
                        if (c == 0) {
                            if (!mbar_wait(smem_u32(&aux->aempty[slot]), ((C::RING == 4 ? sb >> 1 : sb) & 1) ^ 1, abort_flag, 0xC10 + slot)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                        }
                        tmem_st(a_base + slot * 64 + c * 16, r);
                    }
                    if (!ok) break;
                    if (Q4 && half == 1) {                                   // free since the half's last use was: its MMAs come after
                        const uint2 mn = *(const uint2*)(st + C::OFF_MN + n * 8);
                        uint8_t* mb = smem + C::OFF_MB + (sb & 1) * C::MB + n * 16;
                        const uint2 h0 = halves_s8(mn.x, 0x3C00), h1 = halves_s8(mn.y, 0x3C00);
                        *(uint4*)mb = *(uint4*)(mb + TS_BM * 16) = make_uint4(h0.x, h0.y, h1.x, h1.y);
                        if (n < hn * NBU) {
                            const uint4 s = *(const uint4*)(st + C::OFF_XS + n * 16);
                            uint8_t* o = smem + C::OFF_SUM + (sb & 1) * C::SB16 + (n / NBU) * (NBU * 32) + (n % NBU) * 16;
                            const uint2 l0 = halves_s8(s.x, 0x3C00), l1 = halves_s8(s.y, 0x3C00);
                            const uint2 u0 = halves_s8(s.z, 0x5400), u1 = halves_s8(s.w, 0x5400);   // 64
                            *(uint4*)o = make_uint4(l0.x, l0.y, l1.x, l1.y);
                            *(uint4*)(o + NBU * 16) = make_uint4(u0.x, u0.y, u1.x, u1.y);
                        }
                        fence_async_smem();
                    }
                    tmem_st_wait();                                          // this warp's rows of the half are in tensor memory
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&aux->afull[slot]));
                }
                if (!ok) break;
                if (lane == 0) mbar_arrive(smem_u32(&aux->empty[stage]));
                if (++stage == C::STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: 32 lanes x a share of a unit's columns per warp
        const int q = warp & 3, ch = (warp - C::EPI0) >> 2;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16);
        float* ring = (float*)(smem + C::OFF_RING) + (warp - C::EPI0) * (C::SLOTS * C::SLOT_F);
        for (int i = lane; i < C::SLOTS * C::SLOT_F; i += 32) ring[i] = 0.0f;
        __syncwarp();
        unsigned u = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            const int m0 = (t % num_m) * (NBU * HMAX), n0 = (t / num_m) * TS_BM;
            const int hn = live - m0 > NBU ? 2 : 1;
            const int n = n0 + q * 32 + lane;
            int cw[HMAX];                                                // this warp's columns of a unit
#pragma unroll
            for (int h = 0; h < HMAX; ++h) {
                const int cols = live - m0 - h * NBU;
                cw[h] = (cols < 0 ? 0 : cols < NBU ? (cols + 15) & ~15 : NBU) / C::CG;
            }
            // the scales of super-block b: each lane copies its weight row's and one activation row's of each unit
            auto fetch = [&](int b) {
                if (b < NSB) {
                    float* s = ring + (b % C::SLOTS) * C::SLOT_F + lane;
                    if (n < p.N) {
                        cp_async4(smem_u32(s), p.d + (long)b * p.N + n);
                        if (Q4) cp_async4(smem_u32(s + 32), p.dm + (long)b * p.N + n);
                    }
#pragma unroll
                    for (int h = 0; h < HMAX; ++h) {
                        const int m = m0 + h * NBU + ch * cw[h] + lane;
                        if (lane < cw[h] && m < live) cp_async4(smem_u32(s + 64 + h * C::AW), p.a + (long)b * p.Ma + m);
                    }
                }
                cp_async_commit();
            };
#pragma unroll
            for (int b = 0; b < C::SLOTS - 1; ++b) fetch(b);
            float2 y2[HMAX][C::AW / 2];
#pragma unroll
            for (int h = 0; h < HMAX; ++h)
#pragma unroll
                for (int j = 0; j < C::AW / 2; ++j) y2[h][j] = make_float2(0.0f, 0.0f);
            for (int b = 0; b < NSB && ok; ++b) {
                cp_async_wait<C::SLOTS - 2>();
                __syncwarp();
                const float* s = ring + (b % C::SLOTS) * C::SLOT_F;
                const float dn = s[lane], dmn = Q4 ? -s[32 + lane] : 0.0f;
                const float2 d2 = make_float2(dn, dn), dm2 = make_float2(dmn, dmn);
#pragma unroll
                for (int h = 0; h < HMAX; ++h) {
                    if (h >= hn) break;
                    const uint32_t e = u & 1;
                    if (!mbar_wait(smem_u32(&aux->acc_full[e]), (u >> 1) & 1, abort_flag, 0xD00 + e)) {
                        ok = false;
                        break;
                    }
                    ++u;
                    tc_fence_after();
                    const uint32_t set = lane_base + e * C::SETC + ch * cw[h];
                    const float* av = s + 64 + h * C::AW;
#pragma unroll
                    for (int c = 0; c < C::AW; c += 8) {                 // cw is a multiple of 8: no column of a neighbour is read
                        if (c >= cw[h]) break;
                        uint32_t p0[8], p1[8], mf[8];
                        tmem_ld8(set + c, p0);
                        tmem_ld8(set + NBU + c, p1);
                        if (Q4) tmem_ld8(set + 2 * NBU + c, mf);
                        float4 av4[2] = {*(const float4*)(av + c), *(const float4*)(av + c + 4)};
                        const float2* a2 = (const float2*)av4;
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            constexpr int R = Q4 ? 8 : 256;
                            const float2 fa = make_float2(__int2float_rn((int)p0[j] + R * (int)p1[j]),
                                                          __int2float_rn((int)p0[j + 1] + R * (int)p1[j + 1]));
                            float2 v = __fmul2_rn(d2, fa);
                            if (Q4) v = __ffma2_rn(dm2, make_float2(__uint_as_float(mf[j]), __uint_as_float(mf[j + 1])), v);
                            y2[h][(c + j) >> 1] = __ffma2_rn(a2[j >> 1], v, y2[h][(c + j) >> 1]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&aux->acc_empty[e]));
                }
                fetch(b + C::SLOTS - 1);                                 // its slot was read one super-block ago
            }
            cp_async_wait<0>();
            __syncwarp();
            // a lane holds one output column: a warp's store of one row is 32 neighbouring columns
            if (ok && n < p.N) {
#pragma unroll
                for (int h = 0; h < HMAX; ++h) {
                    const int mu = m0 + h * NBU + ch * cw[h];
                    if (p.epi == 0) {
                        __nv_bfloat16* o = (__nv_bfloat16*)p.out + n;
#pragma unroll
                        for (int c = 0; c < C::AW; ++c)
                            if (c < cw[h] && mu + c < live)
                                o[(long)(mu + c) * p.ldo] = __float2bfloat16_rn((c & 1) ? y2[h][c >> 1].y : y2[h][c >> 1].x);
                    } else {
                        float* o = (float*)p.out + n;
#pragma unroll
                        for (int c0 = 0; c0 < C::AW; c0 += 8) {
                            float v[8];
#pragma unroll
                            for (int c = 0; c < 8; ++c)
                                if (c0 + c < cw[h] && mu + c0 + c < live) v[c] = __ldcg(o + (long)(mu + c0 + c) * p.ldo);
#pragma unroll
                            for (int c = 0; c < 8; ++c)
                                if (c0 + c < cw[h] && mu + c0 + c < live)
                                    o[(long)(mu + c0 + c) * p.ldo] = __fadd_rn(v[c], (c & 1) ? y2[h][(c0 + c) >> 1].y : y2[h][(c0 + c) >> 1].x);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace w4a8
