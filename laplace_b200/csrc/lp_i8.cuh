// lp_i8.cuh - one super-block (256 values) of 16 weight rows against 8 activation rows per tile on mma.sync int8, for Q4_0,
// Q8_0, Q4_K and Q6_K, and the layout of quantized activations that it reads.
//
// Quantized activations of a tile of 8 rows, per super-block: four pairs of 32-value blocks, 512 bytes each, lane l = 4 * row
// + tq holding 16 bytes: its two B-fragment words of the even block, then of the odd one; then the block scales d of a pair,
// 16 bytes per tq (rows 2 tq and 2 tq + 1 of the even block, then of the odd one); then, Q4_K only, the sums d * sum(q) as three
// bf16 pieces that add up to the fp32 value, 16 bytes per lane: the pieces of blocks 2 tq and 2 tq + 1 as B-fragment words. Which eight of a block's 32 values a lane holds follows from how the weight type packs its values, so that the A
// fragment needs no shuffling: bytes 8 tq .. 8 tq + 7 for Q4_K (one 8-byte load of nibbles serves two blocks), bytes
// 4 tq .. + 3 and 16 + 4 tq .. + 3 for the others.
#pragma once

#include <cuda_bf16.h>

#include "lp_common.cuh"

namespace lp {
namespace i8 {

template <int N> struct Tag { static constexpr int value = N; };

// UNIT: what one copy brings, 16 rows x UNIT_SB super-blocks at PITCH bytes. The pitches keep the fragment loads free of bank
// conflicts (Q4_K: 8-byte loads, 32 mod 128; Q4_0 and Q8_0: 4-byte loads, 16 mod 128) except Q6_K's, two-way.
template <uint32_t TYPE> struct Geo;
template <> struct Geo<LAPLACE_TYPE_Q4_K> {
    static constexpr int SB_BYTES = Q4_K_BYTES, UNIT_SB = 2, PITCH = 288, UNIT_BYTES = 16 * PITCH, ACT_BYTES = 2816;
    static constexpr bool SUMS = true, LANE8 = true;
    __device__ static int first_word(int sb) { return sb * (SB_BYTES / 4); }
    __device__ static uint32_t offset_in_unit(int, int k) { return k * SB_BYTES; }
};
template <> struct Geo<LAPLACE_TYPE_Q8_0> {
    static constexpr int SB_BYTES = 8 * Q8_0_BYTES, UNIT_SB = 1, PITCH = 272, UNIT_BYTES = 16 * PITCH, ACT_BYTES = 2304;
    static constexpr bool SUMS = false, LANE8 = false;
    __device__ static int first_word(int sb) { return sb * (SB_BYTES / 4); }
    __device__ static uint32_t offset_in_unit(int, int) { return 0; }
};
template <> struct Geo<LAPLACE_TYPE_Q4_0> {
    static constexpr int SB_BYTES = 8 * Q4_0_BYTES, UNIT_SB = 1, PITCH = 144, UNIT_BYTES = 16 * PITCH, ACT_BYTES = 2304;
    static constexpr bool SUMS = false, LANE8 = false;
    __device__ static int first_word(int sb) { return sb * (SB_BYTES / 4); }
    __device__ static uint32_t offset_in_unit(int, int) { return 0; }
};
template <> struct Geo<LAPLACE_TYPE_Q6_K> {       // 210-byte super-blocks: a copy starts at the 16-byte boundary below
    static constexpr int SB_BYTES = Q6_K_BYTES, UNIT_SB = 1, PITCH = 224, UNIT_BYTES = 16 * PITCH, ACT_BYTES = 2304;
    static constexpr bool SUMS = false, LANE8 = false;
    __device__ static int first_word(int sb) { return ((sb * SB_BYTES) & ~15) / 4; }
    __device__ static uint32_t offset_in_unit(int sb, int) { return (sb * SB_BYTES) & 15; }
};

// One super-block a unit: what fits beside many activations. Q4_K rows bring 16 bytes more than a super-block, for the pitch.
template <uint32_t TYPE> struct GeoWide : Geo<TYPE> {};
template <> struct GeoWide<LAPLACE_TYPE_Q4_K> : Geo<LAPLACE_TYPE_Q4_K> { static constexpr int UNIT_SB = 1, PITCH = 160, UNIT_BYTES = 16 * PITCH; };

// Four packed int8 from four integers, each clamped to [-128, 127].
__device__ __forceinline__ uint32_t pack4_sat(int a, int b, int c, int d) {
    uint32_t r;
    asm("{\n\t.reg .u32 t;\n\tcvt.pack.sat.s8.s32.b32 t, %4, %3, 0;\n\tcvt.pack.sat.s8.s32.b32 %0, %2, %1, t;\n\t}" : "=r"(r) : "r"(a), "r"(b), "r"(c), "r"(d));
    return r;
}
// One 32-value block in four adjacent lanes (lane t4 holds values 8 t4 .. 8 t4 + 7 in u, v), quantized exactly as the reference
// does (src/matmul_simd.cpp:348-410: d = amax / 127, q = rne(x * (1 / d)), the sum from the unclamped integers). Every lane gets
// the scale and the block's integer sum. Two lanes' worth of values a lane halves the divisions of quantize_block_8lanes.
__device__ __forceinline__ float quantize_block_4lanes(const float4& u, const float4& v, uint32_t& w0, uint32_t& w1, int& sum) {
    float amax = max_nan(max_nan(max_nan(fabsf(u.x), fabsf(u.y)), max_nan(fabsf(u.z), fabsf(u.w))), max_nan(max_nan(fabsf(v.x), fabsf(v.y)), max_nan(fabsf(v.z), fabsf(v.w))));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f);
    const float id = d > 0.0f ? __frcp_rn(d) : 0.0f;
    const int q0 = __float2int_rn(__fmul_rn(u.x, id)), q1 = __float2int_rn(__fmul_rn(u.y, id)), q2 = __float2int_rn(__fmul_rn(u.z, id)), q3 = __float2int_rn(__fmul_rn(u.w, id));
    const int q4 = __float2int_rn(__fmul_rn(v.x, id)), q5 = __float2int_rn(__fmul_rn(v.y, id)), q6 = __float2int_rn(__fmul_rn(v.z, id)), q7 = __float2int_rn(__fmul_rn(v.w, id));
    w0 = pack4_sat(q0, q1, q2, q3);
    w1 = pack4_sat(q4, q5, q6, q7);
    sum = ((q0 + q1) + (q2 + q3)) + ((q4 + q5) + (q6 + q7));
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    return d;
}

// Stores what lane t4 of such a group holds of block j of activation row m (0..7): `sb_act` = this tile's super-block.
template <bool LANE8, bool SUMS>
__device__ __forceinline__ void store_act_as(uint8_t* sb_act, int j, int m, int t4, uint32_t w0, uint32_t w1, float d, int isum) {
    const int pair = j >> 1, odd = j & 1;
    uint8_t* q = sb_act + pair * 512 + m * 64 + odd * 8;
    if (LANE8) {
        *reinterpret_cast<uint2*>(q + t4 * 16) = make_uint2(w0, w1);
    } else {                        // values 4 i .. 4 i + 3, i = 2 t4 and 2 t4 + 1: lane i & 3, word i >> 2
        q += (2 * t4 & 3) * 16 + (t4 >> 1) * 4;
        *reinterpret_cast<uint32_t*>(q) = w0;
        *reinterpret_cast<uint32_t*>(q + 16) = w1;
    }
    if (t4 == 0) {
        reinterpret_cast<float*>(sb_act + 2048)[pair * 16 + (m >> 1) * 4 + odd * 2 + (m & 1)] = d;
        if (SUMS) {
            const float sum = d * static_cast<float>(isum);
            __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(sb_act + 2304 + m * 64 + (j >> 1) * 16) + (j & 1);
            const __nv_bfloat16 b1 = __float2bfloat16_rn(sum);
            const float r1 = sum - __bfloat162float(b1);
            const __nv_bfloat16 b2 = __float2bfloat16_rn(r1);
            w[0] = b1; w[2] = b2; w[4] = __float2bfloat16_rn(r1 - __bfloat162float(b2));
        }
    }
}
template <uint32_t TYPE>
__device__ __forceinline__ void store_act(uint8_t* sb_act, int j, int m, int t4, uint32_t w0, uint32_t w1, float d, int isum) {
    store_act_as<Geo<TYPE>::LANE8, Geo<TYPE>::SUMS>(sb_act, j, m, t4, w0, w1, d, isum);
}

// Block sums on top of the bit pattern of 1.5 * 2^23 (see lp_gemm_i8.cu).
constexpr int MAGIC = 0x4B400000;
__device__ __forceinline__ void mma_us(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(MAGIC));
}
__device__ __forceinline__ void mma_ss(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(MAGIC));
}
__device__ __forceinline__ void mma_ss16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(MAGIC));
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
// acc[row][activation pair] += U * (scale of the row * scales of the two activation rows)
__device__ __forceinline__ void add_block(float2 (&acc)[2], const int (&c)[4], float sa, float sb, float2 d) {
    const float2 off = both(-12582912.f);
    const float2 ua = __fadd2_rn(make_float2(__int_as_float(c[0]), __int_as_float(c[1])), off);
    const float2 ub = __fadd2_rn(make_float2(__int_as_float(c[2]), __int_as_float(c[3])), off);
    acc[0] = __ffma2_rn(ua, __fmul2_rn(both(sa), d), acc[0]);
    acc[1] = __ffma2_rn(ub, __fmul2_rn(both(sb), d), acc[1]);
}
__device__ __forceinline__ float2 lo2(const uint4& v) { return make_float2(__uint_as_float(v.x), __uint_as_float(v.y)); }
__device__ __forceinline__ float2 hi2(const uint4& v) { return make_float2(__uint_as_float(v.z), __uint_as_float(v.w)); }
// four bytes from a shared address that is 2-byte aligned; MIS = the address modulo 4, known where the code is built
template <int MIS>
__device__ __forceinline__ uint32_t lds32_mis(uint32_t addr) {
    static_assert(MIS == 0 || MIS == 2, "2-byte aligned data");
    if (MIS == 0) return lds32(addr);
    return __funnelshift_r(lds32(addr - 2), lds32(addr + 2), 16);
}

// mn . (sum pieces) of 16 weight rows x 8 activation rows over the eight sub-blocks of a super-block: f for the leading pieces, g
// for the other two. mn is exact in bf16 and the pieces add up to the fp32 sums, so every product is exact; apart, the leading
// pieces' sum fits the accumulator, whose truncation would otherwise show (2.7e-7 against 2.0e-7 of error on 4096 x 14336).
__device__ __forceinline__ void mma_mins(float (&f)[4], float (&g)[4], uint32_t mna, uint32_t mnb, const uint4& s) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "r"(mna), "r"(mnb), "r"(s.x), "f"(0.f));
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%4,%5}, {%6,%7}, {%8,%8,%8,%8};"
        : "=f"(g[0]), "=f"(g[1]), "=f"(g[2]), "=f"(g[3]) : "r"(mna), "r"(mnb), "r"(s.y), "r"(s.z), "f"(0.f));
}
// mins of sub-blocks 2 tq and 2 tq + 1 of a row as two bf16 (0x4300 | m is 128 + m), and -dmin
__device__ __forceinline__ uint32_t min_pair(const uint4& h, int tq) {
    const uint32_t lo = h.z & 0x3f3f3f3fu, hi = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u);
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(tq < 2 ? lo : hi), "r"(0x43434343u), "r"((tq & 1) ? 0x4342u : 0x4140u));
    const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&r), __float2bfloat162_rn(128.f));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// acc[s][g][tile][0 / 1] stands for weight rows gq / gq + 8 of 16-row group g (the lane's: gq = lane / 4)
// against activation rows 2 tq, 2 tq + 1 of every tile, for tiles 0 .. live - 1. S = 1: acc[0] += them. S = 2: acc[0] = their sum over
// the super-block (the caller sets both to zero), the four block pairs in two chains, so that no long chain of roundings arises; Q4_K's
// min term, as large as the products' sum and mostly taken back by it, comes last. `row` = shared address of row gq's super-block in the first group; row gq + 8 lies 8
// PITCHes on, the next group 16. `act` = the super-block of the first tile, tiles `act_stride` apart.
// MIS = `row` modulo 4 (Q6_K: 2 for odd super-blocks; otherwise 0).
template <uint32_t TYPE, int PITCH, int MT, int NT, int MIS, int S>
__device__ __forceinline__ void super_block_at(uint32_t row, uint32_t act, uint32_t act_stride, int lane, int live, float2 (&acc)[S][MT][NT][2]) {
    const int tq = lane & 3;
    const uint32_t frag = act + lane * 16, dbase = act + 2048 + tq * 16;
    auto join = [&] {                                        // S = 2: the two chains of a super-block
#pragma unroll
        for (int g = 0; g < MT; ++g)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) acc[0][g][t][h] = __fadd2_rn(acc[0][g][t][h], acc[S - 1][g][t][h]);
    };
    if constexpr (TYPE == LAPLACE_TYPE_Q4_K) {
        // Scales of sub-blocks tq and tq + 4 of both rows (Laplace src/kernels.h:82-90); the other six come by shuffle. High
        // nibbles stay in place (16 times their value), which the scale of an odd sub-block takes back exactly. The min term
        //   sum_j (-dmin * mn_j) * sum_x[j]
        // is a contraction over the eight sub-blocks: two small MMAs and one packed multiply-add per row instead of eight.
        float sc[MT][2][2], ndmin[MT][2];
        uint32_t mn[MT][2];
        auto header = [&](int g, int r, bool scales, bool mins) {
            const uint4 h = lds128(row + (16 * g + 8 * r) * PITCH);
            if (scales) {
                const uint32_t b_lo = (h.y >> (8 * tq)) & 0xff, b_hi = (h.w >> (8 * tq)) & 0xf;
                const float d = half_bits_to_float(h.x) * ((tq & 1) ? 0.0625f : 1.0f);
                sc[g][r][0] = d * static_cast<float>(b_lo & 63);
                sc[g][r][1] = d * static_cast<float>(b_hi | ((b_lo >> 6) << 4));
            }
            if (mins) {
                ndmin[g][r] = -half_bits_to_float(h.x >> 16);
                mn[g][r] = min_pair(h, tq);
            }
        };
        auto min_term = [&](int t) {
            const uint4 s = lds128(frag + t * act_stride + 2304);
#pragma unroll
            for (int g = 0; g < MT; ++g) {
                float f[4], e[4];
                mma_mins(f, e, mn[g][0], mn[g][1], s);
                acc[0][g][t][0] = __ffma2_rn(both(ndmin[g][0]), __fadd2_rn(make_float2(f[0], f[1]), make_float2(e[0], e[1])), acc[0][g][t][0]);
                acc[0][g][t][1] = __ffma2_rn(both(ndmin[g][1]), __fadd2_rn(make_float2(f[2], f[3]), make_float2(e[2], e[3])), acc[0][g][t][1]);
            }
        };
#pragma unroll
        for (int g = 0; g < MT; ++g)
#pragma unroll
            for (int r = 0; r < 2; ++r) header(g, r, true, S == 1);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint2 wa[MT], wb[MT];
            float s0[MT][2], s1[MT][2];
            const int l0 = (lane & ~3) | ((2 * c) & 3), l1 = l0 + 1;
#pragma unroll
            for (int g = 0; g < MT; ++g) {
                wa[g] = lds64(row + 16 * g * PITCH + 16 + 32 * c + 8 * tq);
                wb[g] = lds64(row + (16 * g + 8) * PITCH + 16 + 32 * c + 8 * tq);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    s0[g][r] = __shfl_sync(0xffffffffu, sc[g][r][c >> 1], l0);
                    s1[g][r] = __shfl_sync(0xffffffffu, sc[g][r][c >> 1], l1);
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t >= live) break;
                const uint4 x = lds128(frag + t * act_stride + c * 512), d = lds128(dbase + t * act_stride + c * 64);
#pragma unroll
                for (int g = 0; g < MT; ++g) {
                    int u[4], v[4];
                    mma_us(u, wa[g].x & 0x0f0f0f0fu, wb[g].x & 0x0f0f0f0fu, wa[g].y & 0x0f0f0f0fu, wb[g].y & 0x0f0f0f0fu, x.x, x.y);
                    mma_us(v, wa[g].x & 0xf0f0f0f0u, wb[g].x & 0xf0f0f0f0u, wa[g].y & 0xf0f0f0f0u, wb[g].y & 0xf0f0f0f0u, x.z, x.w);
                    add_block(acc[c % S][g][t], u, s0[g][0], s0[g][1], lo2(d));
                    add_block(acc[c % S][g][t], v, s1[g][0], s1[g][1], hi2(d));
                }
                if (S == 1 && c == 0) min_term(t);
            }
        }
        if constexpr (S == 2) {
            join();
#pragma unroll
            for (int g = 0; g < MT; ++g)
#pragma unroll
                for (int r = 0; r < 2; ++r) header(g, r, false, true);           // read again: registers held over the loop would spill
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t >= live) break;
                min_term(t);
            }
        }
    } else if constexpr (TYPE == LAPLACE_TYPE_Q8_0 || TYPE == LAPLACE_TYPE_Q4_0) {
        constexpr int BB = TYPE == LAPLACE_TYPE_Q8_0 ? Q8_0_BYTES : Q4_0_BYTES;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t a[MT][2][4];
            float sc[MT][2][2];                              // [group][block of the pair][row]
            // quants of an even block (34 or 18 bytes each, the rows 4-byte aligned) lie 2 bytes off a word, those of an odd one on it
            auto load = [&](auto odd) {
                constexpr int o = decltype(odd)::value, MIS = o ? 0 : 2;
#pragma unroll
                for (int g = 0; g < MT; ++g) {
                    const uint32_t ba = row + 16 * g * PITCH + (2 * c + o) * BB, bb = ba + 8 * PITCH;
                    sc[g][o][0] = half_bits_to_float(lds16(ba)); sc[g][o][1] = half_bits_to_float(lds16(bb));
                    if constexpr (TYPE == LAPLACE_TYPE_Q8_0) {
                        a[g][o][0] = lds32_mis<MIS>(ba + 2 + 4 * tq); a[g][o][2] = lds32_mis<MIS>(ba + 18 + 4 * tq);
                        a[g][o][1] = lds32_mis<MIS>(bb + 2 + 4 * tq); a[g][o][3] = lds32_mis<MIS>(bb + 18 + 4 * tq);
                    } else {
                        // byte l: value l in the low nibble, l + 16 in the high one; the signed byte 16 * (nibble - 8) is the
                        // nibble on top with its first bit flipped
                        const uint32_t wa = lds32_mis<MIS>(ba + 2 + 4 * tq), wb = lds32_mis<MIS>(bb + 2 + 4 * tq);
                        a[g][o][0] = ((wa << 4) & 0xf0f0f0f0u) ^ 0x80808080u; a[g][o][2] = (wa & 0xf0f0f0f0u) ^ 0x80808080u;
                        a[g][o][1] = ((wb << 4) & 0xf0f0f0f0u) ^ 0x80808080u; a[g][o][3] = (wb & 0xf0f0f0f0u) ^ 0x80808080u;
                        sc[g][o][0] *= 0.0625f; sc[g][o][1] *= 0.0625f;
                    }
                }
            };
            load(Tag<0>{});
            load(Tag<1>{});
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t >= live) break;
                const uint4 x = lds128(frag + t * act_stride + c * 512), d = lds128(dbase + t * act_stride + c * 64);
#pragma unroll
                for (int g = 0; g < MT; ++g) {
                    int u[4], v[4];
                    mma_ss(u, a[g][0][0], a[g][0][1], a[g][0][2], a[g][0][3], x.x, x.y);
                    mma_ss(v, a[g][1][0], a[g][1][1], a[g][1][2], a[g][1][3], x.z, x.w);
                    add_block(acc[c % S][g][t], u, sc[g][0][0], sc[g][0][1], lo2(d));
                    add_block(acc[c % S][g][t], v, sc[g][1][0], sc[g][1][1], hi2(d));
                }
            }
        }
        if constexpr (S == 2) join();
    } else {
        // Q6_K (Laplace src/kernels.h:46-54, src/matmul.cpp:180-195): half h, group g of 32 values, s = which 16 of them: low four
        // bits from ql[64 h + 32 (g & 1) + l], nibble g / 2, two more from qh[32 h + l] at bit 2 g, scale sc[8 h + 2 g + s].
        // The signed byte 4 * (q6 - 32) is the six bits on top with the first one flipped; the scale carries the quarter.
        float dq[MT][2];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) dq[m][r] = half_bits_to_float(lds16(row + (16 * m + 8 * r) * PITCH + 208)) * 0.25f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float k[MT][2][2];                               // lane tq: scales of group tq, [row][s]
            uint32_t ql[MT][2][2][2], qh[MT][2][2];          // [row][s][g & 1], [row][s]
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t base = row + (16 * m + 8 * r) * PITCH;
                    const uint32_t q = lds16(base + 192 + 8 * h + 2 * tq);
                    k[m][r][0] = dq[m][r] * static_cast<float>(static_cast<int8_t>(q & 0xff));
                    k[m][r][1] = dq[m][r] * static_cast<float>(static_cast<int8_t>(q >> 8));
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const uint32_t at = base + 16 * s + 4 * tq;
                        ql[m][r][s][0] = lds32_mis<MIS>(at + 64 * h);
                        ql[m][r][s][1] = lds32_mis<MIS>(at + 64 * h + 32);
                        qh[m][r][s] = lds32_mis<MIS>(at + 128 + 32 * h);
                    }
                }
#pragma unroll
            for (int gp = 0; gp < 2; ++gp) {                 // groups 2 gp and 2 gp + 1: one pair of activation blocks
                uint32_t a[MT][2][2][2];                     // [g & 1][s][row]
                float sc[MT][2][2][2];
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int o = 0; o < 2; ++o)
#pragma unroll
                        for (int s = 0; s < 2; ++s)
#pragma unroll
                            for (int r = 0; r < 2; ++r) {
                                const int g = 2 * gp + o;
                                sc[m][o][s][r] = __shfl_sync(0xffffffffu, k[m][r][s], (lane & ~3) | g);
                                const uint32_t low = (gp == 0 ? ql[m][r][s][o] << 2 : ql[m][r][s][o] >> 2) & 0x3c3c3c3cu;
                                const uint32_t top = (g < 3 ? qh[m][r][s] << (6 - 2 * g) : qh[m][r][s]) & 0xc0c0c0c0u;
                                a[m][o][s][r] = (low | top) ^ 0x80808080u;
                            }
                const int c = 2 * h + gp;
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    if (t >= live) break;
                    const uint4 x = lds128(frag + t * act_stride + c * 512), d = lds128(dbase + t * act_stride + c * 64);
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        int u[4], v[4];
                        mma_ss16(u, a[m][0][0][0], a[m][0][0][1], x.x);
                        mma_ss16(v, a[m][0][1][0], a[m][0][1][1], x.y);
                        add_block(acc[c % S][m][t], u, sc[m][0][0][0], sc[m][0][0][1], lo2(d));
                        add_block(acc[c % S][m][t], v, sc[m][0][1][0], sc[m][0][1][1], lo2(d));
                        mma_ss16(u, a[m][1][0][0], a[m][1][0][1], x.z);
                        mma_ss16(v, a[m][1][1][0], a[m][1][1][1], x.w);
                        add_block(acc[c % S][m][t], u, sc[m][1][0][0], sc[m][1][0][1], hi2(d));
                        add_block(acc[c % S][m][t], v, sc[m][1][1][0], sc[m][1][1][1], hi2(d));
                    }
                }
            }
        }
        if constexpr (S == 2) join();
    }
}

template <uint32_t TYPE, int PITCH, int MT, int NT, int S>
__device__ __forceinline__ void super_block(uint32_t row, uint32_t act, uint32_t act_stride, int lane, int live, float2 (&acc)[S][MT][NT][2]) {
    if (TYPE == LAPLACE_TYPE_Q6_K && (row & 2)) super_block_at<TYPE, PITCH, MT, NT, 2, S>(row, act, act_stride, lane, live, acc);
    else super_block_at<TYPE, PITCH, MT, NT, 0, S>(row, act, act_stride, lane, live, acc);
}

// ---- quantized rows in fragment order, for calls whose CTAs do not quantize themselves -----------------------------------
// One CTA per activation row; the int8 values, scales and sums are the reference's (see quantize_block_4lanes).
// `sb_stride` = bytes between super-blocks of the row's tile.
template <class Load>
__device__ __forceinline__ void quantize_row_i8(Load load, int K, bool lane8, uint32_t sb_stride, uint8_t* tile, int m) {
    const int bpr = K / 32, grp = threadIdx.x >> 2, t4 = threadIdx.x & 3, groups = blockDim.x >> 2;
    for (int base = 0; base < bpr; base += groups) {           // whole warps iterate together: the shuffles stay converged
        const int b = base + grp;
        const bool live = b < bpr;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 u = live ? load(b, 2 * t4) : zero, v = live ? load(b, 2 * t4 + 1) : zero;
        uint32_t w0, w1; int isum;
        const float d = quantize_block_4lanes(u, v, w0, w1, isum);
        if (!live) continue;
        uint8_t* sb = tile + static_cast<size_t>(b >> 3) * sb_stride;
        if (lane8) store_act_as<true, true>(sb, b & 7, m, t4, w0, w1, d, isum);       // Q4_K
        else store_act_as<false, false>(sb, b & 7, m, t4, w0, w1, d, isum);
    }
}

}  // namespace i8
}  // namespace lp
