// lp_gemm_pair.cu - prefill matmul on pairs of SMs (tcgen05 cta_group::2): Q4_K and Q6_K weights, more than 128 activation rows. The
// "scaled activation" formulation of lp_gemm_sa.cu - the activation operand is 2^e d_x q in two fp16 pieces hi + lo, see there - laid
// out for the pair. Replaces gemm_int<dot_row_q4_k_int_neon / q6_k> of Laplace's NEON back-end (src/matmul_simd.cpp:226-342, 432-455) there.
//
// A pair works on 256 weight rows (the MMA's M side: 128 TMEM lanes of each CTA) x 256 tokens (its N side). Every CTA converts its own 128
// rows and fetches half of the tokens. What bounds the one-CTA kernel of lp_gemm_sa.cu is shared memory: a 16-value step of 128 x 128
// outputs reads 12 KB of operands and takes in 13 KB, some 210 cycles of its bandwidth for 128 of the tensor core. Here a step of 128
// rows x 256 tokens per CTA reads 12 KB (the weight operand once for both pieces: it stays in the collector) and takes in 14 KB for 256
// cycles of the tensor core. Measured (us, calls with quantizer and all, one-CTA kernels -> here): Q4_K 4096 x 14336, 512 tokens 180 -> 108,
// 1024 tokens 344 -> 194; 4096 x 4096, 512 tokens 59 -> 45; 2048 x 2048, 144 tokens 21.5 -> 18; Q6_K 14336 x 4096, 512 tokens 315 -> 144, 1024
// tokens 601 -> 292. At 2048 tokens the card's power limit holds the clock at 1.3 to 1.5 GHz.
// hi and lo meet in one accumulator. Sums in it are truncated, not rounded, at every MMA step, so it is drained after every stage or
// two (figures at UNIT), lo goes in before hi, and what goes in is small:
//   Q4_K   weight operand sc * (nibble - 8), exact in fp16. What is then missing is a contraction over the super-block's eight blocks and
//          goes through the same accumulator as three more steps in bf16: (8 sc_j - dmin / d * mn_j) and the sums 2^e d_x sum(q), three
//          pieces each, the products p1 g1 + p2 g1 + p1 g2 + p2 g2 + p3 g1 + p1 g3 of them. They come last, the smallest first: where a
//          block is not centred at 8 they are several times the result, and every step after them is truncated against them (first: random
//          blocks 9.7e-7, min / max packed ones 6.2e-7; last: 3.6 and 6.8e-7, before the accumulator was drained twice a super-block).
//   Q6_K   sc * (q6 - 32) reaches 4096, one bit more than fp16 holds: the rounded value and the rest (-1, 0 or 1). Of a stage's products the
//          smallest go in first: rest x hi (rest x lo is below 2^-22 of the largest and left out), value x lo, value x hi. What is
//          drained after every stage makes long chains of additions in the drain's registers (224 of them at K = 14336, and more error than
//          all else together), so after 28 super-blocks at most the sums are set aside in scratch memory, 128 KB a CTA.
//
// One 512-thread CTA per SM, persistent; roles by warp:
//   0, 2   copies: hi / lo piece of the activations (64 k x up to 128 tokens, 128-byte swizzle); warp 2 the sum pieces too
//   1      MMA issue (one lane of the even CTA, for both); owns the TMEM allocation
//   3      copies: packed weights (128 rows)
//   4-7    converters: packed super-block -> fp16 operand (thread = weight row), and the row's d into a table for the drain
//   8-15   drain: y += d * accumulator (lane = weight row, 128 tokens a warp; two accumulators of 256 columns)
// All waits are bounded; a wait that gives up raises the status word and the CTA's roles leave their loops.
#include <cuda_bf16.h>

#include "lp_i8.cuh"
#include "lp_scratch.cuh"
#include "lp_tc.cuh"

namespace lp {

namespace {

using namespace tc;

constexpr int TOK = 256;                     // most tokens of a tile
constexpr int ROWS = 256;                    // weight rows of a tile, half of them in each CTA
constexpr int BKC = 64;                      // k per operand stage
constexpr int THREADS = 512;
constexpr int MAX_MATS = 8;
constexpr int TABN = 4, RAWN = 2;
constexpr int TILE = 128 * BKC * 2;          // 16 KB: 128 rows of 64 fp16
constexpr int SB_TILE = 128 * 64 * 2;        // 16 KB: 128 tokens' sum pieces
constexpr int SA_TILE = 128 * 32 * 2;        // 8 KB: 128 weight rows' min pieces
constexpr int SLOT = TOK * ROWS;             // floats of a partial tile: [token][weight row]

// PITCH: bytes between the packed rows in shared memory. Q6_K rows are copied from the 16-byte boundary below.
// UNIT: stages that an accumulator takes in: as many as leave no more error than the one-CTA kernels do, for any weights. Relative error
// against 64 bits, 256 x 4096 x 512, N(0, 1) activations, random blocks / min-max packed / absmax packed weights:
//   Q4_K   one-CTA kernel 3.0 / 6.6 / 2.8e-7; four stages 3.6 / 6.8 / 3.6, two 2.1 / 3.8 / 2.1, one 1.5 / 2.4 / 1.5
//   Q6_K   one-CTA kernel 2.0 / 4.4 / 3.2e-7; two stages 2.8 / 4.2 / 3.3, smallest products first 2.1 / 3.1 / 2.5, one stage so 1.2 / 1.4 / 1.3
// Time at 2048 tokens: Q4_K 4096 x 14336 four 356, two 367, one 420 us; Q6_K 14336 x 4096 two 509, one 526 us (before sums were set aside).
// CHAIN: most super-blocks after which the drain sets its sums aside. Q6_K, random blocks, error in 1e-7, one-CTA kernel / after 16 / 28 / 32:
// 2048 x 14336 x 4096 2.25 / 1.67 / 1.99 / 2.07; K = 8192 in one sum is 2.21 where the one-CTA kernel has 2.12, so the line lies below that.
// 14336 x 4096, 512 tokens: 28 144, 32 145 us.
template <uint32_t TYPE> struct Geo;
template <> struct Geo<LAPLACE_TYPE_Q4_K> { static constexpr int SB = Q4_K_BYTES, PITCH = Q4_K_BYTES, STAGES = 3, PIECES = 1, UNIT = 2, CHAIN = 1 << 20; static constexpr bool MINS = true; };
template <> struct Geo<LAPLACE_TYPE_Q6_K> { static constexpr int SB = Q6_K_BYTES, PITCH = 240, STAGES = 2, PIECES = 2, UNIT = 1, CHAIN = 28; static constexpr bool MINS = false; };

template <uint32_t TYPE> struct Lay {
    using G = Geo<TYPE>;
    static constexpr uint32_t A = 0, W = A + G::STAGES * 2 * TILE, SB = W + G::STAGES * G::PIECES * TILE, SA = SB + (G::MINS ? SB_TILE : 0),
                              RAW = SA + (G::MINS ? SA_TILE : 0), TAB = RAW + RAWN * 128 * G::PITCH, BAR = TAB + TABN * 128 * 4;
    static constexpr uint32_t FULL = BAR, EMPTY = FULL + 8 * G::STAGES, FULL_S = EMPTY + 8 * G::STAGES, EMPTY_S = FULL_S + 8, RAW_FULL = EMPTY_S + 8,
                              RAW_EMPTY = RAW_FULL + 8 * RAWN, TMEM_FULL = RAW_EMPTY + 8 * RAWN, TMEM_EMPTY = TMEM_FULL + 16, TAB_FULL = TMEM_EMPTY + 16,
                              TAB_EMPTY = TAB_FULL + 8 * TABN, LAST = TAB_EMPTY + 8 * TABN, TMEM_PTR = LAST + 8, ABORT = TMEM_PTR + 8,
                              BYTES = ABORT + 8 + 1024;       // + slack for the 1024-byte alignment
    static_assert(BYTES <= 227 * 1024, "shared memory budget");
    static_assert(RAW % 1024 == 0 && TAB % 128 == 0, "alignment of copies");
};

struct PairMaps {
    CUtensorMap a[4];              // [2 m_pad][K] fp16 (hi rows, lo rows), boxes of 64 k x {16, 32, 64, 128} rows, 128-byte swizzle
    CUtensorMap s[4];              // [m_pad][K / 4] bf16, boxes of 64 x the same, 128-byte swizzle
    CUtensorMap w[MAX_MATS];       // packed weights, boxes of one super-block x 128 rows
};
struct PairParams {
    const float* inv_s;            // [m_pad]: 2^-e of the row
    int*         err;
    int          M, K, m_pad, tiles_m, n_mats;
    int          rb, by_row;       // bytes per weight row; 1 (Q6_K): rows that a tensor map cannot address are copied one by one
    const uint8_t* w[MAX_MATS];
    float*       y[MAX_MATS];
    int          N[MAX_MATS];
    // How a matrix's tiles (weight rows outside, tokens inside) are shared out, by its own size alone, so that it has the same bits alone and
    // beside others. The first `whole` are dealt round-robin from pair `shift` on; those behind are cut: their super-blocks, `units` in tile
    // order, go evenly to the `cut` pairs from there on (the c-th: [c * units / cut, (c + 1) * units / cut)). The c-th pair's piece
    // of the t-th cut tile is the matrix's partial result c + t: from one piece to the next c or t grows, or both.
    int          tiles[MAX_MATS], whole[MAX_MATS], units[MAX_MATS], cut[MAX_MATS], shift[MAX_MATS], slot0[MAX_MATS];
    float*       part;
    float*       aside;            // [CTA][TOK][128]: sums of K taken out of the drain's registers every CHAIN super-blocks
};
// Row-split over several GPUs: the result goes to row-major [M][ld] buffers of every GPU at column col0 + n instead of y[0].
template <bool PEERS> struct PairPeers {};
template <> struct PairPeers<true> { float* y[MAX_PEERS]; int n, ld, col0; };

struct Seg { int mat, m0, n0, nt, sb0, sb1, part; };      // nt: tokens
__host__ __device__ __forceinline__ int cut_start(int units, int pairs, int c) { return static_cast<int>(static_cast<long long>(units) * c / pairs); }
__device__ __forceinline__ void tile_at(const PairParams& p, int t, Seg& s) {
    s.m0 = (t % p.tiles_m) * TOK;
    s.nt = p.M - s.m0 < TOK ? p.M - s.m0 : TOK;
    s.n0 = (t / p.tiles_m) * ROWS;
}
// A CTA fetches 16, 32, 64 or 128 tokens, half of what the tile has or a little more: token c of the tile is accumulator column c.
__device__ __forceinline__ int box_bucket(int nt) { return nt <= 32 ? 0 : nt <= 64 ? 1 : nt <= 128 ? 2 : 3; }
// Piece i of a pair's work, in the order in which every role walks it; false: there are no more. Worked out anew for every piece (from a
// volatile read of the CTA's number), so that none of it stays in registers meanwhile: the drain has none to spare.
__device__ __forceinline__ bool segment(const PairParams& p, int i, Seg& s) {
    uint32_t cta, grid;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(cta));
    asm volatile("mov.u32 %0, %%nctaid.x;" : "=r"(grid));
    const int pairs = static_cast<int>(grid) >> 1, nsb = p.K / 256;
    for (s.mat = 0; s.mat < p.n_mats; ++s.mat) {
        int vp = (static_cast<int>(cta) >> 1) - p.shift[s.mat];
        if (vp < 0) vp += pairs;
        const int whole = p.whole[s.mat], n_whole = vp < whole ? (whole - vp + pairs - 1) / pairs : 0;
        if (i < n_whole) {
            s.sb0 = 0; s.sb1 = nsb; s.part = -1;
            tile_at(p, vp + i * pairs, s);
            return true;
        }
        i -= n_whole;
        if (vp < p.cut[s.mat]) {
            const int u0 = cut_start(p.units[s.mat], p.cut[s.mat], vp), u1 = cut_start(p.units[s.mat], p.cut[s.mat], vp + 1);
            const int first = u0 / nsb, last = (u1 - 1) / nsb, t = first + i;
            if (t <= last) {
                s.sb0 = t == first ? u0 - first * nsb : 0;
                s.sb1 = t == last ? u1 - last * nsb : nsb;
                s.part = s.sb0 > 0 || s.sb1 < nsb ? p.slot0[s.mat] + vp + t : -1;
                tile_at(p, whole + t, s);
                return true;
            }
            i -= last - first + 1;
        }
    }
    return false;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" :: "r"(addr), "f"(v) : "memory"); }
// a pair of fp32 values as three bf16 pieces each that add up to them
__device__ __forceinline__ void split3(float2 v, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
    const float2 r = make_float2(v.x - __low2float(a), v.y - __high2float(a));
    const __nv_bfloat162 b = __floats2bfloat162_rn(r.x, r.y);
    const __nv_bfloat162 c = __floats2bfloat162_rn(r.x - __low2float(b), r.y - __high2float(b));
    p1 = *reinterpret_cast<const uint32_t*>(&a); p2 = *reinterpret_cast<const uint32_t*>(&b); p3 = *reinterpret_cast<const uint32_t*>(&c);
}

// 64 weight values (chunk c of the super-block at `raw`) of a Q4_K row as fp16: the low nibbles of 32 bytes, less 8, times one scale, then
// the high ones times the next. Within every four values the order is (0, 2, 1, 3), as in the activation operand. A nibble in bits 4..7
// under 0x5400 is fp16(64 + v), and (64 + v) * sc - 72 * sc = (v - 8) * sc exactly.
__device__ __forceinline__ void convert_q4k(uint32_t raw, int c, uint32_t sc_lo, uint32_t sc_hi, uint32_t wrow, int r7) {
    const uint32_t scw = c < 2 ? sc_lo : sc_hi;
    const __half2 s1 = __half2half2(__ushort2half_rn(static_cast<unsigned short>((scw >> (16 * (c & 1))) & 0xff)));
    const __half2 s2 = __half2half2(__ushort2half_rn(static_cast<unsigned short>((scw >> (16 * (c & 1) + 8)) & 0xff)));
    const __half2 o1 = __hmul2(s1, __half2half2(__float2half_rn(-72.f)));
    const __half2 o2 = __hmul2(s2, __half2half2(__float2half_rn(-72.f)));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 qv = lds128(raw + 16 + 32 * c + 16 * h);
        const uint32_t w4[4] = {qv.x, qv.y, qv.z, qv.w};
        uint32_t a[8], b[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t w = w4[i];
            a[2 * i] = h2_bits(__hfma2(bits_h2(((w << 4) & 0x00f000f0u) | 0x54005400u), s1, o1));
            a[2 * i + 1] = h2_bits(__hfma2(bits_h2(((w >> 4) & 0x00f000f0u) | 0x54005400u), s1, o1));
            b[2 * i] = h2_bits(__hfma2(bits_h2((w & 0x00f000f0u) | 0x54005400u), s2, o2));
            b[2 * i + 1] = h2_bits(__hfma2(bits_h2(((w >> 8) & 0x00f000f0u) | 0x54005400u), s2, o2));
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            sts128(wrow + (((2 * h + j) ^ r7) << 4), a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]);
            sts128(wrow + (((4 + 2 * h + j) ^ r7) << 4), b[4 * j], b[4 * j + 1], b[4 * j + 2], b[4 * j + 3]);
        }
    }
}
// Two chunks (half h of the super-block at `raw`) of a Q6_K row (Laplace src/kernels.h:46-54, src/matmul.cpp:180-195): value v of nibble
// side nib: 4 bits from ql[64 h + v], 2 bits from qh[32 h + (v & 31)], scale sc[8 h + 4 nib + (v >> 4)]. sc * (q6 - 32) rounded to fp16
// and the rest, which one fused multiply-add gives exactly. The rest lies
// TILE bytes behind.
struct Q6Half { uint32_t ql[16], qh[8], sc[2]; };
template <int N>
__device__ __forceinline__ void words_at(uint32_t addr, uint32_t (&out)[N]) {        // addr is 2-byte aligned
    const uint32_t sh = (addr & 2u) * 8u, base = addr & ~3u;
    uint32_t w = lds32(base);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const uint32_t next = lds32(base + 4 * i + 4);
        out[i] = __funnelshift_r(w, next, sh);
        w = next;
    }
}
__device__ __forceinline__ void convert_q6k(const Q6Half& q, int nib, bool zero, uint32_t wrow, int r7) {
    const __half2 k1056 = __half2half2(__float2half_rn(1056.f));
    const uint32_t scw = zero ? 0u : nib ? q.sc[1] : q.sc[0];
#pragma unroll
    for (int j4 = 0; j4 < 4; ++j4) {
        const __half2 sc = __half2half2(__short2half_rn(static_cast<short>(static_cast<int8_t>(scw >> (8 * j4)))));
        const int hshift = 2 * (2 * nib + (j4 >> 1));
        uint32_t hw[8], lw[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t q6 = ((q.ql[4 * j4 + i] >> (4 * nib)) & 0x0f0f0f0fu) | (((q.qh[4 * (j4 & 1) + i] >> hshift) << 4) & 0x30303030u);
            const __half2 x02 = __hsub2(bits_h2((q6 & 0x00ff00ffu) | 0x64006400u), k1056), x13 = __hsub2(bits_h2(((q6 >> 8) & 0x00ff00ffu) | 0x64006400u), k1056);
            const __half2 h02 = __hmul2(sc, x02), h13 = __hmul2(sc, x13);
            hw[2 * i] = h2_bits(h02); lw[2 * i] = h2_bits(__hfma2(sc, x02, __hneg2(h02)));
            hw[2 * i + 1] = h2_bits(h13); lw[2 * i + 1] = h2_bits(__hfma2(sc, x13, __hneg2(h13)));
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            sts128(wrow + (((2 * j4 + j) ^ r7) << 4), hw[4 * j], hw[4 * j + 1], hw[4 * j + 2], hw[4 * j + 3]);
            sts128(wrow + TILE + (((2 * j4 + j) ^ r7) << 4), lw[4 * j], lw[4 * j + 1], lw[4 * j + 2], lw[4 * j + 3]);
        }
    }
}

// Where super-block sb of a weight row starts, and how far that is above the 16-byte boundary at which its copy starts.
__device__ __forceinline__ const uint8_t* row_src(const PairParams& p, int mat, int row, int sb, int sb_bytes, uint32_t& mis) {
    const uint8_t* src = p.w[mat] + static_cast<size_t>(row) * p.rb + static_cast<size_t>(sb) * sb_bytes;
    mis = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src) & 15u);
    return src - mis;
}

template <uint32_t TYPE, bool PEERS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps maps, const __grid_constant__ PairParams p, const PairPeers<PEERS> pe) {
    using G = Geo<TYPE>;
    using L = Lay<TYPE>;
    constexpr int STAGES = G::STAGES, UNIT = G::UNIT;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (sbase - smem_u32(smem_raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = pair_rank();
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::ABORT);
    auto leader = [&](uint32_t off) { return map_to_rank(sbase + off, 0); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(sbase + L::FULL + 8 * s, 2 + 8);          // the even CTA's: its copy warps (bytes of both CTAs), the converter warps of both
            mbar_init(sbase + L::EMPTY + 8 * s, 1);             // tcgen05.commit
        }
        mbar_init(sbase + L::FULL_S, 1 + 8);
        mbar_init(sbase + L::EMPTY_S, 1);
        for (int s = 0; s < RAWN; ++s) { mbar_init(sbase + L::RAW_FULL + 8 * s, 1); mbar_init(sbase + L::RAW_EMPTY + 8 * s, 4); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(sbase + L::TMEM_FULL + 8 * s, 1);         // tcgen05.commit
            mbar_init(sbase + L::TMEM_EMPTY + 8 * s, 16);       // the even CTA's: the drain warps of both
        }
        for (int s = 0; s < TABN; ++s) { mbar_init(sbase + L::TAB_FULL + 8 * s, 4); mbar_init(sbase + L::TAB_EMPTY + 8 * s, 8); }
        mbar_init(sbase + L::LAST, 1);
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(sbase + L::TMEM_PTR), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");        // both CTAs' barriers exist before either arrives on them
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + L::TMEM_PTR);

    // Counters that every role advances in the same order: it = operand stage (64 k), sbc = super-block, u = accumulator (4 / UNIT per
    // super-block).
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if ((warp == 0 || warp == 2) && elect_one()) {
            asm volatile("griddepcontrol.wait;" ::: "memory");            // the activations are written by the kernel before
            const int pc = warp >> 1;
            int it = 0, sbc = 0;
            bool ok = true;
            Seg sg;
            for (int i = 0; ok && segment(p, i, sg); ++i) {
                const int bk = box_bucket(sg.nt), box = 16 << bk, row = sg.m0 + static_cast<int>(rank) * box;
                for (int sb = sg.sb0; sb < sg.sb1 && ok; ++sb, ++sbc) {
                    for (int c = 0; c < 4; ++c, ++it) {
                        const int s = it % STAGES;
                        if (!wait_or_abort<false>(sbase + L::EMPTY + 8 * s, ((it / STAGES) & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
                        if (rank == 0) mbar_expect_tx(sbase + L::FULL + 8 * s, 2 * box * 128);
                        tma_load_2d_pair(sbase + L::A + (2 * s + pc) * TILE, &maps.a[bk], sb * 256 + c * BKC, pc * p.m_pad + row, leader(L::FULL + 8 * s));
                        if (G::MINS && pc == 1 && c == 2) {
                            if (!wait_or_abort<false>(sbase + L::EMPTY_S, (sbc & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
                            if (rank == 0) mbar_expect_tx(sbase + L::FULL_S, 2 * box * 128);
                            tma_load_2d_pair(sbase + L::SB, &maps.s[bk], sb * 64, row, leader(L::FULL_S));
                        }
                    }
                }
            }
            // The MMAs that read the last stages are done, so their copies have landed and no commit is under way to this CTA any more.
            // After a wait that gave up the copies are given time to land instead.
            if (ok) {
                for (int k = 1; k <= STAGES && it - k >= 0; ++k) ok &= mbar_wait_bounded(sbase + L::EMPTY + 8 * ((it - k) % STAGES), ((it - k) / STAGES) & 1);
                if (G::MINS && sbc > 0) ok &= mbar_wait_bounded(sbase + L::EMPTY_S, (sbc - 1) & 1);
                if (!ok) report_status(p.err, DEV_TIMEOUT_DRAIN);
            } else {
                for (int k = 0; k < 1000; ++k) __nanosleep(1000);
            }
        } else if (warp == 1 && rank == 0 && elect_one()) {
            int it = 0, sbc = 0, u = 0;
            bool ok = true;
            Seg sg;
            for (int i = 0; ok && segment(p, i, sg); ++i) {
                // fp32 += fp16 x fp16, 256 weight rows x the tile's tokens
                const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>((32 << box_bucket(sg.nt)) >> 3) << 17) | ((ROWS >> 4) << 24);
                const uint32_t idesc_bf16 = idesc | (1u << 7) | (1u << 10);
                for (int sb = sg.sb0; sb < sg.sb1 && ok; ++sb, ++sbc) {
#pragma unroll 1
                    for (int c = 0; c < 4; ++c, ++it) {
                        const int s = it % STAGES;
                        const uint32_t acc = tmem_base + (u & 1) * TOK;
                        const uint32_t more = c % UNIT != 0;
                        if (!more) {
                            if (!wait_pair(sbase + L::TMEM_EMPTY + 8 * (u & 1), ((u >> 1) & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_TMEM)) { ok = false; break; }
                            fence_after();
                        }
                        if (!wait_pair(sbase + L::FULL + 8 * s, (it / STAGES) & 1, abort_flag, p.err, DEV_TIMEOUT_FULL)) { ok = false; break; }
                        fence_after();
                        const uint64_t w = smem_desc_sw128(sbase + L::W + s * G::PIECES * TILE), x = smem_desc_sw128(sbase + L::A + 2 * s * TILE);
                        // (32 bytes >> 4 inside the swizzle row)
                        if constexpr (G::PIECES == 2) {                                // the smallest products first
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) mma_f16_pair(acc, w + (TILE >> 4) + 2 * ks, x + 2 * ks, idesc, more | ks);
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) mma_f16_pair(acc, w + 2 * ks, x + (TILE >> 4) + 2 * ks, idesc, 1);
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) mma_f16_pair(acc, w + 2 * ks, x + 2 * ks, idesc, 1);
                        } else {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                mma_f16_pair_fill(acc, w + 2 * ks, x + (TILE >> 4) + 2 * ks, idesc, more | ks);
                                mma_f16_pair_last(acc, w + 2 * ks, x + 2 * ks, idesc, 1);
                            }
                        }
                        commit_pair(sbase + L::EMPTY + 8 * s);
                        if (G::MINS && c == 3) {                                       // the smallest products first
                            if (!wait_pair(sbase + L::FULL_S, sbc & 1, abort_flag, p.err, DEV_TIMEOUT_FULL)) { ok = false; break; }
                            fence_after();
                            const uint64_t a = smem_desc_sw64(sbase + L::SA), b = smem_desc_sw128(sbase + L::SB);
                            mma_f16_pair(acc, a + 2, b + 4, idesc_bf16, 1);
                            mma_f16_pair(acc, a, b + 2, idesc_bf16, 1);
                            mma_f16_pair(acc, a, b, idesc_bf16, 1);
                            commit_pair(sbase + L::EMPTY_S);
                        }
                        if (c % UNIT == UNIT - 1) { commit_pair(sbase + L::TMEM_FULL + 8 * (u & 1)); ++u; }
                    }
                }
            }
            if (!ok) {                       // MMAs in flight end before the pair's shared memory is given back
                asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(sbase + L::LAST) : "memory");
                mbar_wait_bounded(sbase + L::LAST, 0);
            }
        } else if (warp == 3) {
            // ---------------- packed weights of this CTA's 128 rows (a tensor map fills rows past N with zeros) ----------------
            int sbc = 0;
            bool ok = true;
            Seg sg;
            for (int i = 0; ok && segment(p, i, sg); ++i) {
                const int row = sg.n0 + static_cast<int>(rank) * 128;
                for (int sb = sg.sb0; sb < sg.sb1; ++sb, ++sbc) {
                    const int s = sbc % RAWN;
                    const uint32_t dst = sbase + L::RAW + s * 128 * G::PITCH, bar = sbase + L::RAW_FULL + 8 * s;
                    if (!wait_or_abort<false>(sbase + L::RAW_EMPTY + 8 * s, ((sbc / RAWN) & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
                    if (TYPE == LAPLACE_TYPE_Q4_K || !p.by_row) {
                        if (lane == 0) {
                            mbar_expect_tx(bar, 128 * G::PITCH);
                            tma_load_2d(dst, &maps.w[sg.mat], ((sb * G::SB) & ~15) / 4, row, bar);
                        }
                    } else {
                        int live = p.N[sg.mat] - row;
                        live = live < 0 ? 0 : live > 128 ? 128 : live;
                        uint32_t total = 0, bytes[4];
                        const uint8_t* src[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t mis;
                            src[j] = row_src(p, sg.mat, row + lane + 32 * j, sb, G::SB, mis);
                            bytes[j] = lane + 32 * j < live ? (mis + G::SB + 15u) & ~15u : 0u;
                            total += bytes[j];
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
                        if (lane == 0) mbar_expect_tx(bar, total);
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (bytes[j]) bulk_g2s(dst + (lane + 32 * j) * G::PITCH, src[j], bytes[j], bar);
                    }
                    __syncwarp();
                }
            }
            if (!ok && lane == 0)
                for (int k = 1; k <= RAWN && sbc - k >= 0; ++k) mbar_wait_bounded(sbase + L::RAW_FULL + 8 * ((sbc - k) % RAWN), ((sbc - k) / RAWN) & 1);
        }
        __syncwarp();
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    } else if (warp < 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        // ---------------- converters: thread r owns weight row n0 + 128 * rank + r ----------------
        const int r = threadIdx.x - 128, r7 = r & 7;
        int it = 0, sbc = 0;
        bool ok = true;
        Seg sg;
        for (int i = 0; ok && segment(p, i, sg); ++i) {
            const int row = sg.n0 + static_cast<int>(rank) * 128 + r;
            const bool live = row < p.N[sg.mat];
            for (int sb = sg.sb0; sb < sg.sb1 && ok; ++sb, ++sbc) {
                const int q = sbc % RAWN, slot = sbc % TABN;
                uint32_t raw = sbase + L::RAW + q * 128 * G::PITCH + r * G::PITCH;
                if (!wait_or_abort<false>(sbase + L::RAW_FULL + 8 * q, (sbc / RAWN) & 1, abort_flag, p.err, DEV_TIMEOUT_FULL) ||
                    !wait_or_abort<false>(sbase + L::TAB_EMPTY + 8 * slot, ((sbc / TABN) & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
                // the accumulator is in units of d; a super-block whose d is zero has a zero operand and units of one (its min term stays)
                auto table = [&](float d) {
                    sts32(sbase + L::TAB + (slot * 128 + r) * 4, d);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sbase + L::TAB_FULL + 8 * slot);
                };
                auto begin = [&](int s) { return wait_or_abort<false>(sbase + L::EMPTY + 8 * s, ((it / STAGES) & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY); };
                auto publish = [&](uint32_t off) {
                    fence_proxy_async();          // generic-proxy stores -> visible to the tensor cores' reads
                    __syncwarp();
                    if (lane == 0) arrive_cluster(leader(off));
                };
                if constexpr (TYPE == LAPLACE_TYPE_Q4_K) {
                    const uint4 hdr = lds128(raw);
                    // 6-bit scales / mins, eight of each (Laplace src/kernels.h:82-90), one per byte
                    uint32_t sc_lo = 0, sc_hi = 0;
                    float d = 1.0f;
                    if (hdr.x & 0x7fffu) {
                        sc_lo = hdr.y & 0x3f3f3f3fu;
                        sc_hi = (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
                        d = half_bits_to_float(hdr.x);
                    }
                    table(d);
#pragma unroll 1
                    for (int c = 0; c < 4; ++c, ++it) {
                        const int s = it % STAGES;
                        if (c == 3) {
                            // what a block's sum is multiplied with: 8 sc_j (the nibbles' offset) - dmin / d * mn_j, as three bf16 pieces that add up
                            // to it, in the order p1 p2 p3 p1
                            const float cm = __fdiv_rn(-half_bits_to_float(hdr.x >> 16), d);
                            uint32_t p1[4], p2[4], p3[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const uint32_t mn = j < 2 ? hdr.z & 0x3f3f3f3fu : ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u), sc = j < 2 ? sc_lo : sc_hi;
                                const int at = 16 * (j & 1);
                                split3(make_float2(fmaf(cm, static_cast<float>((mn >> at) & 0xffu), 8.0f * static_cast<float>((sc >> at) & 0xffu)),
                                                   fmaf(cm, static_cast<float>((mn >> (at + 8)) & 0xffu), 8.0f * static_cast<float>((sc >> (at + 8)) & 0xffu))), p1[j], p2[j], p3[j]);
                            }
                            if (!wait_or_abort<false>(sbase + L::EMPTY_S, (sbc & 1) ^ 1, abort_flag, p.err, DEV_TIMEOUT_EMPTY)) { ok = false; break; }
                            const uint32_t srow = sbase + L::SA + r * 64;
                            const int r3 = (r >> 1) & 3;
                            sts128(srow + ((0 ^ r3) << 4), p1[0], p1[1], p1[2], p1[3]);
                            sts128(srow + ((1 ^ r3) << 4), p2[0], p2[1], p2[2], p2[3]);
                            sts128(srow + ((2 ^ r3) << 4), p3[0], p3[1], p3[2], p3[3]);
                            sts128(srow + ((3 ^ r3) << 4), p1[0], p1[1], p1[2], p1[3]);
                            publish(L::FULL_S);
                        }
                        if (!begin(s)) { ok = false; break; }
                        convert_q4k(raw, c, sc_lo, sc_hi, sbase + L::W + s * TILE + r * 128, r7);
                        publish(L::FULL + 8 * s);
                    }
                } else {
                    uint32_t mis = (sb * G::SB) & 15;
                    if (p.by_row) row_src(p, sg.mat, row, sb, G::SB, mis);
                    const uint32_t db = live ? lds16(raw + mis + 208) : 0u;
                    const bool zero = (db & 0x7fffu) == 0;
                    table(zero ? 1.0f : half_bits_to_float(db));
#pragma unroll 1
                    for (int h = 0; h < 2 && ok; ++h) {
                        Q6Half q6;
                        words_at(raw + mis + 64 * h, q6.ql);
                        words_at(raw + mis + 128 + 32 * h, q6.qh);
                        words_at(raw + mis + 192 + 8 * h, q6.sc);
#pragma unroll
                        for (int nib = 0; nib < 2; ++nib, ++it) {
                            const int s = it % STAGES;
                            if (!begin(s)) { ok = false; break; }
                            convert_q6k(q6, nib, zero, sbase + L::W + s * 2 * TILE + r * 128, r7);
                            publish(L::FULL + 8 * s);
                        }
                    }
                }
                if (!ok) break;
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + L::RAW_EMPTY + 8 * q);
            }
        }
    } else {
        // (register budget of the CTA: 4 x 40 + 4 x 88 + 8 x 192 <= 16 x 128 per lane; a sum above what the CTA was
        // launched with would leave setmaxnreg.inc waiting for registers that never come)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
        // ---------------- drain: lane = weight row, 128 tokens per warp ----------------
        const int quad = warp & 3, half = (warp - 8) >> 2;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * 128;
        const uint32_t bar_empty = leader(L::TMEM_EMPTY);
        const int wr = quad * 32 + lane;
        int sbc = 0, u = 0;
        bool ok = true;
        Seg sg;
        for (int i = 0; ok && segment(p, i, sg); ++i) {
            const int live = sg.nt - half * 128;                     // tokens of this warp's columns (warp-uniform)
            float2 y[64];
#pragma unroll
            for (int c = 0; c < 64; ++c) y[c] = make_float2(0.f, 0.f);
            // y of this thread's row set aside: kept here (first) or added to what is kept
            float* aside = TYPE == LAPLACE_TYPE_Q6_K ? p.aside + (static_cast<size_t>(blockIdx.x) * TOK + half * 128) * 128 + wr : nullptr;
            auto add_aside = [&](int h) {                            // sixteen tokens' sums, loads in flight together
                float v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) v[e] = aside[(16 * h + e) * 128];
#pragma unroll
                for (int e = 0; e < 8; ++e) { y[8 * h + e].x += v[2 * e]; y[8 * h + e].y += v[2 * e + 1]; }
            };
            auto set_aside = [&](bool first) {
#pragma unroll
                for (int h = 0; h < 8; ++h) {
                    if (16 * h >= live) break;
                    if (!first) add_aside(h);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        aside[(16 * h + 2 * e) * 128] = y[8 * h + e].x;
                        aside[(16 * h + 2 * e + 1) * 128] = y[8 * h + e].y;
                        y[8 * h + e] = make_float2(0.f, 0.f);
                    }
                }
            };
            const int len = sg.sb1 - sg.sb0, chains = (len + G::CHAIN - 1) / G::CHAIN, step = (len + chains - 1) / chains;
            int left = len - step;                                   // super-blocks to go when the sums are next set aside
            for (int n = len; n > 0 && ok; --n, ++sbc) {
                if (n == left) { set_aside(left == len - step); left -= step; }
                const int slot = sbc % TABN;
                if (!wait_or_abort<false>(sbase + L::TAB_FULL + 8 * slot, (sbc / TABN) & 1, abort_flag, p.err, DEV_TIMEOUT_FULL)) { ok = false; break; }
                const float d = __uint_as_float(lds32(sbase + L::TAB + (slot * 128 + wr) * 4));
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + L::TAB_EMPTY + 8 * slot);
#pragma unroll 1
                for (int k = 0; k < 4 / UNIT; ++k, ++u) {
                    const uint32_t b = u & 1;
                    if (!wait_or_abort<true>(sbase + L::TMEM_FULL + 8 * b, (u >> 1) & 1, abort_flag, p.err, DEV_TIMEOUT_MMA)) { ok = false; break; }
                    fence_after();
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (c * 32 < live) {
                            float v[32];
                            ld32(t_lane + b * TOK + c * 32, v);
                            wait_ld();
#pragma unroll
                            for (int e = 0; e < 16; ++e) y[c * 16 + e] = __ffma2_rn(make_float2(d, d), make_float2(v[2 * e], v[2 * e + 1]), y[c * 16 + e]);
                        }
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_cluster(bar_empty + 8 * b);
                }
            }
            if (!ok) break;
            if (chains > 1) {
#pragma unroll
                for (int h = 0; h < 8; ++h)
                    if (16 * h < live) add_aside(h);
            }
            // for a fixed token the warp's 32 lanes write 32 consecutive floats
            const int n = sg.n0 + static_cast<int>(rank) * 128 + wr, N = p.N[sg.mat], tok0 = half * 128;
            float inv[4];                                            // of column 32 k + lane
#pragma unroll
            for (int k = 0; k < 4; ++k) inv[k] = 32 * k + lane < live ? __ldg(p.inv_s + sg.m0 + tok0 + 32 * k + lane) : 0.f;
            auto store = [&](float* dst, size_t ld, bool in) {
#pragma unroll
                for (int c = 0; c < 128; ++c) {
                    const float v = ((c & 1) ? y[c >> 1].y : y[c >> 1].x) * __shfl_sync(0xffffffffu, inv[c >> 5], c & 31);
                    if (in && c < live) *dst = v;
                    dst += ld;
                }
            };
            if (sg.part >= 0) {
                store(p.part + static_cast<size_t>(sg.part) * SLOT + tok0 * ROWS + rank * 128 + wr, ROWS, true);
            } else {
                if constexpr (PEERS) {
#pragma unroll 1
                    for (int g = 0; g < pe.n; ++g) store(pe.y[g] + static_cast<size_t>(sg.m0 + tok0) * pe.ld + pe.col0 + n, pe.ld, n < N);
                } else {
                    store(p.y[sg.mat] + static_cast<size_t>(sg.m0 + tok0) * N + n, N, n < N);
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");        // neither CTA leaves while the other may still reach into it
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512) : "memory");
    }
}

// ---- activations: one block per row. The int8 values, block scales d and sums are the reference's (src/matmul_simd.cpp:348-410); optional
// RMSNorm in front (src/ops.cpp:34-74: inv = 1 / sqrt(mean(x^2) + eps), x_norm = (x * inv) * w). Scales and sums are brought to a common
// power of two per row, so that neither huge nor tiny rows leave the range of the running sums. ----
struct PairOperand {
    __half* a;                 // [2][m_pad][K]: hi rows, lo rows; within every four values the order (0, 2, 1, 3)
    __nv_bfloat16* s;          // [m_pad][K / 4]: per super-block the sums' pieces, eight each, in the order g1 g1 g2 g2 g1 g3, and 16 unused
    float*  inv_s;             // [m_pad]
    int     m_pad;
};

// Four lanes per 32-value block, 64 blocks at a time. NIT: rounds that a row takes; its values then stay in registers over the norm, the
// row's maximum and the quantization, all loads in flight at once (512 rows of 4096: 9.5 us with three passes over the row, 5 so). 0: rows of
// any length, read again for every pass.
template <int NIT>
__global__ void __launch_bounds__(256) quantize_pair_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps,
                                                            float* __restrict__ x_norm_out, int K, PairOperand op, int sums) {
    __shared__ float red[8], red2[8];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int m = blockIdx.x, bpr = K / 32, grp = threadIdx.x >> 2, t4 = threadIdx.x & 3, warp = threadIdx.x >> 5;
    const int rounds = NIT ? NIT : (bpr + 63) / 64;
    const float4* xr = reinterpret_cast<const float4*>(x + static_cast<size_t>(m) * K) + 2 * t4;
    const float4* nr = reinterpret_cast<const float4*>(norm_w) + 2 * t4;
    float4 v[NIT ? NIT : 1][2];
    auto fetch = [&](int r, float4 (&o)[2]) {
        const int b = r * 64 + grp;
#pragma unroll
        for (int e = 0; e < 2; ++e) o[e] = b < bpr ? __ldg(xr + b * 8 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    if constexpr (NIT > 0) {
#pragma unroll
        for (int r = 0; r < NIT; ++r) fetch(r, v[r]);
    }
    // f(round, the lane's eight values), values as they are in the row or normalised
    float inv = 1.f;
    bool norm = false;
    auto each = [&](auto f) {
#pragma unroll
        for (int r = 0; r < (NIT ? NIT : 1 << 30); ++r) {
            if (NIT == 0 && r >= rounds) break;
            float4 (&o)[2] = v[NIT ? r : 0];
            if (NIT == 0) fetch(r, o);
            if (norm) {
                const int b = r * 64 + grp;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float4 w = b < bpr ? __ldg(nr + b * 8 + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                    o[e] = make_float4(__fmul_rn(__fmul_rn(o[e].x, inv), w.x), __fmul_rn(__fmul_rn(o[e].y, inv), w.y), __fmul_rn(__fmul_rn(o[e].z, inv), w.z),
                                       __fmul_rn(__fmul_rn(o[e].w, inv), w.w));
                }
            }
            f(r, o);
        }
    };
    if (norm_w) {
        float ss = 0.f;
        each([&](int, const float4 (&o)[2]) {
#pragma unroll
            for (int e = 0; e < 2; ++e) ss = fmaf(o[e].x, o[e].x, fmaf(o[e].y, o[e].y, fmaf(o[e].z, o[e].z, fmaf(o[e].w, o[e].w, ss))));
        });
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if ((threadIdx.x & 31) == 0) red2[warp] = ss;
        __syncthreads();
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += red2[w];
        inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(t, static_cast<float>(K)), eps)));
    }
    norm = norm_w != nullptr;
    float amax = 0.f;
    each([&](int r, const float4 (&o)[2]) {
        const int b = r * 64 + grp;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (x_norm_out && b < bpr) reinterpret_cast<float4*>(x_norm_out + static_cast<size_t>(m) * K + b * 32)[2 * t4 + e] = o[e];
            amax = max_nan(amax, max_nan(max_nan(fabsf(o[e].x), fabsf(o[e].y)), max_nan(fabsf(o[e].z), fabsf(o[e].w))));
        }
    });
    norm = norm && NIT == 0;               // values in registers are normalised by now
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[warp] = amax;
    __syncthreads();
    amax = red[0];
    for (int w = 1; w < 8; ++w) amax = max_nan(amax, red[w]);
    // 2^e with e = 13 - floor(log2(amax)), as exponent-field arithmetic; rows of zeros, infinities or NaN use 1
    const int ex = static_cast<int>((__float_as_uint(amax) >> 23) & 0xffu);
    int field = 267 - ex;
    if (ex == 0 || ex == 255) field = 127;
    field = field < 1 ? 1 : (field > 253 ? 253 : field);
    const float s = __uint_as_float(static_cast<uint32_t>(field) << 23);
    if (threadIdx.x == 0) op.inv_s[m] = __uint_as_float(static_cast<uint32_t>(254 - field) << 23);
    __half* hi = op.a + static_cast<size_t>(m) * K;
    __half* lo = hi + static_cast<size_t>(op.m_pad) * K;
    each([&](int r, const float4 (&o)[2]) {                         // whole warps: the shuffles stay converged
        const int b = r * 64 + grp;
        uint32_t w[2];
        int isum;
        const float d = i8::quantize_block_4lanes(o[0], o[1], w[0], w[1], isum);
        if (b >= bpr) return;
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {                               // values e / 2 * 4 + (e & 1) and two further on
            const uint32_t q = w[e >> 1] >> (8 * (e & 1));
            const float fa = __fmul_rn(__fmul_rn(d, static_cast<float>(static_cast<int8_t>(q & 0xff))), s), fb = __fmul_rn(__fmul_rn(d, static_cast<float>(static_cast<int8_t>((q >> 16) & 0xff))), s);
            const __half2 x2 = __floats2half2_rn(fa, fb);
            h[e] = h2_bits(x2);
            l[e] = h2_bits(__floats2half2_rn(fa - __low2float(x2), fb - __high2float(x2)));
        }
        reinterpret_cast<uint4*>(hi + b * 32)[t4] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4*>(lo + b * 32)[t4] = make_uint4(l[0], l[1], l[2], l[3]);
        if (sums) {
            const float sum = __fmul_rn(__fmul_rn(d, static_cast<float>(isum)), s);
            const __nv_bfloat16 p1 = __float2bfloat16_rn(sum);
            const float r1 = sum - __bfloat162float(p1);
            const __nv_bfloat16 p2 = __float2bfloat16_rn(r1);
            __nv_bfloat16* sp = op.s + static_cast<size_t>(m) * (K / 4) + (b >> 3) * 64 + (b & 7) + 16 * t4;      // g1 g1 | g2 g2 | g1 g3
            if (t4 < 3) {
                sp[0] = t4 == 1 ? p2 : p1;
                sp[8] = t4 == 0 ? p1 : t4 == 1 ? p2 : __float2bfloat16_rn(r1 - __bfloat162float(p2));
            }
        }
    });
}

// Adds up the pieces of every cut tile in k order. Block (t, j): tokens 16 j .. 16 j + 15 of cut tile t, four at a time; a thread has four rows.
template <bool PEERS>
__global__ void __launch_bounds__(256) pair_fixup_kernel(const __grid_constant__ PairParams p, const PairPeers<PEERS> pe) {
    int t = blockIdx.x;
    const int nsb = p.K / 256;
    Seg sg;
    for (sg.mat = 0; t >= p.tiles[sg.mat] - p.whole[sg.mat]; ++sg.mat) t -= p.tiles[sg.mat] - p.whole[sg.mat];
    tile_at(p, p.whole[sg.mat] + t, sg);
    const int units = p.units[sg.mat], cut = p.cut[sg.mat], col = (threadIdx.x & 63) * 4, n = sg.n0 + col, N = p.N[sg.mat];
    // the c that holds unit u is the largest with cut_start(c) <= u
    auto owner = [&](int u) {
        int c = static_cast<int>((static_cast<long long>(u + 1) * cut + units - 1) / units) - 1;
        c = c < 0 ? 0 : c >= cut ? cut - 1 : c;
        while (c + 1 < cut && cut_start(units, cut, c + 1) <= u) ++c;
        while (c > 0 && cut_start(units, cut, c) > u) --c;
        return c;
    };
    const int ca = owner(t * nsb), cb = owner(t * nsb + nsb - 1);
    asm volatile("griddepcontrol.wait;" ::: "memory");        // the pieces are there
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tok0 = blockIdx.y * 16 + (threadIdx.x >> 6);
    if (ca == cb || n >= N) return;
    // two pieces' loads in flight: a short wide matrix has a dozen and more a tile (144 rows, 14336 x 1024: 34.1 us one by one, 32.1 so)
    float4 a[4];
    const float* src = p.part + static_cast<size_t>(p.slot0[sg.mat] + ca + t) * SLOT + tok0 * ROWS + col;
    for (int left = cb - ca + 1; left > 0; left -= 2, src += 2 * SLOT) {
        float4 v[2][4];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (q < left && tok0 + 4 * j < sg.nt) v[q][j] = __ldg(reinterpret_cast<const float4*>(src + q * SLOT + 4 * j * ROWS));
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (q < left) a[j] = q == 0 && left == cb - ca + 1 ? v[q][j] : make_float4(a[j].x + v[q][j].x, a[j].y + v[q][j].y, a[j].z + v[q][j].z, a[j].w + v[q][j].w);
    }
    auto store = [&](float* dst, const float4& v) {
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && n + 4 <= N) {
            *reinterpret_cast<float4*>(dst) = v;
        } else {
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (n + k < N) dst[k] = e[k];
        }
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int tok = tok0 + 4 * j;
        if (tok >= sg.nt) continue;
        if constexpr (PEERS) {
            for (int g = 0; g < pe.n; ++g) store(pe.y[g] + static_cast<size_t>(sg.m0 + tok) * pe.ld + pe.col0 + n, a[j]);
        } else {
            store(p.y[sg.mat] + static_cast<size_t>(sg.m0 + tok) * N + n, a[j]);
        }
    }
}

inline size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

// How the tiles are shared out: as many rounds of whole tiles as every pair gets, the rest cut evenly. A pair takes three super-blocks of
// cut tiles or more, two of tiles that have eight at most if half of the pairs are enough for that (2048 x 2048, 144 rows: three 23.7, two
// 18.9 us, the one-CTA kernel 21.7; with more of them the matrices of one call get into each other's way, 2048 x 5632 + 5632, 190 rows:
// 42.7 -> 49.1 us); up to four a pair the pieces are as few as its work allows, beyond that there is one for every pair (320 rows 4096 x 14336,
// nine at most: 68 pieces 91.4, 74 90.6 us). None are cut unless the longest pair's work shrinks by four super-blocks (some 10 us: adding up
// the pieces is one more launch and 256 KB of partial results written and read for each; 4096 x 14336, 256 rows: whole tiles 56.8, cut for
// a gain of three 63.3 us).
struct PairPlan {
    int tiles_m, m_pad, pairs, cut_tiles, tiles[MAX_MATS], whole[MAX_MATS], units[MAX_MATS], cut[MAX_MATS], shift[MAX_MATS], slot0[MAX_MATS];
    size_t a, s, inv, part, aside;
    size_t total() const { return a + s + inv + part + aside; }
};
PairPlan plan_pair(uint32_t type, int M, int K, const int* ns, int n_mats, int max_pairs, bool allow_cut) {
    PairPlan pl{};
    const int nsb = K / 256;
    pl.tiles_m = (M + TOK - 1) / TOK;
    pl.m_pad = (M + 15) & ~15;               // copies past the last row bring other rows or zeros into columns that nobody reads
    const size_t mp = pl.m_pad;
    pl.a = align256(mp * K * 4); pl.s = type == LAPLACE_TYPE_Q4_K ? align256(mp * K / 2) : 0; pl.inv = align256(mp * 4);
    int at = 0, slots = 0;
    for (int i = 0; i < n_mats; ++i) {
        const int tiles = pl.tiles_m * ((ns[i] + ROWS - 1) / ROWS), rest = tiles % max_pairs;
        int used = rest;
        pl.tiles[i] = pl.whole[i] = tiles;
        pl.shift[i] = at;
        pl.slot0[i] = slots;
        if (allow_cut && rest) {
            const int units = rest * nsb, least = nsb <= 8 && units <= max_pairs ? 2 : 3, even = (units + max_pairs - 1) / max_pairs;
            const int longest = even > least ? even : least, cut = longest > 4 ? max_pairs : (units + longest - 1) / longest;
            if (cut > 1 && nsb - longest >= 4) {
                pl.whole[i] = tiles - rest;
                pl.units[i] = units;
                pl.cut[i] = used = cut;
                pl.cut_tiles += rest;
                slots += cut + rest - 1;
            }
        }
        const int need = tiles >= max_pairs ? max_pairs : used;
        if (need > pl.pairs) pl.pairs = need;
        at = (at + used) % max_pairs;
    }
    if (n_mats > 1) pl.pairs = max_pairs;
    pl.part = static_cast<size_t>(slots) * SLOT * sizeof(float);
    pl.aside = type == LAPLACE_TYPE_Q6_K && nsb > Geo<LAPLACE_TYPE_Q6_K>::CHAIN ? static_cast<size_t>(2 * pl.pairs) * TOK * 128 * sizeof(float) : 0;
    return pl;
}

template <uint32_t TYPE, bool PEERS>
int configure() {
    static int rc = cuda_check(cudaFuncSetAttribute(gemm_pair_kernel<TYPE, PEERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Lay<TYPE>::BYTES)),
                               "cudaFuncSetAttribute gemm_pair");
    return rc;
}
template <uint32_t TYPE, bool PEERS>
int launch_kernels(const PairPlan& pl, const PairMaps& maps, const PairParams& p, const PairPeers<PEERS>& pe, cudaStream_t st) {
    int rc = configure<TYPE, PEERS>();
    if (rc) return rc;
    if ((rc = launch_early(gemm_pair_kernel<TYPE, PEERS>, dim3(2 * pl.pairs), THREADS, Lay<TYPE>::BYTES, st, maps, p, pe))) return rc;
    ctx().launches++;
    if (!pl.cut_tiles) return LAPLACE_OK;
    ctx().launches++;
    return launch_early(pair_fixup_kernel<PEERS>, dim3(pl.cut_tiles, ((p.M < TOK ? p.M : TOK) + 15) / 16), 256, 0, st, p, pe);
}

// pairs of SMs that the chip runs at once
int max_pairs() {
    static int n = 0;
    if (n) return n;
    if (configure<LAPLACE_TYPE_Q4_K, false>()) return 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctx().sm_count / 2 * 2); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Lay<LAPLACE_TYPE_Q4_K>::BYTES; cfg.attrs = attr; cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, gemm_pair_kernel<LAPLACE_TYPE_Q4_K, false>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    n = fit < ctx().sm_count / 2 ? fit : ctx().sm_count / 2;
    return n;
}

}  // namespace

// Whether a call of more than 8 rows runs here (its arguments are those the tile kernels of lp_gemm_sa.cu take).
bool gemm_pair_supports(uint32_t type, int M) {
    return (type == LAPLACE_TYPE_Q4_K || type == LAPLACE_TYPE_Q6_K) && M > 128 && max_pairs() > 0;
}

size_t gemm_pair_scratch(uint32_t type, int M, int K, const int* ns, int n_mats, bool cut) { return plan_pair(type, M, K, ns, n_mats, max_pairs(), cut).total(); }

// Matrices of one type and K against the same rows of x: quantizer (with the optional RMSNorm), one matmul launch over all matrices, and
// one that adds up the pieces of cut tiles. `scratch`: gemm_pair_scratch(..., cut) bytes, 256-byte aligned.
int launch_gemm_pair(uint8_t* scratch, bool cut, const float* x, const float* norm_w, float eps, float* x_norm_out, const uint8_t* const* ws, float* const* ys,
                     const int* ns, int n_mats, uint32_t type, int M, int K, cudaStream_t st, const PeerOut* peers) {
    const PairPlan pl = plan_pair(type, M, K, ns, n_mats, max_pairs(), cut);
    PairOperand op;
    op.a = reinterpret_cast<__half*>(scratch);              scratch += pl.a;
    op.s = reinterpret_cast<__nv_bfloat16*>(scratch);       scratch += pl.s;
    op.inv_s = reinterpret_cast<float*>(scratch);           scratch += pl.inv;
    op.m_pad = pl.m_pad;
    const size_t rb = row_bytes(type, K);
    PairParams p{};
    p.inv_s = op.inv_s; p.err = ctx().d_err;
    p.M = M; p.K = K; p.m_pad = pl.m_pad; p.tiles_m = pl.tiles_m; p.n_mats = n_mats;
    p.rb = static_cast<int>(rb);
    p.part = reinterpret_cast<float*>(scratch);             scratch += pl.part;
    p.aside = reinterpret_cast<float*>(scratch);
    p.by_row = rb % 16 != 0;
    for (int i = 0; i < n_mats; ++i) {
        p.w[i] = ws[i]; p.y[i] = ys ? ys[i] : nullptr; p.N[i] = ns[i];
        p.tiles[i] = pl.tiles[i]; p.whole[i] = pl.whole[i]; p.units[i] = pl.units[i]; p.cut[i] = pl.cut[i]; p.shift[i] = pl.shift[i]; p.slot0[i] = pl.slot0[i];
        if (reinterpret_cast<uintptr_t>(ws[i]) & 15) p.by_row = 1;
    }
    PairMaps maps;
    for (int bk = 0; bk < 4; ++bk) {
        if (!make_map_2d(&maps.a[bk], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, op.a, static_cast<uint64_t>(K), 2ull * pl.m_pad, static_cast<uint64_t>(K) * 2, BKC, 16u << bk,
                         CU_TENSOR_MAP_SWIZZLE_128B, "activations"))
            return LAPLACE_ERR_CUDA;
        maps.s[bk] = maps.a[bk];
        if (type == LAPLACE_TYPE_Q4_K && !make_map_2d(&maps.s[bk], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, op.s, static_cast<uint64_t>(K / 4), static_cast<uint64_t>(pl.m_pad),
                                                      static_cast<uint64_t>(K) / 2, 64, 16u << bk, CU_TENSOR_MAP_SWIZZLE_128B, "block sums"))
            return LAPLACE_ERR_CUDA;
    }
    const uint32_t box = (type == LAPLACE_TYPE_Q4_K ? Geo<LAPLACE_TYPE_Q4_K>::PITCH : Geo<LAPLACE_TYPE_Q6_K>::PITCH) / 4;
    for (int i = 0; i < MAX_MATS; ++i) {
        if (i >= n_mats || p.by_row) { maps.w[i] = i && !p.by_row ? maps.w[0] : maps.a[0]; continue; }
        if (!make_map_2d(&maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, ws[i], rb / 4, static_cast<uint64_t>(ns[i]), rb, box, 128, CU_TENSOR_MAP_SWIZZLE_NONE, "weights"))
            return LAPLACE_ERR_CUDA;
    }
    ctx().launches++;
    const int sums = type == LAPLACE_TYPE_Q4_K ? 1 : 0;
    int rc = K <= 4096 ? launch_early(quantize_pair_kernel<2>, dim3(M), 256, 0, st, x, norm_w, eps, x_norm_out, K, op, sums)
           : K <= 8192 ? launch_early(quantize_pair_kernel<4>, dim3(M), 256, 0, st, x, norm_w, eps, x_norm_out, K, op, sums)
           : K <= 16384 ? launch_early(quantize_pair_kernel<8>, dim3(M), 256, 0, st, x, norm_w, eps, x_norm_out, K, op, sums)
                        : launch_early(quantize_pair_kernel<0>, dim3(M), 256, 0, st, x, norm_w, eps, x_norm_out, K, op, sums);
    if (rc) return rc;
    if (peers) {
        PairPeers<true> pe{};
        for (int r = 0; r < peers->world; ++r) pe.y[r] = peers->y[r];
        pe.n = peers->world; pe.ld = peers->ld; pe.col0 = peers->col0;
        rc = type == LAPLACE_TYPE_Q4_K ? launch_kernels<LAPLACE_TYPE_Q4_K, true>(pl, maps, p, pe, st) : launch_kernels<LAPLACE_TYPE_Q6_K, true>(pl, maps, p, pe, st);
    } else {
        const PairPeers<false> none{};
        rc = type == LAPLACE_TYPE_Q4_K ? launch_kernels<LAPLACE_TYPE_Q4_K, false>(pl, maps, p, none, st) : launch_kernels<LAPLACE_TYPE_Q6_K, false>(pl, maps, p, none, st);
    }
    if (rc) return rc;
    ctx().last_path = 2;
    ctx().last_kernel = KERNEL_ON_PAIRS | (type == LAPLACE_TYPE_Q4_K ? KERNEL_TCGEN05 : KERNEL_TCGEN05_TWO_PIECE);
    return cuda_check(cudaGetLastError(), "gemm_pair launch");
}

}  // namespace lp
