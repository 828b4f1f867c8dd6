// lp_gemm_i8_tiles.cu - more than 32 activation rows on the warp-level int8 instruction: tiles of 128 weight rows x up to 128 tokens.
// Integer block sums from mma.sync (super_block in lp_i8.cuh: one super-block of 32 weight rows x up to 64 tokens per consumer warp), the
// fp32 scale chain in registers. Replaces gemm_int<dot_row_*_int_neon> of Laplace's NEON back-end (src/matmul_simd.cpp:143-342, 432-455) for
// the calls that i8_tiles (lp_gemm_sa.cu) sends here.
// Bound by the FP32 pipe: the chain costs 12 cycles of it per 16 x 8 x 32 products, the MMA 8 cycles of the tensor pipe beside
// it. A producer warp fills three stages of one super-block: the packed rows by one tensor-map tile, the quantized tokens by one bulk copy
// per eight.
// All matrices of a call run in one launch, and one more adds up the pieces of the tiles that several CTAs share. (The last of those CTAs
// adding them up itself would save that launch, but the code of it beside the loop costs the loop registers: Q8_0, 512 rows 2816 x 8448
// 77 -> 90 us.)
#include "lp_i8.cuh"
#include "lp_scratch.cuh"
#include "lp_tc.cuh"

namespace lp {

namespace {

using namespace tc;

constexpr int TW = 128, TT = 128, STAGES = 3, MAX_MATS = 8;

// PARTS consumer warps side by side along the tokens (four along the weight rows), NT tiles of 8 tokens each.
template <uint32_t TYPE> using Geo = i8::GeoWide<TYPE>;
template <uint32_t TYPE> struct Lay {
    static constexpr uint32_t RAW = TW * Geo<TYPE>::PITCH, STAGE = RAW + TT / 8 * i8::Geo<TYPE>::ACT_BYTES,
                              SMEM = 128 + STAGES * STAGE + 16;                        // + read-ahead of the unaligned loads
};

struct TileMaps { CUtensorMap w[MAX_MATS]; };
struct TileParams {
    const uint8_t* img;            // quantized rows in fragment order (lp_i8.cuh)
    int*         err;
    float*       part;             // partial results: [slot][TT][TW]
    int          M, K, tiles_m, n_mats;
    int          n_dst, ld, col0;  // 0, or a row-split matrix: y are n_dst GPUs' buffers, rows of ld floats, this slice from column col0 on
    float*       y[MAX_MATS];
    int          N[MAX_MATS];
    // How a matrix's tiles (weight rows outside, tokens inside) are shared out, by its own size alone, so that it has the same bits alone and
    // beside others: the first `whole` are dealt round-robin from CTA `shift` on; of those behind, the super-blocks (`units` in tile order)
    // go evenly to the `cut` CTAs from there on; the c-th CTA's piece of the t-th cut tile is the matrix's partial result c + t (from one
    // piece to the next c or t grows, or both).
    int          whole[MAX_MATS], units[MAX_MATS], tiles[MAX_MATS], cut[MAX_MATS], shift[MAX_MATS], slot0[MAX_MATS];
};
struct Seg { int mat, m0, n0, nt, sb0, sb1, part; };      // nt: tokens
__host__ __device__ __forceinline__ int cut_start(int units, int ctas, int c) { return static_cast<int>(static_cast<long long>(units) * c / ctas); }
__device__ __forceinline__ void tile_at(const TileParams& p, int t, Seg& s) {
    s.m0 = (t % p.tiles_m) * TT;
    s.nt = p.M - s.m0 < TT ? p.M - s.m0 : TT;
    s.n0 = (t / p.tiles_m) * TW;
}
// Piece i of this CTA's work, in the order in which the producer and the consumers walk it; false: there are no more.
__device__ __forceinline__ bool segment(const TileParams& p, int i, Seg& s) {
    const int ctas = static_cast<int>(gridDim.x), nsb = p.K / 256;
    for (s.mat = 0; s.mat < p.n_mats; ++s.mat) {
        int v = static_cast<int>(blockIdx.x) - p.shift[s.mat];
        if (v < 0) v += ctas;
        const int whole = p.whole[s.mat], n_whole = v < whole ? (whole - v + ctas - 1) / ctas : 0;
        s.part = -1;
        if (i < n_whole) {
            s.sb0 = 0; s.sb1 = nsb;
            tile_at(p, v + i * ctas, s);
            return true;
        }
        i -= n_whole;
        if (v < p.cut[s.mat]) {
            const int u0 = cut_start(p.units[s.mat], p.cut[s.mat], v), u1 = cut_start(p.units[s.mat], p.cut[s.mat], v + 1);
            const int first = u0 / nsb, last = (u1 - 1) / nsb, t = first + i;
            if (t <= last) {
                s.sb0 = t == first ? u0 - first * nsb : 0;
                s.sb1 = t == last ? u1 - last * nsb : nsb;
                if (s.sb0 > 0 || s.sb1 < nsb) s.part = p.slot0[s.mat] + v + t;
                tile_at(p, whole + t, s);
                return true;
            }
            i -= last - first + 1;
        }
    }
    return false;
}

// PEERS (a row-split matrix's results, to every GPU's buffer): a template parameter, since as a run-time loop the stores cost the loop above
// registers (512 rows 2816 x 8448 Q8_0 75.7 -> 80.8 us).
template <uint32_t TYPE, int PARTS, int NT, bool PEERS>
__global__ void __launch_bounds__((4 * PARTS + 1) * 32, 1) gemm_i8_tile_kernel(const __grid_constant__ TileMaps maps, const __grid_constant__ TileParams p) {
    using G = Geo<TYPE>;
    constexpr int PITCH = G::PITCH, CONSUMERS = 4 * PARTS;
    extern __shared__ __align__(128) uint8_t smem[];
    static_assert(Lay<TYPE>::SMEM <= 227 * 1024, "shared memory budget");
    const uint32_t sbase = smem_u32(smem), stage0 = sbase + 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto bar_full = [&](int s) { return sbase + 8 * s; };
    auto bar_empty = [&](int s) { return sbase + 32 + 8 * s; };
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), CONSUMERS); }
        fence_barrier_init();
    }
    __syncthreads();
    // the quantized tokens are the kernel's before this one, which this one's launch and set-up overlap
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int nsb = p.K / 256;
    Seg sg;

    if (warp == CONSUMERS) {
        int s = 0, issued = 0;
        uint32_t phase = 0;
        bool gave_up = false;
        for (int i = 0; !gave_up && segment(p, i, sg); ++i) {
            const int nt = (sg.nt + 7) >> 3;
            const uint8_t* act = p.img + static_cast<size_t>(sg.m0 >> 3) * nsb * G::ACT_BYTES;
            for (int sb = sg.sb0; sb < sg.sb1; ++sb) {
                bool free = true;
                if (issued >= STAGES && lane == 0) free = mbar_wait_bounded(bar_empty(s), phase ^ 1);
                if (!__shfl_sync(0xffffffffu, free, 0)) { gave_up = true; break; }
                const uint32_t st = stage0 + s * Lay<TYPE>::STAGE;
                if (lane == 0) {
                    mbar_expect_tx(bar_full(s), Lay<TYPE>::RAW + nt * G::ACT_BYTES);
                    tma_load_2d(st, &maps.w[sg.mat], G::first_word(sb), sg.n0, bar_full(s));
                }
                __syncwarp();
                if (lane < nt)
                    bulk_g2s(st + Lay<TYPE>::RAW + lane * G::ACT_BYTES, act + (static_cast<size_t>(lane) * nsb + sb) * G::ACT_BYTES, G::ACT_BYTES, bar_full(s));
                ++issued;
                if (++s == STAGES) { s = 0; phase ^= 1; }
            }
        }
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        if (gave_up && lane == 0) report_status(p.err, DEV_TIMEOUT_EMPTY);
        // the copies in flight land before the CTA gives its shared memory back
        const int pending = issued < STAGES ? issued : STAGES;
        for (int k = 0; k < pending; ++k) {
            if (s == 0) { s = STAGES; phase ^= 1; }
            --s;
            if (!mbar_wait_bounded(bar_full(s), phase) && lane == 0) report_status(p.err, DEV_TIMEOUT_DRAIN);
        }
        return;
    }

    const int wm = warp & 3, side = warp >> 2, gq = lane >> 2, tq = lane & 3;
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int i = 0; ok && segment(p, i, sg); ++i) {
        const int nt = (sg.nt + 7) >> 3, first = nt * side / PARTS;                     // 8-token tiles: of the tile, before this warp's
        const int live = nt * (side + 1) / PARTS - first;
        float2 acc[1][2][NT][2];
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int t = 0; t < NT; ++t) acc[0][g][t][0] = acc[0][g][t][1] = make_float2(0.f, 0.f);
        for (int sb = sg.sb0; sb < sg.sb1; ++sb) {
            if (!mbar_wait_bounded(bar_full(s), phase)) { ok = false; break; }
            const uint32_t st = stage0 + s * Lay<TYPE>::STAGE;
            const uint32_t row = st + (32 * wm + gq) * PITCH + G::offset_in_unit(sb, 0), act = st + Lay<TYPE>::RAW + first * G::ACT_BYTES;
            // a full tile's count known where the code is built lets the MMAs of one 8-token tile run under the chain of another
            // (512 rows 2816 x 8448 Q8_0 84 -> 76 us); for eight tiles only for the types that run full tiles here, and not for every count:
            // the instruction fetches cost more than it gives (Q4_K, 64 rows: 44.9 against 47.3 us)
            if ((NT <= 4 || TYPE == LAPLACE_TYPE_Q8_0 || TYPE == LAPLACE_TYPE_Q4_0) && live == NT) i8::super_block<TYPE, PITCH, 2, NT>(row, act, G::ACT_BYTES, lane, NT, acc);
            else i8::super_block<TYPE, PITCH, 2, NT>(row, act, G::ACT_BYTES, lane, live, acc);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty(s));
            if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        if (!ok) break;
        // lane: weight rows gq and gq + 8 of two groups of 16, tokens 2 tq and 2 tq + 1 of every eight
        const int N = p.N[sg.mat];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            if (t >= live) break;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = 8 * (first + t) + 2 * tq + e;
                if (col >= sg.nt) continue;
                const float v[4] = {e ? acc[0][0][t][0].y : acc[0][0][t][0].x, e ? acc[0][0][t][1].y : acc[0][0][t][1].x, e ? acc[0][1][t][0].y : acc[0][1][t][0].x, e ? acc[0][1][t][1].y : acc[0][1][t][1].x};
                if (sg.part >= 0) {
                    float* part = p.part + static_cast<size_t>(sg.part) * (TT * TW) + col * TW + 32 * wm + gq;
#pragma unroll
                    for (int k = 0; k < 4; ++k) part[8 * k] = v[k];
                    continue;
                }
                const int n = sg.n0 + 32 * wm + gq;
                auto store = [&](float* y) {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (n + 8 * k < N) y[8 * k] = v[k];
                };
                if constexpr (PEERS) {
                    for (int g = 0; g < p.n_dst; ++g) store(p.y[g] + static_cast<size_t>(sg.m0 + col) * p.ld + p.col0 + n);
                } else {
                    store(p.y[sg.mat] + static_cast<size_t>(sg.m0 + col) * N + n);
                }
            }
        }
    }
    if (!ok && lane == 0) report_status(p.err, DEV_TIMEOUT_FULL);       // the producer drains the copies
}

// Adds up the pieces of every cut tile in k order. Block (t, j): tokens 16 j .. 16 j + 15 of cut tile t, eight at a time; a thread has four rows.
__global__ void __launch_bounds__(256) tile_fixup_kernel(const __grid_constant__ TileParams p) {
    int t = blockIdx.x;
    const int nsb = p.K / 256;
    Seg sg;
    for (sg.mat = 0; t >= p.tiles[sg.mat] - p.whole[sg.mat]; ++sg.mat) t -= p.tiles[sg.mat] - p.whole[sg.mat];
    tile_at(p, p.whole[sg.mat] + t, sg);
    const int units = p.units[sg.mat], cut = p.cut[sg.mat], r = (threadIdx.x & 31) * 4, n = sg.n0 + r, N = p.N[sg.mat], ld = p.n_dst ? p.ld : N;
    // the c that holds unit u is the largest with cut_start(c) <= u
    auto owner = [&](int u) {
        int c = static_cast<int>((static_cast<long long>(u + 1) * cut + units - 1) / units) - 1;
        c = c < 0 ? 0 : c >= cut ? cut - 1 : c;
        while (c + 1 < cut && cut_start(units, cut, c + 1) <= u) ++c;
        while (c > 0 && cut_start(units, cut, c) > u) --c;
        return c;
    };
    const int ca = owner(t * nsb), cb = owner(t * nsb + nsb - 1), tok0 = blockIdx.y * 16 + (threadIdx.x >> 5);
    asm volatile("griddepcontrol.wait;" ::: "memory");        // the pieces are there
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (ca == cb || n >= N) return;
    // four pieces' loads in flight
    float4 a[2];
    const float* src = p.part + static_cast<size_t>(p.slot0[sg.mat] + ca + t) * (TT * TW) + tok0 * TW + r;
    for (int left = cb - ca + 1; left > 0; left -= 4, src += 4 * TT * TW) {
        float4 v[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (q < left && tok0 + 8 * j < sg.nt) v[q][j] = __ldg(reinterpret_cast<const float4*>(src + q * TT * TW + 8 * j * TW));
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (q < left) a[j] = q == 0 && left == cb - ca + 1 ? v[q][j] : make_float4(a[j].x + v[q][j].x, a[j].y + v[q][j].y, a[j].z + v[q][j].z, a[j].w + v[q][j].w);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int tok = tok0 + 8 * j;
        if (tok >= sg.nt) continue;
        for (int g = 0; g < max(p.n_dst, 1); ++g) {
            float* y = p.y[p.n_dst ? g : sg.mat] + static_cast<size_t>(sg.m0 + tok) * ld + p.col0 + n;
            if ((reinterpret_cast<uintptr_t>(y) & 15) == 0 && n + 4 <= N) {
                *reinterpret_cast<float4*>(y) = a[j];
            } else {
                const float e[4] = {a[j].x, a[j].y, a[j].z, a[j].w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (n + k < N) y[k] = e[k];
            }
        }
    }
}

inline size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

// How the tiles are shared out: as many rounds of whole tiles as every CTA gets, the rest cut evenly; a CTA takes no less than two
// super-blocks of cut tiles. Up to four super-blocks a CTA the pieces are as few as its work allows (Q8_0, 120 rows 1536 x 8960: 148 pieces of
// three at most 26.1, 140 of three 21.7 us; 77 rows 14336 x 1024: 25.5 and 24.0; but Q6_K, 96 rows 4096 x 14336: 148 of thirteen at most 90.6,
// 138 of thirteen 102). Tiles are cut if that gives each two CTAs or shortens the longest CTA's work by three super-blocks: pieces of many
// tiles cost more than two are worth (512 rows 4096 x 4096 Q8_0, 128 tiles: cut 57.3, whole 54.9 us; 200 rows 2816 x 8448 44.2 and 40.8; 128
// rows 4096 x 14336, a gain of three: 53.8 and 54.9). Where the last tokens' tiles are much smaller, whole tiles leave the CTAs unequal work,
// and all are cut: a super-block costs some 62 + its tokens (Q8_0 4096 x 14336: 33 rows 31 us, 64 39, 96 45, 128 54), and the line lies at two
// full super-blocks of difference (140 rows 4096 x 14336 twice: whole rounds 166, all cut 148 us).
struct TilePlan {
    int tiles_m, ctas, cut_tiles, most_tokens, tiles[MAX_MATS], whole[MAX_MATS], units[MAX_MATS], cut[MAX_MATS], shift[MAX_MATS], slot0[MAX_MATS];
    size_t img, part;
    size_t total() const { return img + part; }
};
TilePlan plan_tiles(uint32_t type, int M, int K, const int* ns, int n_mats, bool allow_cut) {
    TilePlan pl{};
    const int nsb = K / 256, sms = ctx().sm_count;
    pl.tiles_m = (M + TT - 1) / TT;
    pl.img = align256(static_cast<size_t>((M + 7) / 8) * nsb * gemm_i8_act_bytes(type));
    const int full = 62 + TT, mean = pl.tiles_m == 1 ? full : ((pl.tiles_m - 1) * full + 62 + M - (pl.tiles_m - 1) * TT) / pl.tiles_m;       // work of a super-block
    int at = 0, slots = 0;
    for (int i = 0; i < n_mats; ++i) {
        const int tiles = pl.tiles_m * ((ns[i] + TW - 1) / TW);
        int rest = tiles % sms;
        const bool uneven = rest && static_cast<long long>(tiles / sms) * nsb * (full - mean) >= 2 * full;
        if (uneven && allow_cut) rest = tiles;
        int used = rest;
        pl.tiles[i] = pl.whole[i] = tiles;
        pl.shift[i] = at;
        pl.slot0[i] = slots;
        if (rest && allow_cut) {
            const int units = rest * nsb, even = (units + sms - 1) / sms, longest = even > 2 ? even : 2;
            const int cut = longest > 4 ? sms : (units + longest - 1) / longest;
            if (uneven || cut >= 2 * rest || (cut > rest && nsb - longest >= 3)) {
                pl.whole[i] = tiles - rest;
                pl.units[i] = units;
                pl.cut[i] = used = cut;
                slots += cut + rest - 1;
                pl.cut_tiles += rest;
            }
        }
        const int need = pl.whole[i] >= sms ? sms : used;
        if (need > pl.ctas) pl.ctas = need;
        at = (at + used) % sms;
    }
    if (n_mats > 1) pl.ctas = sms;
    pl.most_tokens = M < TT ? M : TT;
    pl.part = static_cast<size_t>(slots) * TT * TW * sizeof(float);
    return pl;
}

template <uint32_t TYPE, int PARTS, int NT, bool PEERS>
int launch_as(const TilePlan& pl, const TileMaps& maps, const TileParams& p, cudaStream_t st) {
    static const int rc = cuda_check(cudaFuncSetAttribute(gemm_i8_tile_kernel<TYPE, PARTS, NT, PEERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Lay<TYPE>::SMEM)),
                                     "cudaFuncSetAttribute gemm_i8_tile");
    if (rc) return rc;
    return launch_early(gemm_i8_tile_kernel<TYPE, PARTS, NT, PEERS>, dim3(pl.ctas), (4 * PARTS + 1) * 32, Lay<TYPE>::SMEM, st, maps, p);
}
// Up to 96 rows: three warps side by side with up to four 8-token tiles each, whose counts are known where the code is built; their 12 warps
// hide more latency than eight (Q8_0, 77 rows 2816 x 8448 26.9 -> 25.1 us, x 1024 17.4 -> 15.4; 16 warps of up to three tiles unpack every
// weight once more, 26.8 and 17.2). Q6_K's unpacking takes the registers that 12 warps have (77 rows 14336 x 4096 90 -> 118 us), and so do
// the accumulators of more rows (512 rows, 12 warps of up to six tiles, 83.6 -> 87.5 us).
template <uint32_t TYPE>
int launch_type(const TilePlan& pl, const TileMaps& maps, const TileParams& p, cudaStream_t st) {
    if constexpr (TYPE != LAPLACE_TYPE_Q6_K) {
        if (p.M <= 96) return p.n_dst ? launch_as<TYPE, 3, 4, true>(pl, maps, p, st) : launch_as<TYPE, 3, 4, false>(pl, maps, p, st);
    }
    return p.n_dst ? launch_as<TYPE, 2, 8, true>(pl, maps, p, st) : launch_as<TYPE, 2, 8, false>(pl, maps, p, st);
}

}  // namespace

size_t gemm_i8_tiles_scratch(uint32_t type, int M, int K, const int* ns, int n_mats, bool cut) { return plan_tiles(type, M, K, ns, n_mats, cut).total(); }

// Matrices of one type and K against the same rows of x: quantizer (with the optional RMSNorm) and one matmul launch over all matrices.
// `scratch`: gemm_i8_tiles_scratch(..., cut) bytes, 256-byte aligned.
int launch_gemm_i8_tiles(uint8_t* scratch, bool cut, const float* x, const float* norm_w, float eps, float* x_norm_out, const uint8_t* const* ws, float* const* ys,
                         const int* ns, int n_mats, uint32_t type, int M, int K, cudaStream_t st, const PeerOut* peers) {
    const TilePlan pl = plan_tiles(type, M, K, ns, n_mats, cut);
    TileParams p{};
    p.img = scratch;                                        scratch += pl.img;
    p.part = reinterpret_cast<float*>(scratch);
    p.err = ctx().d_err; p.M = M; p.K = K; p.tiles_m = pl.tiles_m; p.n_mats = n_mats;
    if (peers) { p.n_dst = peers->world; p.ld = peers->ld; p.col0 = peers->col0; }
    for (int i = 0; i < n_mats; ++i) {
        p.y[i] = ys ? ys[i] : nullptr; p.N[i] = ns[i];
        p.tiles[i] = pl.tiles[i]; p.whole[i] = pl.whole[i]; p.units[i] = pl.units[i]; p.cut[i] = pl.cut[i]; p.shift[i] = pl.shift[i]; p.slot0[i] = pl.slot0[i];
    }
    if (peers)
        for (int r = 0; r < peers->world; ++r) p.y[r] = peers->y[r];
    int pitch;
    switch (type) {
        case LAPLACE_TYPE_Q4_K: pitch = Geo<LAPLACE_TYPE_Q4_K>::PITCH; break;
        case LAPLACE_TYPE_Q4_0: pitch = Geo<LAPLACE_TYPE_Q4_0>::PITCH; break;
        case LAPLACE_TYPE_Q8_0: pitch = Geo<LAPLACE_TYPE_Q8_0>::PITCH; break;
        default: pitch = Geo<LAPLACE_TYPE_Q6_K>::PITCH; break;
    }
    const uint64_t rb = row_bytes(type, K);
    TileMaps maps;
    for (int i = 0; i < MAX_MATS; ++i) {
        if (i >= n_mats) { maps.w[i] = maps.w[0]; continue; }
        if (!make_map_2d(&maps.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, ws[i], rb / 4, static_cast<uint64_t>(ns[i]), rb, pitch / 4, TW, CU_TENSOR_MAP_SWIZZLE_NONE, "weights"))
            return LAPLACE_ERR_CUDA;
    }
    int rc = launch_quantize_i8(x, norm_w, eps, x_norm_out, type, M, K, const_cast<uint8_t*>(p.img), st);
    if (rc) return rc;
    switch (type) {
        case LAPLACE_TYPE_Q4_K: rc = launch_type<LAPLACE_TYPE_Q4_K>(pl, maps, p, st); break;
        case LAPLACE_TYPE_Q4_0: rc = launch_type<LAPLACE_TYPE_Q4_0>(pl, maps, p, st); break;
        case LAPLACE_TYPE_Q8_0: rc = launch_type<LAPLACE_TYPE_Q8_0>(pl, maps, p, st); break;
        default: rc = launch_type<LAPLACE_TYPE_Q6_K>(pl, maps, p, st); break;
    }
    if (rc) return rc;
    ctx().launches++;
    if (pl.cut_tiles) {
        if ((rc = launch_early(tile_fixup_kernel, dim3(pl.cut_tiles, (pl.most_tokens + 15) / 16), 256, 0, st, p))) return rc;
        ctx().launches++;
    }
    ctx().last_path = 2;
    ctx().last_kernel = KERNEL_INT8_TILES;
    return cuda_check(cudaGetLastError(), "gemm_i8_tile launch");
}

}  // namespace lp
