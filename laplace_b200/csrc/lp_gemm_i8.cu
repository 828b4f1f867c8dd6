// lp_gemm_i8.cu - matmul with a handful of activation rows (2..32), and mixture-of-experts calls with a handful of tokens per
// expert, on the warp-level int8 tensor-core instruction. Replaces gemm_int<dot_row_*> of Laplace's NEON back-end
// (src/matmul_simd.cpp:143-342, 432-455) for Q4_0, Q8_0, Q4_K and Q6_K weights in that range.
//
// The path streams every weight byte once and is bound by HBM as long as the arithmetic keeps up: one
// mma.sync.m16n8k32 forms the integer block sums U of 16 weight rows x 8 activation rows x one 32-value block (Q6_K: two k16
// instructions, its scales cover 16 values), bit for bit the reference's integers, and a fp32 chain follows per block,
//   acc += U * ((d * sc) * d_x)        (and, Q4_K, acc += (-dmin * mn) * sum_x),
// two activation rows per packed instruction. The accumulator operand of the MMA is the bit pattern of 1.5 * 2^23, so that the
// integer result read as a float is 1.5 * 2^23 + U exactly (|U| < 2^22): one packed subtraction instead of two conversions.
//
// Shape of the kernel (one CTA per SM, sixteen consumer warps, two copy warps, two that add up):
//   * K is cut over a cluster of up to eight CTAs, so that a CTA needs its part of the quantized activations only (they stay
//     in shared memory for the whole call) and a long-K matrix with few rows still occupies every SM. The cut depends on
//     K, type and row count (see plan_dense), so a matrix has the same bits alone and beside others on this kernel;
//   * every consumer warp takes groups of 16 weight rows for itself (two warps share a group when the CTA's part of K is
//     eight super-blocks or more): its copies are 2-D tensor-map tiles of 16 rows x one or two super-blocks into a ring of
//     its own, so that warps never wait for one another while they stream;
//   * the partial results of a row group go to one CTA of the cluster by asynchronous stores that a barrier there counts (no fence,
//     no wait on the sender's side); two warps of that CTA add them up in a fixed order and write them once, while the others
//     stream on. With all warps of the cluster meeting after every sixteen to thirty-two row groups instead, a quarter of the
//     warps' time went into that (24 rows, Q4_K 4096 x 28672: 36 % of the issue slots used): 46.1 -> 32.9 us, 16 rows 36.5 -> 25.7,
//     8 rows 20.1 -> 18.8, Q6_K 14336 x 4096, 24 rows 40.6 -> 38.2. One adding warp: 34.3, 27.3 and 21.1 us. No scratch in device
//     memory and no second launch;
//   * with up to 8 activation rows every CTA quantizes its part of the rows itself (with the RMSNorm in front when asked for,
//     the row sums meeting through distributed shared memory); with more rows, and for experts, a small kernel writes the
//     quantized rows in fragment order into device scratch and the CTAs fetch their part with bulk copies.
// Every wait is bounded; a wait that gives up raises the status word and the CTA drains its copies and leaves.
#include "lp_i8.cuh"
#include "lp_scratch.cuh"
#include "lp_tc.cuh"

namespace lp {
namespace {

using namespace i8;

constexpr int CW = 16;                     // consumer warps
constexpr int PW = 2;                      // copy warps: lane l of warp i serves consumer warp 8 i + l
constexpr int THREADS = (CW + PW) * 32;
constexpr int MAX_SLOTS = 8;
constexpr int MAX_MATS = 8;
constexpr int MAX_PARTS = 8;               // row groups whose partial results a CTA of a cluster holds at a time
constexpr int RW = 2;                      // warps of a CTA that add up, group i of the CTA's by warp i mod RW
constexpr int PART_BYTES = 512;            // partial results of 16 weight rows x 8 activation rows, in the order in which the lanes hold them

// Shared memory: barriers, row sums of the norm, then the activations, the partial results, the rings.
constexpr uint32_t OFF_BAR_FULL = 0, OFF_BAR_EMPTY = OFF_BAR_FULL + CW * MAX_SLOTS * 8, OFF_BAR_MISC = OFF_BAR_EMPTY + CW * MAX_SLOTS * 8,
                   OFF_RED = OFF_BAR_MISC + 256, OFF_ACT = OFF_RED + 128;
static_assert(OFF_ACT % 128 == 0, "bulk copies land on 128-byte boundaries");
// inside OFF_BAR_MISC; BAR_ACT*: two each, BAR_PART: MAX_PARTS, TAKEN: RW words for every CTA of the cluster
constexpr uint32_t BAR_ACT = 0, BAR_ACT_EMPTY = 16, BAR_NORM = 32, BAR_NORM_READ = 40, BAR_PART = 64, TAKEN = BAR_PART + 8 * MAX_PARTS;
static_assert(RW == 2 && MAX_PARTS % RW == 0, "places are dealt to the adding warps");
static_assert(TAKEN + 8 * RW * 4 <= 256, "barrier area");

struct I8Params {
    const float*   x;              // M <= 8: fp32 rows, quantized by every CTA
    const float*   norm_w;         // optional RMSNorm in front (M <= 8)
    float          norm_eps;
    float*         x_norm_out;
    const uint8_t* img;            // quantized rows in fragment order (more rows, experts): [tile of 8 rows][K / 256][i8::act_bytes]
    int*           err;
    int            M, K, nsb;
    int            n_mats;
    float*         mat_y[MAX_MATS];
    int            mat_end[MAX_MATS];      // rows of the matrices one behind the other: where each ends
    int            total_rows;
    int            kw;                     // warps that share a row group
    int            n_parts;                // row groups whose partial results shared memory holds: 1 or a multiple of RW, at most MAX_PARTS
    uint32_t       off_part, off_ring;
    int            n_slots;
    // experts
    const int4*    tile_tab;               // {first activation row, first weight row inside the expert, the expert's first row, tokens}
    const int*     n_tiles_dev;
    const int*     out_row;                // activation row -> row of y (-1: padding)
    int            out_identity;           // 1: a live activation row r is written to row r of y
    int            N;
    int            act_bufs;               // activation buffers (2: the next job's tile is fetched early)
    uint32_t       act_buf_bytes;
};
struct I8Maps { CUtensorMap w[MAX_MATS]; };

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_remote(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(addr) : "memory");
}
__device__ __forceinline__ float ld_remote(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// 16 bytes into another CTA's shared memory, counted by a barrier there: no fence, nothing to wait for on this side
__device__ __forceinline__ void st_remote_counted(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%2, %3, %4, %5}, [%1];"
                 :: "r"(addr), "r"(bar), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
        if (ok) return true;
    }
    return false;
}

__device__ __forceinline__ bool wait_taken(uint32_t addr, int count) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        int v;
        asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
        if (v >= count) return true;
        if (it > 16) __nanosleep(200);
    }
    return false;
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
    const uint4 v = lds128(addr);
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// The row groups of rows [r0, r1) of the concatenated ones, 16 rows each, cut at matrix boundaries.
struct Group { int mat, row, rows; };              // matrix, first row inside it, live rows
__device__ __forceinline__ int row_groups(const I8Params& p, int r0, int r1) {
    int n = 0;
    for (int i = 0, b = 0; i < p.n_mats; ++i) {
        const int lo = r0 > b ? r0 : b, hi = r1 < p.mat_end[i] ? r1 : p.mat_end[i];
        if (hi > lo) n += (hi - lo + 15) >> 4;
        b = p.mat_end[i];
    }
    return n;
}
__device__ __forceinline__ Group row_group(const I8Params& p, int r0, int r1, int g) {
    for (int i = 0, b = 0; i < p.n_mats; ++i) {
        const int lo = r0 > b ? r0 : b, hi = r1 < p.mat_end[i] ? r1 : p.mat_end[i];
        if (hi > lo) {
            const int n = (hi - lo + 15) >> 4;
            if (g < n) { const int at = lo + 16 * g; return {i, at - b, hi - at < 16 ? hi - at : 16}; }
            g -= n;
        }
        b = p.mat_end[i];
    }
    return {0, 0, 0};
}

// QUANT: the CTA quantizes the (at most 8) activation rows itself. MOE: jobs from the table, whole K, results straight to y.
template <uint32_t TYPE, int NT, int C, bool QUANT, bool MOE>
__global__ void __launch_bounds__(THREADS + (C > 1 ? 32 * RW : 0), 1) gemm_i8_kernel(const __grid_constant__ I8Maps maps, const I8Params p) {
    using G = Geo<TYPE>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0;
    auto bar_full = [&](int w, int s) { return sbase + OFF_BAR_FULL + (w * MAX_SLOTS + s) * 8; };
    auto bar_empty = [&](int w, int s) { return sbase + OFF_BAR_EMPTY + (w * MAX_SLOTS + s) * 8; };
    auto misc = [&](uint32_t b) { return sbase + OFF_BAR_MISC + b; };
    auto ring_of = [&](int w) { return sbase + p.off_ring + static_cast<uint32_t>(w) * p.n_slots * G::UNIT_BYTES; };

    if (threadIdx.x < CW) {
        for (int s = 0; s < p.n_slots; ++s) { mbar_init(bar_full(threadIdx.x, s), 1); mbar_init(bar_empty(threadIdx.x, s), 1); }
    }
    if (threadIdx.x == CW) {
        for (int b = 0; b < 2; ++b) { mbar_init(misc(BAR_ACT + 8 * b), 1); mbar_init(misc(BAR_ACT_EMPTY + 8 * b), CW); }
        mbar_init(misc(BAR_NORM), C);
        mbar_init(misc(BAR_NORM_READ), C);
        for (int b = 0; b < MAX_PARTS; ++b) mbar_init(misc(BAR_PART + 8 * b), 1);
        for (int r = 0; r < C * RW; ++r) reinterpret_cast<volatile uint32_t*>(smem + OFF_BAR_MISC + TAKEN)[r] = 0u;
    }
    fence_barrier_init();
    __syncthreads();
    if constexpr (C > 1) {            // the barriers exist before another CTA of the cluster arrives on them
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    // dense: this cluster's contiguous share of the rows, this CTA's part of K, this warp's part of that
    const int clusters = gridDim.x / C, cl = blockIdx.x / C;
    const int r0 = MOE ? 0 : static_cast<int>(static_cast<long long>(p.total_rows) * cl / clusters);
    const int r1 = MOE ? 0 : static_cast<int>(static_cast<long long>(p.total_rows) * (cl + 1) / clusters);
    const int sb0 = p.nsb * rank / C, sb1 = p.nsb * (rank + 1) / C;
    const int lanes = CW / p.kw;                                   // row groups in work at a time

    if (C > 1 && warp >= CW + PW) {
        // ------------------------------ adds up the partial results of the cluster: row groups rank, rank + C, ... ------------------------------
        // [group in work][rank and warp they come from][tile][lane]; a barrier counts a group's bytes. The consumer warps go on meanwhile.
        const int ng = row_groups(p, r0, r1), n = ng > rank ? (ng - rank + C - 1) / C : 0, n_src = C * p.kw;
        const uint32_t src_bytes = NT * PART_BYTES, group_bytes = static_cast<uint32_t>(n_src) * src_bytes;
        const int gq = lane >> 2, tq = lane & 3, rw = warp - (CW + PW), step = p.n_parts == 1 ? 1 : RW;
        // a place always belongs to the same warp, which meets every phase of its barrier
        if (lane < p.n_parts && lane < n && lane % step == rw) mbar_expect_tx(misc(BAR_PART + 8 * lane), group_bytes);
        __syncwarp();
        asm volatile("griddepcontrol.wait;" ::: "memory");             // y may be read by the kernel before this one
        bool ok = true;
        for (int i = rw, at = rw, phase = 0; rw < step && i < n; i += step) {
            const uint32_t src = sbase + p.off_part + static_cast<uint32_t>(at) * group_bytes + lane * 16;
            const Group gr = row_group(p, r0, r1, i * C + rank);
            const size_t ld = p.mat_end[gr.mat] - (gr.mat ? p.mat_end[gr.mat - 1] : 0);
            float* y = p.mat_y[gr.mat] + gr.row + gq;
            if (!wait_cluster(misc(BAR_PART + 8 * at), phase)) { ok = false; break; }
            float4 v[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                float4 part[C];                                        // of the CTAs, added in pairs
#pragma unroll
                for (int r = 0; r < C; ++r) {
                    const uint32_t a = src + t * PART_BYTES + (p.kw == 2 ? 2 * r : r) * src_bytes;
                    part[r] = lds_f4(a);
                    if (p.kw == 2) part[r] = add4(part[r], lds_f4(a + src_bytes));
                }
#pragma unroll
                for (int o = 1; o < C; o *= 2)
#pragma unroll
                    for (int r = 0; r < C; r += 2 * o) part[r] = add4(part[r], part[r + o]);
                v[t] = part[0];
            }
            __syncwarp();
            if (i + p.n_parts < n) {                                   // the place may take a group further on
                if (lane == 0) mbar_expect_tx(misc(BAR_PART + 8 * at), group_bytes);
                __syncwarp();
                if (lane < C)
                    asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" :: "r"(map_rank(misc(TAKEN + 4 * (rank * RW + rw)), lane)), "r"(i + 1) : "memory");
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int m = 8 * t + 2 * tq;
                float* ym = y + m * ld;
                if (m < p.M) {
                    if (gq < gr.rows) ym[0] = v[t].x;
                    if (gq + 8 < gr.rows) ym[8] = v[t].z;
                }
                if (m + 1 < p.M) {
                    if (gq < gr.rows) ym[ld] = v[t].y;
                    if (gq + 8 < gr.rows) ym[ld + 8] = v[t].w;
                }
            }
            if ((at += step) >= p.n_parts) { at = rw; phase ^= 1; }
        }
        // the other CTAs have read this one's row sums
        if (QUANT && rw == 0 && p.norm_w && !wait_cluster(misc(BAR_NORM_READ), 0)) ok = false;
        if (!ok && lane == 0) report_status(p.err, DEV_TIMEOUT_FULL);
        return;
    }
    if (warp >= CW) {
        // ------------------------------ copy warps: a lane walks the units of one consumer warp ------------------------------
        if constexpr (MOE) asm volatile("griddepcontrol.wait;" ::: "memory");        // the job table is written by the kernel before
        const int w = (warp - CW) * (CW / PW) + lane;
        const bool serving = lane < CW / PW;
        const bool act_lane = !QUANT && warp == CW + PW - 1 && lane == CW / PW;       // fetches the quantized rows
        bool gave_up = false;
        int ui = 0;
        if (serving) {
            const uint32_t ring = ring_of(w);
            int slot = 0;
            uint32_t phase = 0;
            auto copy = [&](const CUtensorMap* map, int sb, int row) {
                if (ui >= p.n_slots && !mbar_wait_bounded(bar_empty(w, slot), phase ^ 1)) { gave_up = true; return; }
                mbar_expect_tx(bar_full(w, slot), G::UNIT_BYTES);
                tc::tma_load_2d(ring + slot * G::UNIT_BYTES, map, G::first_word(sb), row, bar_full(w, slot));
                ++ui;
                if (++slot == p.n_slots) { slot = 0; phase ^= 1; }
            };
            if constexpr (MOE) {
                const int nt_jobs = *reinterpret_cast<const volatile int*>(p.n_tiles_dev);
                for (int j = blockIdx.x; j < nt_jobs && !gave_up; j += gridDim.x) {
                    const int4 t = __ldg(p.tile_tab + j);
                    if (t.y + 16 * w >= p.N) continue;
                    for (int sb = 0; sb < p.nsb && !gave_up; sb += G::UNIT_SB) copy(&maps.w[0], sb, t.z + t.y + 16 * w);
                }
            } else {
                const int part = w / lanes, gl = w - part * lanes, len = sb1 - sb0;
                const int s0 = sb0 + len * part / p.kw, s1 = sb0 + len * (part + 1) / p.kw;
                const int ng = row_groups(p, r0, r1);
                for (int g = gl; g < ng && !gave_up; g += lanes) {
                    const Group gr = row_group(p, r0, r1, g);
                    for (int sb = s0; sb < s1 && !gave_up; sb += G::UNIT_SB) copy(&maps.w[gr.mat], sb, gr.row);
                }
            }
        } else if (act_lane) {
            const uint32_t tile_bytes = static_cast<uint32_t>(p.nsb) * G::ACT_BYTES;
            if constexpr (MOE) {
                const int nt_jobs = *reinterpret_cast<const volatile int*>(p.n_tiles_dev);
                int jb = 0;
                for (int j = blockIdx.x; j < nt_jobs && !gave_up; j += gridDim.x, ++jb) {
                    const int4 t = __ldg(p.tile_tab + j);
                    const int nt = (t.w + 7) >> 3, buf = jb % p.act_bufs, round = jb / p.act_bufs;
                    if (round > 0 && !mbar_wait_bounded(misc(BAR_ACT_EMPTY + 8 * buf), (round - 1) & 1)) { gave_up = true; break; }
                    mbar_expect_tx(misc(BAR_ACT + 8 * buf), nt * tile_bytes);
                    bulk_g2s(sbase + OFF_ACT + buf * p.act_buf_bytes, p.img + static_cast<size_t>(t.x >> 3) * tile_bytes, nt * tile_bytes, misc(BAR_ACT + 8 * buf));
                }
                // the copies in flight land before the CTA gives its shared memory back
                for (int k = 0; k < p.act_bufs && k < jb; ++k) {
                    const int v = jb - 1 - k;
                    if (!mbar_wait_bounded(misc(BAR_ACT + 8 * (v % p.act_bufs)), (v / p.act_bufs) & 1)) report_status(p.err, DEV_TIMEOUT_DRAIN);
                }
            } else {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                const uint32_t part = static_cast<uint32_t>(sb1 - sb0) * G::ACT_BYTES;
                mbar_expect_tx(misc(BAR_ACT), NT * part);
                for (int t = 0; t < NT && part; ++t)
                    bulk_g2s(sbase + OFF_ACT + t * part, p.img + static_cast<size_t>(t) * tile_bytes + static_cast<size_t>(sb0) * G::ACT_BYTES, part, misc(BAR_ACT));
                if (!mbar_wait_bounded(misc(BAR_ACT), 0)) report_status(p.err, DEV_TIMEOUT_DRAIN);
            }
        }
        __syncwarp();
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // the next kernel may start as SMs free up
        if (gave_up) report_status(p.err, DEV_TIMEOUT_EMPTY);
        if (serving) {
            const int pending = ui < p.n_slots ? ui : p.n_slots;
            for (int k = 0; k < pending; ++k) {
                const int v = ui - 1 - k;
                if (!mbar_wait_bounded(bar_full(w, v % p.n_slots), (v / p.n_slots) & 1)) report_status(p.err, DEV_TIMEOUT_DRAIN);
            }
        }
        return;
    }

    // ------------------------------ consumers ------------------------------
    // x may be produced, and y read, by the kernel before this one in the stream (the weights are not: the copies above start at once)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = true;
    const int gq = lane >> 2, tq = lane & 3;
    if constexpr (QUANT) {
        // quantize this CTA's part of every row, exactly as the reference does (src/matmul_simd.cpp:348-410)
        const int nblk = (sb1 - sb0) * 8, total = p.M * nblk, kb0 = sb0 * 8;
        float inv[8];
        if (p.norm_w) {
            // RMSNorm (src/ops.cpp:34-74): inv = 1 / sqrt(mean(x^2) + eps), x_norm = (x * inv) * w. Two warps per row add up
            // this CTA's part; the parts of the cluster's CTAs are added in rank order.
            const int m = warp & 7, half = warp >> 3;
            float ss = 0.f;
            if (m < p.M) {
                const int n4 = nblk * 8, lo = n4 * half / 2, hi = n4 * (half + 1) / 2;
                const float4* xr = reinterpret_cast<const float4*>(p.x + static_cast<size_t>(m) * p.K + kb0 * 32);
                for (int i = lo + lane; i < hi; i += 32) {
                    const float4 v = __ldg(xr + i);
                    ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            float* red = reinterpret_cast<float*>(smem + OFF_RED);
            if (lane == 0) red[m * 2 + half] = ss;
            named_bar_sync(1, CW * 32);
            if constexpr (C > 1) {
                if (threadIdx.x < C) arrive_remote(map_rank(misc(BAR_NORM), threadIdx.x));
                if (!wait_cluster(misc(BAR_NORM), 0)) ok = false;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float t = 0.f;
                if (i < p.M) {
#pragma unroll
                    for (int r = 0; r < C; ++r) {
                        const uint32_t a = sbase + OFF_RED + i * 8, ra = C > 1 ? map_rank(a, r) : a;
                        t += C > 1 ? ld_remote(ra) + ld_remote(ra + 4) : red[2 * i] + red[2 * i + 1];
                    }
                }
                inv[i] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(t, static_cast<float>(p.K)), p.norm_eps)));
            }
        }
        constexpr int GR = CW * 8, DEPTH = 2;          // 32-value blocks in work at a time, rounds of loads in flight
        const int grp = threadIdx.x >> 2, t4 = threadIdx.x & 3;
        for (int base = 0; base < total; base += GR * DEPTH) {                   // whole warps iterate together
            float4 v[DEPTH][2], nw[DEPTH][2];
#pragma unroll
            for (int i = 0; i < DEPTH; ++i) {
                const int b = base + i * GR + grp;
                const int m = b < total ? b / nblk : 0, kb = kb0 + (b < total ? b - m * nblk : 0);
                const float4* xs = reinterpret_cast<const float4*>(p.x + static_cast<size_t>(m) * p.K + kb * 32) + 2 * t4;
                const float4* ns = reinterpret_cast<const float4*>(p.norm_w + kb * 32) + 2 * t4;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    v[i][e] = b < total ? __ldg(xs + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                    nw[i][e] = p.norm_w ? __ldg(ns + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
#pragma unroll
            for (int i = 0; i < DEPTH; ++i) {
                if (base + i * GR >= total) break;
                const int b = base + i * GR + grp;
                const bool live = b < total;
                const int m = live ? b / nblk : 0, kl = live ? b - m * nblk : 0;
                if (p.norm_w) {
                    float iv = inv[0];
#pragma unroll
                    for (int q = 1; q < 8; ++q) iv = m == q ? inv[q] : iv;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        v[i][e].x = __fmul_rn(__fmul_rn(v[i][e].x, iv), nw[i][e].x); v[i][e].y = __fmul_rn(__fmul_rn(v[i][e].y, iv), nw[i][e].y);
                        v[i][e].z = __fmul_rn(__fmul_rn(v[i][e].z, iv), nw[i][e].z); v[i][e].w = __fmul_rn(__fmul_rn(v[i][e].w, iv), nw[i][e].w);
                        if (p.x_norm_out && cl == 0 && live)
                            reinterpret_cast<float4*>(p.x_norm_out + static_cast<size_t>(m) * p.K + (kb0 + kl) * 32)[2 * t4 + e] = v[i][e];
                    }
                }
                uint32_t w0, w1; int isum;
                const float d = quantize_block_4lanes(v[i][0], v[i][1], w0, w1, isum);
                if (live) store_act<TYPE>(smem + OFF_ACT + (kl >> 3) * G::ACT_BYTES, kl & 7, m, t4, w0, w1, d, isum);
            }
        }
        named_bar_sync(1, CW * 32);
        if (C > 1 && p.norm_w && threadIdx.x < C) arrive_remote(map_rank(misc(BAR_NORM_READ), threadIdx.x));
    } else if constexpr (!MOE) {
        if (!mbar_wait_bounded(misc(BAR_ACT), 0)) ok = false;
    }

    int slot = 0;                                       // of this warp's ring, and its barriers' phase
    uint32_t phase = 0;
    const uint32_t ring = ring_of(warp), full0 = bar_full(warp, 0), empty0 = bar_empty(warp, 0);
    // Up to 8 rows: every super-block is summed on its own, even and odd block pairs apart, and then added, so that no chain of
    // roundings is longer than a few dozen terms: error against 64 bits at 8 rows, one running sum / this / the dp4a kernel, Q6_K 4096 x
    // 1024 15.2 / 8.7 / 9.0e-8, 28672 x 1024 27.2 / 10.9 / 14.9e-8, Q8_0 4096 x 14336 11.6 / 8.1 / 8.0e-8. It costs 0.5 % (Q4_K 1.2 %).
    // More rows are below what the tcgen05 kernels show (4e-7) without it.
    constexpr int SETS = QUANT ? 2 : 0;
    // one row group: units of super-blocks [s0, s1); `act` = shared address of the activations of super-block s0
    auto run_group = [&](auto nt_tag, int s0, int s1, uint32_t act, uint32_t act_stride, auto& acc) {
        constexpr int NTC = decltype(nt_tag)::value;
        for (int sb = s0; sb < s1; sb += G::UNIT_SB) {
            if (!mbar_wait_bounded(full0 + 8 * slot, phase)) { ok = false; return; }
            const uint32_t row = ring + slot * G::UNIT_BYTES + gq * G::PITCH;
#pragma unroll
            for (int k = 0; k < G::UNIT_SB; ++k) {
                if (G::UNIT_SB > 1 && sb + k >= s1) break;
                const uint32_t r = row + G::offset_in_unit(sb, k), a = act + static_cast<uint32_t>(sb - s0 + k) * G::ACT_BYTES;
                if constexpr (SETS) {
                    float2 own[SETS][1][NTC][2];
#pragma unroll
                    for (int q = 0; q < SETS; ++q)
#pragma unroll
                        for (int t = 0; t < NTC; ++t) own[q][0][t][0] = own[q][0][t][1] = make_float2(0.f, 0.f);
                    super_block<TYPE, G::PITCH, 1, NTC>(r, a, act_stride, lane, NTC, own);
#pragma unroll
                    for (int t = 0; t < NTC; ++t)
#pragma unroll
                        for (int h = 0; h < 2; ++h) acc[0][0][t][h] = __fadd2_rn(acc[0][0][t][h], own[0][0][t][h]);
                } else {
                    super_block<TYPE, G::PITCH, 1, NTC>(r, a, act_stride, lane, NTC, acc);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * slot);                   // the slot may be refilled
            if (++slot == p.n_slots) { slot = 0; phase ^= 1; }
        }
    };

    if constexpr (MOE) {
        const int n_tiles = *reinterpret_cast<const volatile int*>(p.n_tiles_dev);
        int jb = 0;
        for (int j = blockIdx.x; j < n_tiles && ok; j += gridDim.x, ++jb) {
            const int4 t = __ldg(p.tile_tab + j);
            const int buf = jb % p.act_bufs;
            if (!mbar_wait_bounded(misc(BAR_ACT + 8 * buf), (jb / p.act_bufs) & 1)) { ok = false; break; }
            const int row0 = t.y + 16 * warp, nt = (t.w + 7) >> 3;
            const uint32_t act = sbase + OFF_ACT + buf * p.act_buf_bytes, act_stride = static_cast<uint32_t>(p.nsb) * G::ACT_BYTES;
            auto tile = [&](auto nt_tag) {
                constexpr int NTC = decltype(nt_tag)::value;
                float2 acc[1][1][NTC][2];
#pragma unroll
                for (int i = 0; i < NTC; ++i) acc[0][0][i][0] = acc[0][0][i][1] = make_float2(0.f, 0.f);
                run_group(nt_tag, 0, p.nsb, act, act_stride, acc);
#pragma unroll
                for (int i = 0; i < NTC; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int tok = 8 * i + 2 * tq + e;
                        if (tok >= t.w) continue;
                        int orow = __ldg(p.out_row + t.x + tok);
                        if (orow < 0) continue;
                        if (p.out_identity) orow = t.x + tok;
                        float* y = p.mat_y[0] + static_cast<size_t>(orow) * p.N + row0 + gq;
                        if (row0 + gq < p.N) y[0] = e ? acc[0][0][i][0].y : acc[0][0][i][0].x;
                        if (row0 + gq + 8 < p.N) y[8] = e ? acc[0][0][i][1].y : acc[0][0][i][1].x;
                    }
            };
            if (row0 < p.N) {
                if (nt == 1) tile(Tag<1>{});
                else if (NT >= 2 && nt == 2) tile(Tag<NT >= 2 ? 2 : 1>{});
                else if (NT >= 3 && nt == 3) tile(Tag<NT >= 3 ? 3 : 1>{});
                else if (NT >= 4 && nt == 4) tile(Tag<NT >= 4 ? 4 : 1>{});
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(misc(BAR_ACT_EMPTY + 8 * buf));
        }
    } else {
        const int part = warp / lanes, gl = warp - part * lanes, len = sb1 - sb0;
        const int s0 = sb0 + len * part / p.kw, s1 = sb0 + len * (part + 1) / p.kw;
        const uint32_t act_stride = static_cast<uint32_t>(len) * G::ACT_BYTES;
        const uint32_t act = sbase + OFF_ACT + static_cast<uint32_t>(s0 - sb0) * G::ACT_BYTES;
        // Partial results go to the CTA of the cluster that adds them up, row group g to rank g mod C.
        const uint32_t src_at = static_cast<uint32_t>((rank * p.kw + part) * NT * PART_BYTES + lane * 16), group_bytes = static_cast<uint32_t>(C * p.kw * NT * PART_BYTES);
        const int ng = row_groups(p, r0, r1);
        for (int g = gl; g < ng && ok; g += lanes) {
            float2 acc[1][1][NT][2];
#pragma unroll
            for (int i = 0; i < NT; ++i) acc[0][0][i][0] = acc[0][0][i][1] = make_float2(0.f, 0.f);
            run_group(Tag<NT>{}, s0, s1, act, act_stride, acc);
            if constexpr (C == 1) {                          // whole K: straight to y
                const Group gr = row_group(p, r0, r1, g);
                float* y = p.mat_y[gr.mat] + gr.row + gq;
                const int n = p.mat_end[gr.mat] - (gr.mat ? p.mat_end[gr.mat - 1] : 0);
#pragma unroll
                for (int i = 0; i < NT; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int tok = 8 * i + 2 * tq + e;
                        if (tok >= p.M) continue;
                        if (gq < gr.rows) y[static_cast<size_t>(tok) * n] = e ? acc[0][0][i][0].y : acc[0][0][i][0].x;
                        if (gq + 8 < gr.rows) y[static_cast<size_t>(tok) * n + 8] = e ? acc[0][0][i][1].y : acc[0][0][i][1].x;
                    }
            } else {
                if (!ok) break;
                const int owner = g % C, gi = g / C, at = gi % p.n_parts;
                // the place is free once that CTA has taken the group n_parts before (it takes them in order)
                if (gi >= p.n_parts && !wait_taken(misc(TAKEN + 4 * (owner * RW + (p.n_parts == 1 ? 0 : at % RW))), gi - p.n_parts + 1)) { ok = false; break; }
                const uint32_t dst = map_rank(sbase + p.off_part + static_cast<uint32_t>(at) * group_bytes + src_at, owner);
                const uint32_t bar = map_rank(misc(BAR_PART + 8 * at), owner);
#pragma unroll
                for (int i = 0; i < NT; ++i)
                    st_remote_counted(dst + i * PART_BYTES, bar, acc[0][0][i][0].x, acc[0][0][i][0].y, acc[0][0][i][1].x, acc[0][0][i][1].y);
            }
        }
    }
    if (!ok && lane == 0) report_status(p.err, DEV_TIMEOUT_FULL);      // the copy warps drain the copies
}

__global__ void __launch_bounds__(256) quantize_i8_kernel(const float* __restrict__ x, const float* __restrict__ norm_w, float eps,
                                                          float* __restrict__ x_norm_out, int K, int lane8, uint32_t act_bytes, uint8_t* __restrict__ img) {
    __shared__ float red[8];
    asm volatile("griddepcontrol.wait;" ::: "memory");                    // x is there, and the call before has read the scratch
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");       // the matmul's copies of weights may start (all before this call is done)
    const int m = blockIdx.x;
    const float* xr = x + static_cast<size_t>(m) * K;
    uint8_t* tile = img + static_cast<size_t>(m >> 3) * (K / 256) * act_bytes;
    if (!norm_w) {
        quantize_row_i8([&](int b, int t8) { return __ldg(reinterpret_cast<const float4*>(xr + b * 32) + t8); }, K, lane8, act_bytes, tile, m & 7);
        return;
    }
    float ss = 0.f;
    for (int i = threadIdx.x; i < K / 4; i += blockDim.x) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(xr) + i);
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w];
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(t, static_cast<float>(K)), eps)));
    quantize_row_i8([&](int b, int t8) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(xr + b * 32) + t8), w = __ldg(reinterpret_cast<const float4*>(norm_w + b * 32) + t8);
        const float4 n = make_float4(__fmul_rn(__fmul_rn(v.x, inv), w.x), __fmul_rn(__fmul_rn(v.y, inv), w.y),
                                     __fmul_rn(__fmul_rn(v.z, inv), w.z), __fmul_rn(__fmul_rn(v.w, inv), w.w));
        if (x_norm_out) reinterpret_cast<float4*>(x_norm_out + static_cast<size_t>(m) * K + b * 32)[t8] = n;
        return n;
    }, K, lane8, act_bytes, tile, m & 7);
}

struct TypeGeo { int pitch, act_bytes; bool lane8; };
template <uint32_t TYPE> TypeGeo geo_of() { return {Geo<TYPE>::PITCH, Geo<TYPE>::ACT_BYTES, Geo<TYPE>::LANE8}; }
bool type_geo(uint32_t type, TypeGeo& g) {
    switch (type) {
        case LAPLACE_TYPE_Q4_K: g = geo_of<LAPLACE_TYPE_Q4_K>(); return true;
        case LAPLACE_TYPE_Q8_0: g = geo_of<LAPLACE_TYPE_Q8_0>(); return true;
        case LAPLACE_TYPE_Q4_0: g = geo_of<LAPLACE_TYPE_Q4_0>(); return true;
        case LAPLACE_TYPE_Q6_K: g = geo_of<LAPLACE_TYPE_Q6_K>(); return true;
        default: return false;
    }
}

constexpr int MAX_NT = 4;
struct DensePlan { int nt, c, kw, smax, n_slots; uint32_t act, part_budget; };

// How K is cut: by K, type and row count, except for Q4_K with 3 to 8 rows and few weight rows. A CTA of the cluster gets two super-blocks
// or more; eight CTAs where the activations of four would not leave room for two ring slots a warp. False: the plan does not fit,
// the call takes another kernel.
// Q4_K, K = 4096..8192, up to 2048 weight rows: eight CTAs, whose shorter prologue is worth more than their weight rows (8 rows: 4096 x 1024
// 6.6 -> 5.8 us, 6144 x 1024 8.4 -> 6.9, 8192 x 2048 9.2 -> 8.1; 6144 x 4096 9.7 -> 9.7, 4096 x 16384 13.9 -> 16.6).
bool plan_dense(uint32_t type, int M, int K, long long rows, DensePlan& d) {
    TypeGeo g;
    if (!type_geo(type, g) || M < 2 || M > 8 * MAX_NT || K <= 0 || K % 256) return false;
    const int nsb = K / 256;
    d.nt = (M + 7) / 8;
    const bool wide = type == LAPLACE_TYPE_Q4_K && M <= 8 && rows <= 2048 && nsb >= 16 && nsb <= 32;
    for (int c = wide ? 8 : nsb >= 8 ? 4 : nsb >= 4 ? 2 : 1; c <= 8; c = c < 4 ? 4 : 2 * c) {
        d.c = c;
        d.smax = (nsb + c - 1) / c;
        d.kw = d.smax >= 8 ? 2 : 1;
        d.act = (static_cast<uint32_t>(d.nt * d.smax * g.act_bytes) + 127u) & ~127u;
        // Two ring slots a warp; then partial results, a row group taking kw x 8 nt x 16 floats from every CTA of the cluster: room for
        // two rounds of row groups, at least for half a round and for two places in every CTA of four (with less room eight CTAs, whose
        // activations take half of it, have more places than four would); then more slots.
        const long long slot = static_cast<long long>(CW) * 16 * g.pitch, group = d.kw * 8 * d.nt * 16 * 4, round = CW / d.kw * group;
        long long rest = static_cast<long long>(ctx().smem_optin) - OFF_ACT - d.act - 128 - 2 * slot;
        const long long least = c == 1 ? 0 : (round / 2 > 9 * group ? round / 2 : 9 * group), most = c == 1 ? 0 : 2 * round > 32 * 1024 ? 2 * round : 32 * 1024;
        if (rest < least) continue;
        d.part_budget = static_cast<uint32_t>(rest < most ? rest : most) & ~127u;
        rest -= d.part_budget;
        d.n_slots = 2 + static_cast<int>(rest / slot);
        if (d.n_slots > MAX_SLOTS) d.n_slots = MAX_SLOTS;
        return true;
    }
    return false;
}

template <uint32_t TYPE, int NT, int C, bool QUANT, bool MOE>
int launch_as(const I8Maps& maps, I8Params& p, int work_items, size_t part_bytes, size_t smem, cudaStream_t st) {
    auto k = gemm_i8_kernel<TYPE, NT, C, QUANT, MOE>;
    static int max_clusters = 0;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = C; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = C > 1 ? 2 : 1;
    cfg.blockDim = dim3(THREADS + (C > 1 ? 32 * RW : 0));
    cfg.stream = st;
    if (!max_clusters) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ctx().smem_optin));
        if (e != cudaSuccess) return cuda_check(e, "cudaFuncSetAttribute gemm_i8");
        int n = ctx().sm_count / C;
        if (C > 1) {
            // how many clusters the chip's groups of SMs hold at once: more of them would run as a second wave
            cudaLaunchConfig_t q = cfg;
            cudaLaunchAttribute only = attr[1];
            q.attrs = &only; q.numAttrs = 1;
            q.gridDim = dim3(n * C);
            q.dynamicSmemBytes = ctx().smem_optin;
            int fit = 0;
            e = cudaOccupancyMaxActiveClusters(&fit, k, &q);
            if (e != cudaSuccess) return cuda_check(e, "cudaOccupancyMaxActiveClusters gemm_i8");
            if (fit < 1) return LAPLACE_UNSUPPORTED;
            if (fit < n) n = fit;
        }
        max_clusters = n;
    }
    const int clusters = work_items < max_clusters ? work_items : max_clusters;
    if constexpr (C > 1) {
        p.n_parts = static_cast<int>(part_bytes / (C * p.kw * NT * PART_BYTES));
        if (p.n_parts > MAX_PARTS) p.n_parts = MAX_PARTS;
        if (p.n_parts > 1) p.n_parts = p.n_parts / RW * RW;
        if (p.n_parts < 1) return fail(LAPLACE_ERR_STATE, "gemm_i8: internal planning error (no room for partial results)");
    }
    cfg.gridDim = dim3(clusters * C);
    cfg.dynamicSmemBytes = smem;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, maps, p);
    ctx().launches++;
    ctx().last_kernel = KERNEL_INT8;
    return cuda_check(e, "gemm_i8 launch");
}

template <uint32_t TYPE, int NT, bool QUANT>
int launch_c(int c, const I8Maps& maps, I8Params& p, int work_items, size_t part_bytes, size_t smem, cudaStream_t st) {
    switch (c) {
        case 1: return launch_as<TYPE, NT, 1, QUANT, false>(maps, p, work_items, part_bytes, smem, st);
        case 2: return launch_as<TYPE, NT, 2, QUANT, false>(maps, p, work_items, part_bytes, smem, st);
        case 4: return launch_as<TYPE, NT, 4, QUANT, false>(maps, p, work_items, part_bytes, smem, st);
        default: return launch_as<TYPE, NT, 8, QUANT, false>(maps, p, work_items, part_bytes, smem, st);
    }
}
template <uint32_t TYPE>
int launch_nt(int nt, bool quant, int c, const I8Maps& maps, I8Params& p, int work_items, size_t part_bytes, size_t smem, cudaStream_t st) {
    if (quant) return launch_c<TYPE, 1, true>(c, maps, p, work_items, part_bytes, smem, st);
    switch (nt) {
        case 2: return launch_c<TYPE, 2, false>(c, maps, p, work_items, part_bytes, smem, st);
        case 3: return launch_c<TYPE, 3, false>(c, maps, p, work_items, part_bytes, smem, st);
        default: return launch_c<TYPE, 4, false>(c, maps, p, work_items, part_bytes, smem, st);
    }
}

template <uint32_t TYPE>
int launch_jobs_nt(int nt, const I8Maps& maps, I8Params& p, int jobs_max, size_t smem, cudaStream_t st) {
    switch (nt) {
        case 1: return launch_as<TYPE, 1, 1, false, true>(maps, p, jobs_max, 0, smem, st);
        case 2: return launch_as<TYPE, 2, 1, false, true>(maps, p, jobs_max, 0, smem, st);
        default: return launch_as<TYPE, 4, 1, false, true>(maps, p, jobs_max, 0, smem, st);
    }
}

// Shared memory of a job call with activation tiles of 8 nt rows; false: it does not fit.
bool plan_jobs(const TypeGeo& g, int K, int nt, I8Params& p, size_t& smem) {
    const uint32_t buf = (static_cast<uint32_t>(nt * (K / 256) * g.act_bytes) + 127u) & ~127u;
    for (p.act_bufs = 2; p.act_bufs >= 1; --p.act_bufs) {
        p.act_buf_bytes = buf;
        p.off_part = p.off_ring = OFF_ACT + p.act_bufs * buf;
        const long long ring = static_cast<long long>(ctx().smem_optin) - p.off_ring - 16;
        p.n_slots = static_cast<int>(ring / (static_cast<long long>(CW) * 16 * g.pitch));
        if (p.n_slots > MAX_SLOTS) p.n_slots = MAX_SLOTS;
        smem = p.off_ring + static_cast<size_t>(CW) * p.n_slots * 16 * g.pitch + 16;
        if (ring > 0 && p.n_slots >= 2) return true;
    }
    return false;
}

bool map_weights(CUtensorMap* m, const uint8_t* w, uint32_t type, int K, uint64_t rows, const TypeGeo& g) {
    const uint64_t rb = row_bytes(type, K);
    return tc::make_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_UINT32, w, rb / 4, rows, rb, g.pitch / 4, 16, CU_TENSOR_MAP_SWIZZLE_NONE, "weights");
}

}  // namespace

// Up to 8 rows: where the dp4a kernel is the faster one. It starts sooner (no cluster, no exchange; with a norm in front the
// difference grows, since here the row sums cross the cluster) but its time grows with rows x values, so the line is one on their
// product and, because that growth is per activation value, one on M x super-blocks. `rows`: weight rows of the whole call. Measured,
// dp4a against this kernel (us):
//   two rows: 4096 x 4096 Q4_K 6.7 / 7.6, Q6_K 8.5 / 9.5; 14336 x 4096 21.3 / 14.7, 26.7 / 20.2;
//   Q8_0, three rows, K = 1024: 1024 rows 3.3 / 4.6, 4096 4.3 / 4.9, 8192 5.6 / 5.4; K = 2048: 1024 4.2 / 4.9, 4096 6.4 / 5.8;
//   K = 3072: 5.5 / 5.5; eight rows, K = 1024: 512 rows 4.7 / 4.0; with a norm, three rows, K = 2048: 3072 rows 8.5 / 9.4, 6144 11.3 / 10.9;
//   Q6_K, three rows, 4096 x 1024: 6.8 / 7.1, x 2048 8.4 / 7.5; four rows, 2048 x 1024: 5.2 / 5.7, x 4096 8.1 / 6.5;
//   Q4_K, three rows, K = 1024: 2048 rows 4.6 / 5.1, 4096 5.6 / 5.1; with a norm, 6144 rows 8.8 / 9.4, 16384 15.7 / 10.3.
// Rows of one to three super-blocks: Q4_K eight rows 768 x 16384 24.0 / 5.6; the other types have not been taken off the dp4a kernel.
bool dp4a_wins(uint32_t type, int M, int nsb, long long rows, bool norm) {
    if (M == 2) return nsb < 32;
    const long long work = rows * M * nsb * 256;
    if (type == LAPLACE_TYPE_Q4_K) {
        if (nsb < 4) return norm ? M <= 4 && rows * M <= 12000 : M * nsb <= 6 && work <= 1000000;
        return norm ? M <= 4 && M * nsb <= 30 && work <= 20000000 : M == 3 && nsb <= 8 && work <= 9000000;
    }
    if (nsb < 4) return true;
    if (type == LAPLACE_TYPE_Q6_K) return M <= 4 && M * nsb <= 48 && work <= 20000000;
    return M * nsb <= 32 && (norm ? M <= 4 && work <= 28000000 : M <= 6 && work <= 20000000);
}

// Matrices the kernel takes: 16-byte aligned rows (the copies are tensor-map tiles), a plan that fits, and not faster elsewhere.
// `rows`: of all matrices.
bool gemm_i8_supports(uint32_t type, int M, int K, const uint8_t* const* ws, int n_mats, long long rows, bool norm) {
    DensePlan d;
    if (n_mats < 1 || n_mats > MAX_MATS || !plan_dense(type, M, K, rows, d) || row_bytes(type, K) % 16) return false;
    if (M <= 8 && dp4a_wins(type, M, K / 256, rows, norm)) return false;
    for (int i = 0; i < n_mats; ++i)
        if (reinterpret_cast<uintptr_t>(ws[i]) & 15) return false;
    return true;
}

// Rows of x, optionally RMS-normalised, in the order lp_i8.cuh describes: tile of 8 rows, super-block.
int launch_quantize_i8(const float* x, const float* norm_w, float eps, float* x_norm_out, uint32_t type, int M, int K, uint8_t* img, cudaStream_t st) {
    TypeGeo g;
    if (!type_geo(type, g)) return LAPLACE_UNSUPPORTED;
    ctx().launches++;
    return launch_early(quantize_i8_kernel, dim3(M), 256, 0, st, x, norm_w, eps, x_norm_out, K, g.lane8 ? 1 : 0, static_cast<uint32_t>(g.act_bytes), img);
}

// `scratch`: where more than 8 rows are quantized to (gemm_i8_act_bytes for every 8 rows and 256 values, 16-byte aligned);
// nullptr: the library's own.
int launch_gemm_i8(const float* x, const float* norm_w, float eps, float* x_norm_out, const uint8_t* const* ws, float* const* ys,
                   const int* ns, int n_mats, uint32_t type, int M, int K, cudaStream_t st, uint8_t* scratch) {
    Context& c = ctx();
    DensePlan d;
    TypeGeo g;
    long long total = 0;
    for (int i = 0; i < n_mats; ++i) total += ns[i];
    if (total >= (1LL << 30)) return fail(LAPLACE_ERR_LIMIT, "gemm: more than 2^30 weight rows");
    if (!plan_dense(type, M, K, total, d) || !type_geo(type, g)) return LAPLACE_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(x) & 15) return fail(LAPLACE_ERR_ARG, "gemm: x not 16-byte aligned");
    if (norm_w && ((reinterpret_cast<uintptr_t>(norm_w) & 15) || (x_norm_out && (reinterpret_cast<uintptr_t>(x_norm_out) & 15))))
        return fail(LAPLACE_ERR_ARG, "gemm_multi: the norm weights (and the optional output) must be 16-byte aligned");
    I8Maps maps;
    I8Params p{};
    for (int i = 0, end = 0; i < n_mats; ++i) {
        if (!map_weights(&maps.w[i], ws[i], type, K, static_cast<uint64_t>(ns[i]), g)) return LAPLACE_ERR_CUDA;
        end += ns[i];
        p.mat_y[i] = ys[i];
        p.mat_end[i] = end;
    }
    for (int i = n_mats; i < MAX_MATS; ++i) maps.w[i] = maps.w[0];
    p.x = x; p.norm_w = norm_w; p.norm_eps = eps; p.x_norm_out = x_norm_out; p.err = c.d_err;
    p.M = M; p.K = K; p.nsb = K / 256; p.n_mats = n_mats; p.total_rows = static_cast<int>(total); p.kw = d.kw;
    p.off_part = OFF_ACT + d.act;
    p.off_ring = (p.off_part + d.part_budget + 127u) & ~127u;
    p.n_slots = d.n_slots;
    const size_t smem = p.off_ring + static_cast<size_t>(CW) * d.n_slots * 16 * g.pitch + 16;      // + read-ahead of the unaligned loads
    const bool quant = M <= 8;
    int rc;
    if (!quant) {
        const size_t bytes = static_cast<size_t>(d.nt) * p.nsb * g.act_bytes;
        if (!scratch && (rc = gemm_scratch().ensure(bytes, st))) return rc;
        uint8_t* img = scratch ? scratch : static_cast<uint8_t*>(gemm_scratch().p);
        if ((rc = launch_quantize_i8(x, norm_w, eps, x_norm_out, type, M, K, img, st))) return rc;
        p.img = img;
    }
    const int items = static_cast<int>((total + 15) / 16);
    switch (type) {
        case LAPLACE_TYPE_Q4_K: rc = launch_nt<LAPLACE_TYPE_Q4_K>(d.nt, quant, d.c, maps, p, items, d.part_budget, smem, st); break;
        case LAPLACE_TYPE_Q8_0: rc = launch_nt<LAPLACE_TYPE_Q8_0>(d.nt, quant, d.c, maps, p, items, d.part_budget, smem, st); break;
        case LAPLACE_TYPE_Q4_0: rc = launch_nt<LAPLACE_TYPE_Q4_0>(d.nt, quant, d.c, maps, p, items, d.part_budget, smem, st); break;
        default: rc = launch_nt<LAPLACE_TYPE_Q6_K>(d.nt, quant, d.c, maps, p, items, d.part_budget, smem, st); break;
    }
    c.last_path = M <= 8 ? 1 : 2;
    return rc;
}

// The largest activation tile (in rows, at most 32) that expert jobs over this matrix take; 0: none.
int gemm_i8_job_tokens(uint32_t type, int K, const uint8_t* w) {
    TypeGeo g;
    I8Params p{};
    size_t smem;
    if (!type_geo(type, g) || K <= 0 || K % 256 || row_bytes(type, K) % 16 || (reinterpret_cast<uintptr_t>(w) & 15)) return 0;
    for (int nt : {4, 2, 1})
        if (plan_jobs(g, K, nt, p, smem)) return 8 * nt;
    return 0;
}
uint32_t gemm_i8_act_bytes(uint32_t type) { TypeGeo g; return type_geo(type, g) ? g.act_bytes : 0; }
bool     gemm_i8_lane8(uint32_t type) { TypeGeo g; return type_geo(type, g) && g.lane8; }

// One launch over the jobs of a device-built table (see I8Params): JOB_ROWS weight rows x up to `tokens` activation rows each.
int launch_gemm_i8_jobs(const uint8_t* w, uint32_t type, long long w_rows, const uint8_t* img, float* y, int K, int N, int tokens, int jobs_max,
                        const int4* tab, const int* n_jobs, const int* out_row, int out_identity, cudaStream_t st) {
    TypeGeo g;
    I8Params p{};
    size_t smem;
    if (!type_geo(type, g) || !plan_jobs(g, K, tokens / 8, p, smem)) return LAPLACE_UNSUPPORTED;
    I8Maps maps;
    if (!map_weights(&maps.w[0], w, type, K, static_cast<uint64_t>(w_rows), g)) return LAPLACE_ERR_CUDA;
    for (int i = 1; i < MAX_MATS; ++i) maps.w[i] = maps.w[0];
    p.img = img; p.err = ctx().d_err; p.K = K; p.nsb = K / 256; p.n_mats = 1; p.mat_y[0] = y; p.kw = 1; p.N = N;
    p.tile_tab = tab; p.n_tiles_dev = n_jobs; p.out_row = out_row; p.out_identity = out_identity;
    switch (type) {
        case LAPLACE_TYPE_Q4_K: return launch_jobs_nt<LAPLACE_TYPE_Q4_K>(tokens / 8, maps, p, jobs_max, smem, st);
        case LAPLACE_TYPE_Q8_0: return launch_jobs_nt<LAPLACE_TYPE_Q8_0>(tokens / 8, maps, p, jobs_max, smem, st);
        case LAPLACE_TYPE_Q4_0: return launch_jobs_nt<LAPLACE_TYPE_Q4_0>(tokens / 8, maps, p, jobs_max, smem, st);
        default: return launch_jobs_nt<LAPLACE_TYPE_Q6_K>(tokens / 8, maps, p, jobs_max, smem, st);
    }
}

}  // namespace lp
