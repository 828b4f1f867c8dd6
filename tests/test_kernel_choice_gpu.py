"""Which kernel a call runs on, at the lines between them, and parity of the tcgen05 kernels on calls that only they take: rows that a
tensor map cannot address, prompts above the int8 tiles' row counts, experts above the job kernel's pair counts; and of the
int8 job kernel with experts far above their average."""
import os

import numpy as np
import pytest

from laplace_b200.ggml import GGMLType
from laplace_b200.moe import seeded_routing
from tests import synth
from tests.parity import SMALL_N_MASS_TOL, check_close
from tests.test_baseline_shapes_gpu import _expected_from_blocksums
from tests.test_moe_ffn_gpu import _host_activation

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 1
DP4A, INT8, INT8_TILES, TCGEN05, TCGEN05_TWO_PIECE = 1, 2, 3, 4, 5
Q4_K, Q6_K, Q8_0, Q4_0 = GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0


def _upload(w, off=0):
    """Rows on the device, `off` bytes from a 16-byte boundary."""
    import torch
    flat = np.ascontiguousarray(w).reshape(-1)
    buf = torch.zeros(flat.size + 64 + off, dtype=torch.uint8, device="cuda")
    buf[off:off + flat.size].copy_(torch.from_numpy(flat))
    return buf[off:]


def _gemm(t, x, w, M, K, N, off=0):
    import torch
    from laplace_b200 import device
    y = device.gemm(torch.from_numpy(x).cuda(), _upload(w, off), t, M, K, N)
    device.sync()
    return y.cpu().numpy(), device.lib().laplace_cuda_last_kernel()


@pytest.mark.parametrize("t,M,K,off,kernel", [
    (Q4_K, 1, 4096, 0, DP4A), (Q4_K, 2, 7936, 0, DP4A), (Q4_K, 2, 8192, 0, INT8), (Q4_K, 3, 512, 0, DP4A), (Q4_K, 3, 768, 0, INT8), (Q4_K, 3, 2048, 0, DP4A), (Q4_K, 3, 2304, 0, INT8),
    (Q6_K, 3, 4096, 0, DP4A), (Q6_K, 4, 4096, 0, INT8), (Q8_0, 4, 2048, 0, DP4A), (Q8_0, 4, 2304, 0, INT8), (Q4_0, 7, 1024, 0, INT8), (Q8_0, 8, 768, 0, DP4A), (Q4_K, 9, 256, 0, INT8), (Q4_K, 32, 4096, 0, INT8), (Q4_K, 33, 4096, 0, INT8_TILES), (Q4_K, 80, 2048, 0, INT8_TILES), (Q4_K, 81, 2048, 0, TCGEN05),
    (Q6_K, 32, 2048, 0, INT8), (Q6_K, 112, 2048, 0, INT8_TILES), (Q6_K, 113, 2048, 0, TCGEN05_TWO_PIECE), (Q6_K, 24, 2816, 0, TCGEN05_TWO_PIECE),
    (Q8_0, 16, 512, 0, INT8), (Q8_0, 130, 512, 0, INT8_TILES), (Q8_0, 16, 512, 2, TCGEN05_TWO_PIECE), (Q4_0, 200, 768, 0, INT8_TILES), (Q4_0, 200, 768, 2, TCGEN05_TWO_PIECE),
    (Q8_0, 20, 544, 0, DP4A)])
def test_lines_between_the_kernels(t, M, K, off, kernel):
    w, x = synth.weights(t, K, 40, seed=860, how="random"), synth.normal_f32(861, (M, K))
    assert _gemm(t, x, w, M, K, 40, off)[1] == kernel


@pytest.mark.parametrize("t,M,K,N", [(Q8_0, 3, 1024, 6511), (Q4_K, 3, 1024, 2930), (Q6_K, 4, 2048, 2442), (Q4_K, 4, 256, 1000)])
def test_line_on_the_weight_rows(oracle, t, M, K, N):
    """The last row count of the dp4a kernel and the first of the int8 one, with room for neither's rounding in between."""
    w, x = synth.weights(t, K, N, seed=874, how="random"), synth.normal_f32(875, (M, K))
    ref = oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS)
    kernels = []
    for n in (N - N // 8, N):
        y, kernel = _gemm(t, x, w[:n], M, K, n)
        kernels.append(kernel)
        check_close(y, ref[:, :n], f"{t.name} {M} x {K} x {n}")
    assert kernels == [DP4A, INT8]


@pytest.mark.parametrize("t,M,K,Ns", [(Q4_K, 8, 4096, (1024, 1000, 24)), (Q4_K, 5, 6144, (17,)), (Q4_K, 3, 8192, (700, 1349)), (Q4_K, 8, 256, (40, 9)), (Q4_K, 6, 768, (1000, 33)),
                                      (Q4_K, 3, 512, (5000, 16))])
@pytest.mark.parametrize("norm", [False, True])
def test_q4k_plans_of_up_to_eight_rows(oracle, t, M, K, Ns, norm):
    """Clusters of eight up to 2048 weight rows and of four beyond, single CTAs for rows of one to three super-blocks."""
    import torch
    from laplace_b200 import device
    ws = [synth.random_blocks(t, K, n, seed=876 + i) for i, n in enumerate(Ns)]
    x = synth.normal_f32(877, (M, K))
    nw = torch.from_numpy((1.0 + 0.1 * synth.normal_f32(878, (K,))).astype(np.float32)).cuda() if norm else None
    ys, xn = device.gemm_multi(torch.from_numpy(x).cuda(), [_upload(w) for w in ws], t, M, K, list(Ns), norm_weight=nw, eps=1e-5, want_x_norm=True)
    device.sync()
    assert device.lib().laplace_cuda_last_kernel() == INT8
    x_in = xn.cpu().numpy() if norm else x
    for y, w, n in zip(ys, ws, Ns):
        mass = oracle.gemm(x_in, w, t, M, K, n, mode=2, threads=THREADS)
        check_close(y.cpu().numpy(), oracle.gemm(x_in, w, t, M, K, n, mode=1, threads=THREADS), f"Q4_K M={M} K={K} N={n}", mass)


@pytest.mark.parametrize("t,off", [(Q6_K, 2), (Q8_0, 2), (Q4_0, 2), (Q6_K, 0)])
@pytest.mark.parametrize("M,K,N", [(130, 768, 129), (9, 512, 40), (64, 2816, 200), (200, 1024, 136)])
def test_two_piece_kernels(oracle, t, off, M, K, N):
    w, x = synth.weights(t, K, N, seed=862, how="random"), synth.normal_f32(863 + M, (M, K))
    y, kernel = _gemm(t, x, w, M, K, N, off)
    assert kernel == TCGEN05_TWO_PIECE
    check_close(y, oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"two pieces {t.name} +{off} M={M} K={K} N={N}")


@pytest.mark.parametrize("t,off", [(Q4_K, 0), (Q6_K, 0), (Q8_0, 2), (Q4_0, 2)])
def test_block_sums_of_the_tcgen05_kernels_bit_exact(oracle, t, off):
    M, K, N = 128, 2048, 136
    for live in list(range(8)) + [8 * 5 + 3, K // 32 - 1]:
        w, x1, sc = synth.single_live_block(t, K, N, 3000 + live, live)
        x = np.concatenate([x1 * np.float32(2.0 ** -(m % 5)) * (-1) ** m for m in range(M)])
        y, kernel = _gemm(t, x, w, M, K, N, off)
        assert kernel == (TCGEN05 if t == Q4_K else TCGEN05_TWO_PIECE)
        want = _expected_from_blocksums(oracle, t, w, x, sc, K, N, live)
        assert np.array_equal(y, want), f"{t.name} live block {live}: {np.abs(y - want).max()}"


@pytest.mark.parametrize("ql,qh,sc", [(0x00, 0x00, -128), (0x00, 0x00, 127), (0xFF, 0xFF, -128), (0xFF, 0xFF, 127), (0x0F, 0xAA, -1)])
def test_q6k_extreme_blocks_on_tcgen05(oracle, ql, qh, sc):
    """Weights of the largest magnitude against full-scale activations: the sums stay exact (see test_q6k_prefill_extreme_blocks)."""
    M, K, N = 128, 2048, 16
    blk = np.zeros(210, dtype=np.uint8)
    blk[0:128], blk[128:192], blk[192:208] = ql, qh, np.uint8(sc & 0xFF)
    blk[208:210] = np.frombuffer(np.float16(2.0 ** -12).tobytes(), dtype=np.uint8)
    w = np.tile(blk, (N, K // 256))
    x = np.full((M, K), 1.27, dtype=np.float32)
    x[1::2] *= -1.0
    x[:, ::7] *= 0.5
    y, kernel = _gemm(Q6_K, x, w, M, K, N)
    assert kernel == TCGEN05_TWO_PIECE
    assert np.allclose(y, oracle.gemm(x, w, Q6_K, M, K, N, mode=1, threads=THREADS), rtol=2e-5, atol=0.0)


@pytest.mark.parametrize("t,K,off", [(Q4_K, 512, 0), (Q6_K, 2048, 0), (Q8_0, 512, 2), (Q4_0, 512, 2)])
def test_special_rows_on_tcgen05(oracle, t, K, off):
    """A row of zeros, a value that is not a number, a single large value; the other rows do not notice."""
    M, N = 128, 128
    w, x = synth.weights(t, K, N, seed=864, how="random"), synth.normal_f32(865, (M, K))
    x[3] = 0.0
    x[7, 33] = np.nan
    x[11] = 0.0
    x[11, K - 1] = 1.0e6
    y, kernel = _gemm(t, x, w, M, K, N, off)
    assert kernel in (TCGEN05, TCGEN05_TWO_PIECE)
    ref = oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS)
    assert np.isnan(y[7]).all() and not y[3].any()
    keep = [m for m in range(M) if m != 7]
    check_close(y[keep], ref[keep], f"{t.name} special rows")
    # one live value: each output is one product. Q4_0's (q - 8) can be zero, where the oracle is left with the rounding of its fp32
    # offset sum: held to the parity bar's share of the mass
    mass = oracle.gemm(x[11:12], w, t, 1, K, N, mode=2)[0]
    assert (np.abs(y[11] - ref[11]) <= np.where(t == Q4_0, SMALL_N_MASS_TOL * mass, 2e-6 * np.abs(ref[11]))).all()


def _grouped(t, x, w, pair_expert, E, K, N):
    import torch
    from laplace_b200 import device
    y = device.moe_grouped(torch.from_numpy(x).cuda(), device.upload_weights(w), t, torch.from_numpy(pair_expert).cuda(), None, E, K, N)
    device.sync()
    assert device.lib().laplace_cuda_last_path() == 3
    return y.cpu().numpy(), device.lib().laplace_cuda_last_kernel()


@pytest.mark.parametrize("t", [Q4_K, Q6_K, Q8_0, Q4_0])
@pytest.mark.parametrize("counts,int8", [((40, 60, 0, 33), False), ((150, 0, 31, 1, 9, 32, 33, 0), True)])
def test_experts_on_either_side_of_the_line(oracle, t, counts, int8):
    """More pairs than the int8 jobs are for on average: tcgen05 tiles. Fewer on average, but single experts with far more than
    one job holds: several jobs of such an expert."""
    K, N, E = 2048, 136, len(counts)
    pair_expert = np.repeat(np.arange(E, dtype=np.int32), counts)
    np.random.default_rng(866).shuffle(pair_expert)
    w, x = synth.weights(t, K, N * E, seed=867, how="random"), synth.normal_f32(868, (pair_expert.size, K))
    y, kernel = _grouped(t, x, w, pair_expert, E, K, N)
    assert kernel == (INT8 if int8 else TCGEN05 if t == Q4_K else TCGEN05_TWO_PIECE)
    check_close(y, oracle.moe_gemv(x, w, t, pair_expert, K, N, multi=True, mode=1, threads=THREADS), f"experts {t.name} {counts}")


@pytest.mark.parametrize("t_gu,t_dn,H,I", [(Q4_K, Q6_K, 512, 256), (Q8_0, Q4_0, 512, 256), (Q6_K, Q8_0, 2048, 512)])
def test_fused_ffn_on_tcgen05(oracle, t_gu, t_dn, H, I):
    """More pairs per expert than the int8 jobs are for; stage by stage as in test_moe_ffn_gpu."""
    import torch
    from laplace_b200 import device
    E, k, T = 3, 2, 80
    w_gu, w_dn = synth.weights(t_gu, H, E * 2 * I, seed=870, how="random"), synth.weights(t_dn, I, E * H, seed=871, how="random")
    x = synth.normal_f32(872, (T, H))
    idx, wts = seeded_routing(873, T, E, k)
    h_dev = torch.zeros((T * k, I), dtype=torch.float32, device="cuda")
    out = device.moe_ffn(torch.from_numpy(x).cuda(), device.upload_weights(w_gu), device.upload_weights(w_dn), t_gu, t_dn, torch.from_numpy(idx).cuda(),
                         torch.from_numpy(wts).cuda(), E, H, I, h_out=h_dev)
    device.sync()
    assert device.lib().laplace_cuda_last_kernel() == TCGEN05_TWO_PIECE
    h_dev = h_dev.cpu().numpy()
    gu = np.concatenate([oracle.moe_gemv(x[tok], w_gu, t_gu, idx[tok], H, 2 * I, multi=False, mode=1) for tok in range(T)])
    check_close(h_dev, _host_activation(gu, I, 0), "activation(gate/up)")
    want = np.zeros((T, H), dtype=np.float64)
    for tok in range(T):
        dn = oracle.moe_gemv(h_dev[tok * k:(tok + 1) * k], w_dn, t_dn, idx[tok], I, H, multi=True, mode=1)
        want[tok] = (dn.astype(np.float64) * wts[tok][:, None]).sum(axis=0)
    check_close(out.cpu().numpy(), want.astype(np.float32), f"fused FFN {t_gu.name} {t_dn.name}")
