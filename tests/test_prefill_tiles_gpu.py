"""GPU parity of the prefill kernels with more than one tile: pairs of SMs (Q4_K and Q6_K above 128 activation rows) and the int8 tiles
(above 32 rows), at the edges of a tile of weight rows, of activation rows and of K, with rows that no tensor map can address, with
super-blocks and activation rows of zeros; of the pairs also their error against 64 bits, exact block sums, special values and extreme
blocks. Oracle and bar as in the other GPU tests."""
import os
import subprocess
import sys

import numpy as np
import pytest

from laplace_b200.ggml import GGMLType
from tests import synth
from tests.parity import SMALL_N_MASS_TOL, check_close
from tests.test_baseline_shapes_gpu import _expected_from_blocksums

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 1
Q4_K, Q6_K, Q8_0, Q4_0 = GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0


def _run(t, x, ws, M, K, Ns):
    import torch
    from laplace_b200 import device
    xd, wd = torch.from_numpy(x).cuda(), [device.upload_weights(w) for w in ws]
    ys = [device.gemm(xd, wd[0], t, M, K, Ns[0])] if len(ws) == 1 else device.gemm_multi(xd, wd, t, M, K, Ns)
    device.sync()
    return [y.cpu().numpy() for y in ys]


@pytest.mark.parametrize("t,M,K,N", [(Q4_K, 129, 256, 1), (Q4_K, 256, 1024, 127), (Q4_K, 257, 512, 255), (Q4_K, 300, 2304, 257), (Q4_K, 144, 4096, 6000), (Q4_K, 513, 16640, 130),
                                     (Q6_K, 129, 256, 129), (Q6_K, 256, 2048, 256), (Q6_K, 257, 768, 33), (Q6_K, 290, 4096, 4100), (Q6_K, 160, 14336, 300), (Q6_K, 270, 16896, 100),
                                     (Q4_K, 144, 2048, 300), (Q4_K, 150, 14336, 260), (Q6_K, 300, 2048, 600),
                                     (Q8_0, 33, 256, 1), (Q8_0, 130, 1792, 9600), (Q8_0, 96, 2816, 129), (Q8_0, 97, 2816, 4000), (Q4_0, 129, 768, 127), (Q4_0, 64, 14336, 640), (Q4_K, 80, 1024, 700), (Q6_K, 112, 2048, 128)])
def test_edges_of_tiles(oracle, t, M, K, N):
    w = synth.weights(t, K, N, seed=700 + M, how="random")
    x = synth.normal_f32(701 + K, (M, K))
    (y,) = _run(t, x, [w], M, K, [N])
    mass = oracle.gemm(x, w, t, M, K, N, mode=2, threads=THREADS)
    check_close(y, oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"{t.name} M={M} K={K} N={N}", mass)


@pytest.mark.parametrize("t,M,K,Ns", [(Q4_K, 200, 4096, (700, 1, 300)), (Q6_K, 130, 2048, (64, 1000)), (Q8_0, 77, 2816, (2816, 1024, 40)), (Q4_0, 140, 1024, (5, 600))])
def test_matrices_of_one_call_have_the_bits_of_single_calls(oracle, t, M, K, Ns):
    ws = [synth.weights(t, K, n, seed=710 + i, how="affine") for i, n in enumerate(Ns)]
    x = synth.normal_f32(711, (M, K))
    for y, w, n in zip(_run(t, x, ws, M, K, Ns), ws, Ns):
        check_close(y, oracle.gemm(x, w, t, M, K, n, mode=1, threads=THREADS), f"multi {t.name} M={M} K={K} N={n}", oracle.gemm(x, w, t, M, K, n, mode=2, threads=THREADS))
        (single,) = _run(t, x, [w], M, K, [n])
        assert np.array_equal(single, y)


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("pack", ["random", "affine", "ref"])
@pytest.mark.parametrize("rows", ["normal", "outliers", "positive"])
def test_pairs_are_no_further_from_64_bits_than_single_ctas(oracle, t, pack, rows):
    """256 rows in one call, on pairs of SMs, against two calls of 128 rows, which run on the one-CTA kernels: other sums of the same
    products, no larger error. 256 x 384 independent errors put 1 / sqrt(2 x 98304) = 0.23 % of spread on either norm; 2 % between the two
    is six times that of their quotient."""
    M, K, N = 256, 4096, 384
    w = synth.random_blocks(t, K, N, seed=740) if pack == "random" else synth.weights(t, K, N, seed=740, how=pack)
    x = synth.normal_f32(741, (M, K))
    if rows == "outliers":
        x[:, ::97] *= np.float32(50.0)
    elif rows == "positive":
        x = np.abs(x)
    ref = oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS).astype(np.float64)
    (y,) = _run(t, x, [w], M, K, [N])
    one = np.concatenate([_run(t, x[m:m + 128], [w], 128, K, [N])[0] for m in (0, 128)])
    err, err_one = (np.linalg.norm(v - ref) for v in (y, one))
    assert err <= 1.02 * err_one, f"{err / np.linalg.norm(ref):.3e} against {err_one / np.linalg.norm(ref):.3e}"


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("K", [7168, 8192, 18432])
def test_long_rows_on_pairs_are_no_further_from_64_bits(oracle, t, K):
    """The same with whole tiles for every pair, so that a tile's K is summed by one CTA, at one go (7168) or, Q6_K, with sums set aside
    once (8192) and twice (18432); 16 of the 130 rows, 16 x 18944 errors: 0.13 %."""
    M, N = 130, 18944
    w, x = synth.random_blocks(t, K, N, seed=750), synth.normal_f32(751, (M, K))
    ref = oracle.gemm(x[:16], w, t, 16, K, N, mode=1, threads=THREADS).astype(np.float64)
    (y,) = _run(t, x, [w], M, K, [N])
    (one,) = _run(t, x[:128], [w], 128, K, [N])
    err, err_one = (np.linalg.norm(v[:16] - ref) for v in (y, one))
    assert err <= 1.02 * err_one, f"{err / np.linalg.norm(ref):.3e} against {err_one / np.linalg.norm(ref):.3e}"


def _on_pairs(t, x, w, M, K, N):
    from laplace_b200 import device
    (y,) = _run(t, x, [w], M, K, [N])
    assert device.lib().laplace_cuda_last_cta_group() == 2
    return y


@pytest.mark.parametrize("t,M,K,off,ctas", [(Q4_K, 128, 512, 0, 1), (Q4_K, 129, 512, 0, 2), (Q6_K, 128, 2048, 0, 1), (Q6_K, 129, 2048, 0, 2), (Q6_K, 129, 512, 2, 2), (Q8_0, 129, 512, 0, 1),
                                            (Q8_0, 300, 512, 2, 1)])
def test_line_to_the_pairs(t, M, K, off, ctas):
    import torch
    from laplace_b200 import device
    w = np.ascontiguousarray(synth.weights(t, K, 40, seed=742, how="random")).reshape(-1)
    buf = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    buf[off:off + w.size].copy_(torch.from_numpy(w))
    device.gemm(torch.ones(M, K, device="cuda"), buf[off:], t, M, K, 40)
    device.sync()
    assert device.lib().laplace_cuda_last_cta_group() == ctas


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("M", [129, 300])
def test_block_sums_on_pairs_bit_exact(oracle, t, M):
    K, N = 2048, 136
    for live in list(range(8)) + [8 * 5 + 3, K // 32 - 1]:
        w, x1, sc = synth.single_live_block(t, K, N, 7500 + live, live)
        x = np.concatenate([x1 * np.float32(2.0 ** -(m % 5)) * (-1) ** m for m in range(M)])
        y = _on_pairs(t, x, w, M, K, N)
        want = _expected_from_blocksums(oracle, t, w, x, sc, K, N, live)
        assert np.array_equal(y, want), f"{t.name} M={M} live block {live}: {np.abs(y - want).max()}"


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("M", [140, 257])
def test_special_rows_on_pairs(oracle, t, M):
    """A row of zeros, a value that is not a number, an infinity, a single large value; the other rows do not notice."""
    K, N = 2048, 128
    w, x = synth.weights(t, K, N, seed=743, how="random"), synth.normal_f32(744, (M, K))
    x[3] = 0.0
    x[7, 33] = np.nan
    x[M - 1, 100] = np.inf
    x[11] = 0.0
    x[11, K - 1] = 1.0e6
    y = _on_pairs(t, x, w, M, K, N)
    ref = oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS)
    assert np.isnan(y[7]).all() and np.isnan(y[M - 1]).all() and not y[3].any()
    keep = [m for m in range(M) if m not in (7, M - 1)]
    check_close(y[keep], ref[keep], f"{t.name} special rows")
    # one live value: each output is one product (Q4_K: and one min term), held to the parity bar's share of its mass. Q4_K's nibbles go in
    # less 8, and 8 times the scale comes back with the min term: a row's rounding also scales with the mass of nibbles of 8
    mass = oracle.gemm(x[11:12], w, t, 1, K, N, mode=2)[0]
    if t == Q4_K:
        eights = w.reshape(N, K // 256, 144).copy()
        eights[:, :, 2:4], eights[:, :, 16:] = 0, 0x88
        mass = mass + oracle.gemm(x[11:12], eights.reshape(N, -1), t, 1, K, N, mode=2)[0]
    assert (np.abs(y[11] - ref[11]) <= SMALL_N_MASS_TOL * mass).all()


@pytest.mark.parametrize("ql,qh,sc", [(0x00, 0x00, -128), (0x00, 0x00, 127), (0xFF, 0xFF, -128), (0xFF, 0xFF, 127), (0x0F, 0xAA, -1)])
def test_q6k_extreme_blocks_on_pairs(oracle, ql, qh, sc):
    """Weights of the largest magnitude, 4096 and what lies just below, against full-scale activations."""
    M, K, N = 130, 2048, 16
    blk = np.zeros(210, dtype=np.uint8)
    blk[0:128], blk[128:192], blk[192:208] = ql, qh, np.uint8(sc & 0xFF)
    blk[208:210] = np.frombuffer(np.float16(2.0 ** -12).tobytes(), dtype=np.uint8)
    w = np.tile(blk, (N, K // 256))
    x = np.full((M, K), 1.27, dtype=np.float32)
    x[1::2] *= -1.0
    x[:, ::7] *= 0.5
    y = _on_pairs(Q6_K, x, w, M, K, N)
    assert np.allclose(y, oracle.gemm(x, w, Q6_K, M, K, N, mode=1, threads=THREADS), rtol=2e-5, atol=0.0)


@pytest.mark.parametrize("d,dmin", [(6.0e-8, 1.0), (-0.02, 0.05), (0.03, -0.7), (2.0e-7, 6.0e4), (0.0, 0.5), (65504.0, 6.0e-8)])
def test_q4k_scales_far_apart_on_pairs(oracle, d, dmin):
    """Scales of either sign, subnormal ones, and offsets many orders above or below the values: all super-blocks, and every other one."""
    M, K, N = 130, 1024, 72
    x = synth.normal_f32(745, (M, K))
    for step in (1, 2):
        w = synth.random_blocks(Q4_K, K, N, seed=746).reshape(N, K // 256, 144).copy()
        w[:, ::step, 0:4] = np.frombuffer(np.array([d, dmin], dtype=np.float16).tobytes(), dtype=np.uint8)
        w = w.reshape(N, -1)
        y = _on_pairs(Q4_K, x, w, M, K, N)
        ref, mass = (oracle.gemm(x, w, Q4_K, M, K, N, mode=mode, threads=THREADS) for mode in (1, 2))
        assert np.isfinite(y).all() and (np.abs(y - ref) <= SMALL_N_MASS_TOL * mass).all(), f"{d} {dmin}: {(np.abs(y - ref) / mass).max():.3e} of the mass"


@pytest.mark.parametrize("t,M,K,Ns", [(Q4_K, 130, 16640, (40, 9)), (Q6_K, 130, 16640, (24,)), (Q4_K, 131, 8448, (33,)), (Q4_K, 129, 4352, (20,)), (Q6_K, 150, 2816, (300, 130))])
def test_normalised_rows_on_pairs(oracle, t, M, K, Ns):
    """Every form of the quantizer (rows in registers up to 4096, 8192 and 16384 values, longer ones read again) with the norm in front
    and its result asked for; the last one's weight rows are copied one by one, past a tile's end in both matrices."""
    import torch
    from laplace_b200 import device
    ws = [synth.random_blocks(t, K, n, seed=747 + i) for i, n in enumerate(Ns)]
    x, nw = synth.normal_f32(748, (M, K)), (1.0 + 0.1 * synth.normal_f32(749, (K,))).astype(np.float32)
    ys, xn = device.gemm_multi(torch.from_numpy(x).cuda(), [device.upload_weights(w) for w in ws], t, M, K, list(Ns), norm_weight=torch.from_numpy(nw).cuda(), eps=1e-5,
                               want_x_norm=True)
    device.sync()
    assert device.lib().laplace_cuda_last_cta_group() == 2
    xn = xn.cpu().numpy()
    want = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(axis=1, keepdims=True) + 1e-5) * nw
    assert np.linalg.norm(xn - want) <= 1e-6 * np.linalg.norm(want)
    for y, w, n in zip(ys, ws, Ns):
        check_close(y.cpu().numpy(), oracle.gemm(xn, w, t, M, K, n, mode=1, threads=THREADS), f"norm {t.name} M={M} K={K} N={n}")


def test_few_super_blocks_gained_are_not_worth_a_cut():
    """Launches: quantizer and matmul, and one more where pieces are added up (see the plans)."""
    import torch
    from laplace_b200 import device
    L = device.lib()
    for t, M, K, N, launches in ((Q8_0, 200, 2816, 8448, 2), (Q8_0, 77, 2816, 1024, 3), (Q4_K, 256, 4096, 14336, 2), (Q4_K, 144, 2048, 2048, 3)):
        w = torch.zeros(synth.row_bytes(t, K) * N, dtype=torch.uint8, device="cuda")
        L.laplace_cuda_launch_count(1)
        device.gemm(torch.ones(M, K, device="cuda"), w, t, M, K, N)
        assert L.laplace_cuda_launch_count(0) == launches, (t.name, M, K, N)
    device.sync()


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
def test_zero_super_blocks_and_rows(oracle, t):
    """A super-block with d = 0 (Q4_K: dmin stays) and activation rows of zeros, beside ordinary ones."""
    M, K, N = 140, 1024, 200
    w = np.array(synth.weights(t, K, N, seed=720, how="random")).view(np.uint8).reshape(N, K // 256, -1).copy()
    at = 0 if t == Q4_K else 208
    w[::3, 1, at:at + 2] = 0
    x = synth.normal_f32(721, (M, K))
    x[5] = 0.0
    x[131, 256:512] = 0.0
    w = w.reshape(-1)
    (y,) = _run(t, x, [w], M, K, [N])
    check_close(y, oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"zero blocks {t.name}")
    assert not y[5].any()


def test_scratch_of_a_call_with_several_matrices():
    """q / k / v of 512 rows: the operand, and partial results of at most pairs + tiles - 1 pieces a matrix (and the eighth that scratch
    grows by beyond what is asked for). In a process of its own, whose scratch is empty; a first small call loads the kernels."""
    code = """
import torch
from laplace_b200 import device
from laplace_b200.ggml import GGMLType
K, Ns = 4096, [4096, 1024, 1024]
ws = [torch.zeros(n * K // 256 * 144, dtype=torch.uint8, device="cuda") for n in Ns]
x, ys = torch.ones(512, K, device="cuda"), None
device.gemm(x[:130, :2048].contiguous(), ws[2], GGMLType.Q4_K, 130, 2048, 256)
keep = [torch.empty(512, n, device="cuda") for n in Ns]
del keep
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
device.gemm_multi(x, ws, GGMLType.Q4_K, 512, K, Ns)
device.sync()
print(before - torch.cuda.mem_get_info()[0], torch.cuda.get_device_properties(0).multi_processor_count // 2)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr
    grown, pairs = map(int, r.stdout.split())
    operand = 512 * 4096 * 4.5 + 512 * 4
    tiles = [2 * 16, 2 * 4, 2 * 4]
    assert grown <= 9 / 8 * (operand + sum(pairs + t - 1 for t in tiles) * 256 * 256 * 4) + (4 << 20), f"{grown / 2 ** 20:.1f} MiB"


@pytest.mark.parametrize("t,off", [(Q6_K, 2), (Q6_K, 8)])
def test_rows_off_the_copy_boundary(oracle, t, off):
    """Weights that begin between 16-byte boundaries are fetched row by row."""
    import torch
    from laplace_b200 import device
    M, K, N = 150, 2048, 300
    w = np.array(synth.weights(t, K, N, seed=730, how="random")).view(np.uint8).reshape(-1)
    x = synth.normal_f32(731, (M, K))
    buf = torch.zeros(w.size + 64, dtype=torch.uint8, device="cuda")
    wd = buf[off:off + w.size]
    wd.copy_(torch.from_numpy(w))
    y = device.gemm(torch.from_numpy(x).cuda(), wd, t, M, K, N)
    device.sync()
    check_close(y.cpu().numpy(), oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"{t.name} off by {off}")
