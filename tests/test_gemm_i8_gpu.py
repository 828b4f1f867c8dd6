"""GPU parity of the int8 tensor-core matmul for 2..32 activation rows (one or several matrices, RMSNorm in front) against the CPU
oracle, at the edges of its plan: one super-block of K, cuts of K over one to eight CTAs that do not come out even, a
group of 16 rows with one live row, every number of 8-row tiles, more rows than the partial results of a cluster have room for."""
import os

import numpy as np
import pytest

from laplace_b200.ggml import GGMLType
from tests import synth
from tests.parity import check_close

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 1
TYPES = [GGMLType.Q4_K, GGMLType.Q6_K, GGMLType.Q8_0, GGMLType.Q4_0]


def _run(t, x, ws, M, K, Ns, norm=None):
    import torch
    from laplace_b200 import device
    xd, wd = torch.from_numpy(x).cuda(), [device.upload_weights(w) for w in ws]
    if norm is None and len(ws) == 1:
        ys, xn = [device.gemm(xd, wd[0], t, M, K, Ns[0])], None
    else:
        ys, xn = device.gemm_multi(xd, wd, t, M, K, Ns, norm_weight=None if norm is None else torch.from_numpy(norm).cuda(), eps=1e-5, want_x_norm=True)
    device.sync()
    return [y.cpu().numpy() for y in ys], x if norm is None else xn.cpu().numpy()


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("M,K,N", [(2, 256, 1), (8, 512, 17), (9, 1024, 33), (3, 2048, 16), (16, 2816, 129), (17, 3840, 200), (24, 14336, 100), (32, 4096, 300), (25, 5888, 40)])
def test_small_batches(oracle, t, M, K, N):
    w = synth.weights(t, K, N, seed=600 + M, how="random")
    x = synth.normal_f32(601 + K, (M, K))
    (y,), _ = _run(t, x, [w], M, K, [N])
    mass = oracle.gemm(x, w, t, M, K, N, mode=2, threads=THREADS)
    check_close(y, oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"int8 {t.name} M={M} K={K} N={N}", mass)


@pytest.mark.parametrize("M", [8, 24])
def test_more_rows_than_one_panel(oracle, M):
    """Far more row groups than a CTA has places for partial results: some 130 of a cluster's share, 33 a CTA, for eight places (8 rows) or
    six (24 rows), the last group ragged."""
    t, K, N = GGMLType.Q4_K, 4096, 70001
    w = synth.weights(t, K, N, seed=610, how="affine")
    x = synth.normal_f32(611, (M, K))
    (y,), _ = _run(t, x, [w], M, K, [N])
    check_close(y, oracle.gemm(x, w, t, M, K, N, mode=1, threads=THREADS), f"panels M={M}")


@pytest.mark.parametrize("t,M,K,Ns", [(GGMLType.Q4_K, 8, 4096, (40, 1, 17)), (GGMLType.Q8_0, 12, 2816, (64, 33)), (GGMLType.Q6_K, 7, 14336, (5, 48)), (GGMLType.Q4_0, 31, 768, (24, 24, 9))])
def test_matrices_that_share_normalised_rows(oracle, t, M, K, Ns):
    ws = [synth.weights(t, K, n, seed=620 + i, how="affine") for i, n in enumerate(Ns)]
    x = synth.normal_f32(621, (M, K)) * np.float32(2.5)
    nw = (1.0 + 0.1 * synth.normal_f32(622, (K,))).astype(np.float32)
    ys, xn = _run(t, x, ws, M, K, Ns, nw)
    for y, w, n in zip(ys, ws, Ns):
        mass = oracle.gemm(xn, w, t, M, K, n, mode=2)
        check_close(y, oracle.gemm(xn, w, t, M, K, n, mode=1), f"int8 multi {t.name} M={M} K={K} N={n}", mass)
        (single,), _ = _run(t, np.ascontiguousarray(xn), [w], M, K, [n])
        assert np.array_equal(single, y)            # how K is cut does not depend on the rows of a call


@pytest.mark.parametrize("t,M,K", [(GGMLType.Q4_K, 16, 11008), (GGMLType.Q4_K, 24, 14336), (GGMLType.Q4_K, 8, 24832), (GGMLType.Q8_0, 24, 8192), (GGMLType.Q6_K, 32, 8192),
                                   (GGMLType.Q4_0, 32, 11520), (GGMLType.Q8_0, 24, 16384)])
def test_eight_matrices_where_partial_results_have_little_room(oracle, t, M, K):
    """Two places and one for partial results in every CTA of clusters of four and of eight (one: one of the two adding warps has nothing to
    do; with one warp a row group and with two), the groups cut at the ends of several matrices."""
    Ns = (1500, 1, 700, 16, 5, 1290, 64, 800)
    ws = [synth.random_blocks(t, K, n, seed=650 + i) for i, n in enumerate(Ns)]
    x = synth.normal_f32(651, (M, K))
    ys, _ = _run(t, x, ws, M, K, Ns)
    for y, w, n in zip(ys, ws, Ns):
        mass = oracle.gemm(x, w, t, M, K, n, mode=2, threads=THREADS)
        check_close(y, oracle.gemm(x, w, t, M, K, n, mode=1, threads=THREADS), f"eight matrices {t.name} M={M} K={K} N={n}", mass)
        (single,), _ = _run(t, x, [w], M, K, [n])
        assert np.array_equal(single, y)


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("K,N", [(4096, 2048), (14336, 1024)])
def test_no_further_from_64_bits_than_one_row_calls(oracle, t, K, N):
    """Eight rows in one call against eight calls of one row, which run on the dp4a kernel: other sums of the same products, no
    larger error. 8 x N independent errors put 1 / sqrt(16 N) = 0.8 % of spread on either norm; 8 % between the two is ten of it."""
    w, x = synth.weights(t, K, N, seed=660, how="affine"), synth.normal_f32(661, (8, K))
    ref = oracle.gemm(x, w, t, 8, K, N, mode=1, threads=THREADS)
    (y,), _ = _run(t, x, [w], 8, K, [N])
    one = np.concatenate([_run(t, x[m:m + 1], [w], 1, K, [N])[0][0] for m in range(8)])
    err, err_one = (np.linalg.norm(v.astype(np.float64) - ref) for v in (y, one))
    assert err <= 1.08 * err_one, f"{err / np.linalg.norm(ref):.3e} against {err_one / np.linalg.norm(ref):.3e}"


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("M", [5, 20])
def test_special_rows(oracle, t, M):
    """A row of zeros gives zeros, a value that is not a number takes its own row only, so does an infinity."""
    K, N = 1024, 48
    w = synth.weights(t, K, N, seed=630, how="random")
    x = synth.normal_f32(631, (M, K))
    x[0] = 0.0
    x[2, 40] = np.nan
    x[3, 100] = np.inf
    (y,), _ = _run(t, x, [w], M, K, [N])
    ref = oracle.gemm(x, w, t, M, K, N, mode=1)
    assert not y[0].any()
    assert np.isnan(y[2]).all() and np.isnan(y[3]).all()
    keep = [m for m in range(M) if m not in (2, 3)]
    check_close(y[keep], ref[keep], f"{t.name} special rows")


def test_unaligned_weights_take_the_streaming_kernel(oracle):
    """Rows that a tensor-map copy cannot address (a base that is not 16-byte aligned, rows of 11 Q6_K super-blocks) run as before."""
    import torch
    from laplace_b200 import device
    for t, K, off in ((GGMLType.Q8_0, 512, 2), (GGMLType.Q6_K, 2816, 0)):
        M, N = 4, 40
        w = synth.weights(t, K, N, seed=640, how="random")
        x = synth.normal_f32(641, (M, K))
        flat = w.reshape(-1)
        buf = torch.zeros(flat.size + 64 + off, dtype=torch.uint8, device="cuda")
        buf[off:off + flat.size].copy_(torch.from_numpy(flat))
        y = device.gemm(torch.from_numpy(x).cuda(), buf[off:], t, M, K, N)
        device.sync()
        check_close(y.cpu().numpy(), oracle.gemm(x, w, t, M, K, N, mode=1), f"unaligned {t.name}")
