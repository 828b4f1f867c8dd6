"""GPU parity of the prefill kernels with more than one tile: pairs of SMs (Q4_K and Q6_K above 128 activation rows) and the int8 tiles
(above 32 rows), at the edges of a tile of weight rows, of activation rows and of K, with rows that no tensor map can address, with
super-blocks and activation rows of zeros, and where partial results have no room. Oracle and bar as in the other GPU tests."""
import os
import subprocess
import sys

import numpy as np
import pytest

from laplace_b200.ggml import GGMLType
from tests import synth
from tests.parity import check_close

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
                                     (Q6_K, 129, 256, 129), (Q6_K, 256, 2048, 256), (Q6_K, 257, 768, 33), (Q6_K, 290, 4096, 4100), (Q6_K, 160, 14336, 300),
                                     (Q8_0, 33, 256, 1), (Q8_0, 96, 2816, 129), (Q8_0, 97, 2816, 4000), (Q4_0, 129, 768, 127), (Q4_0, 64, 14336, 640), (Q4_K, 80, 1024, 700), (Q6_K, 112, 2048, 128)])
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
