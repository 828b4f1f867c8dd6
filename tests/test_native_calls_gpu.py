"""The native host side of the torch-tensor calls: the same results as the general path, which still takes (and refuses) everything else."""
import numpy as np
import pytest

from laplace_b200.ggml import GGMLType
from tests import synth

pytestmark = pytest.mark.gpu


def _both(device, call):
    fast = call()
    native, device._native = device._native, None
    try:
        return fast, call()
    finally:
        device._native = native


def test_native_and_general_paths_agree():
    import torch
    from laplace_b200 import device
    device.lib()
    assert device._native is not None
    t, M, K, N, E, I = GGMLType.Q4_K, 3, 512, 96, 4, 256
    x = torch.from_numpy(synth.normal_f32(700, (M, K))).cuda()
    w = device.upload_weights(synth.weights(t, K, N * E, seed=701, how="affine"))
    gu, dn = (device.upload_weights(synth.weights(t, k, n * E, seed=702, how="affine")) for k, n in ((K, 2 * I), (I, K)))
    idx = torch.tensor([2, 0], dtype=torch.int32, device="cuda")
    norm = torch.ones(K, device="cuda")
    top_idx, top_w = torch.tensor([[0, 1], [2, 3], [1, 3]], dtype=torch.int32, device="cuda"), torch.full((M, 2), 0.5, device="cuda")
    for call in (lambda: device.gemm(x, w, t, M, K, N), lambda: device.gemm_multi(x, [w, w], t, M, K, (N, 64), norm_weight=norm, eps=1e-5),
                 lambda: device.moe_gemv(x, w, t, idx, K, N, per_expert_x=True), lambda: device.lm_head(x, w, t, M, K, N, softcap=5.0),
                 lambda: device.moe_route(x[:, :8].contiguous(), 2), lambda: device.moe_ffn(x, gu, dn, t, t, top_idx, top_w, E, K, I)):
        a, b = _both(device, call)
        a, b = (a, b) if isinstance(a, (list, tuple)) else ([a], [b])
        assert len(a) == len(b) and all(u.shape == v.shape and torch.equal(u, v) for u, v in zip(a, b))
    y = torch.empty((M, N), device="cuda")
    assert device.gemm(x, w, t, M, K, N, y=y) is y
    # on the caller's stream
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        z = device.gemm(x, w, t, M, K, N)
    s.synchronize()
    assert torch.equal(y, z)
    device.sync()


def test_what_was_refused_is_refused():
    import torch
    from laplace_b200 import device
    from laplace_b200.matmul import LaplaceCudaError
    t, M, K, N = GGMLType.Q4_K, 2, 512, 64
    x = torch.zeros((M, K), device="cuda")
    w = device.upload_weights(np.zeros(N * K // 256 * 144, dtype=np.uint8))
    for bad in (x.t(), x.double(), x.cpu(), x[:1]):
        with pytest.raises(AssertionError):
            device.gemm(bad, w, t, M, K, N)
    with pytest.raises(AssertionError):
        device.gemm(x, w[:100], t, M, K, N)
    with pytest.raises(LaplaceCudaError):
        device.gemm(x, w, t, 0, K, N)
    with pytest.raises(LaplaceCudaError):
        device.gemm(torch.zeros(M * K + 1, device="cuda")[1:], w, t, M, K, N)          # x not 16-byte aligned
    device.sync()


@pytest.mark.parametrize("transform", ["vmap", "grad", "jvp"])
@pytest.mark.parametrize("native", [True, False])
def test_tensors_without_storage_are_refused(transform, native):
    """Inside a function transform tensors have no storage: every call raises, with the native host side as without it."""
    import torch
    from laplace_b200 import device
    device.lib()
    t, K, N, E = GGMLType.Q4_K, 256, 8, 2
    w = torch.zeros(E * 2 * K * 144 + 64, dtype=torch.uint8, device="cuda")
    idx = torch.zeros((1, 2), dtype=torch.int32, device="cuda")
    wts = torch.zeros((1, 2), device="cuda")
    calls = [lambda x: device.gemm(x, w, t, 1, K, N), lambda x: device.gemm_multi(x, [w], t, 1, K, [N]), lambda x: device.moe_gemv(x, w, t, idx[0], K, N, per_expert_x=False),
             lambda x: device.lm_head(x, w, t, 1, K, N), lambda x: device.moe_route(x.reshape(1, -1), 2), lambda x: device.moe_ffn(x.reshape(1, -1), w, w, t, t, idx, wts, E, K, K)]
    x = torch.zeros((3, K), device="cuda")
    kept = device._native
    try:
        if not native:
            device._native = None
        for call in calls:
            def f(v):
                with pytest.raises(RuntimeError, match="data pointer"):
                    call(v)
                return v.sum()
            if transform == "vmap":
                torch.vmap(f)(x)
            elif transform == "grad":
                torch.func.grad(f)(x[0])
            else:
                torch.func.jvp(f, (x[0],), (x[0],))
    finally:
        device._native = kept
    assert device.gemm(x, w, t, 3, K, N).shape == (3, N)
    device.sync()
