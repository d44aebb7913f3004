"""The paired quantised GEMM (csrc/gemm_pair.cu) against fp32 products of the same dequantised weights: token counts around
the edges of its tiles, odd numbers of weight tiles, K ranges shorter than its rings, INT4 and INT8, all epilogues."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from zse_b200.ops import native
from zse_b200.ops import reference as ref


@pytest.fixture(scope="module")
def ops():
    from zse_b200.ops.backend import CudaOps
    o = CudaOps("cuda")
    yield o
    o.check()


def _part(kind, N, K, seed):
    """(part as files hold it, the fp16 weights the kernels multiply with)."""
    rng = np.random.default_rng(seed)
    s = (0.002 + 0.004 * rng.random((N, K // 128))).astype(np.float16)
    if kind == "int8":
        q = rng.integers(-127, 128, (N, K), dtype=np.int8)
        w = (q.reshape(N, -1, 128).astype(np.float32) * s[..., None]).astype(np.float16)
        return {"dtype": "int8", "data": q, "scales": s, "shape": (N, K)}, torch.from_numpy(w.reshape(N, K)).cuda()
    z = (-8 * s).astype(np.float16)
    q = rng.integers(0, 16, (N, K), dtype=np.uint8)
    w = (q.reshape(N, -1, 128).astype(np.float32) * s[..., None] + z[..., None]).astype(np.float16)
    return ({"dtype": "int4", "data": q[:, 0::2] | (q[:, 1::2] << 4), "scales": s, "zeros": z, "shape": (N, K)},
            torch.from_numpy(w.reshape(N, K)).cuda())


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


# one unit; several units per pair (more than 74); odd tile counts; columns that end inside a tile; 1 to 44 K stages
@pytest.mark.parametrize("kind", ["int4", "int8"])
@pytest.mark.parametrize("M,N,K", [(65, 256, 128), (77, 384, 640), (96, 4608, 512), (160, 1000, 1152), (255, 19200, 384),
                                   (257, 640, 5632), (300, 20480, 256), (1030, 3584, 1024)])
def test_pair_epilogues(ops, kind, M, N, K):
    p, wd = _part(kind, N, K, N + K)
    bias = (torch.randn(N, device="cuda") * 0.1).half()
    w = ops.make_linear([p], K, 128, bias)
    x = (torch.randn(M + 5, K, device="cuda") * 0.5).half()
    out = torch.full((M + 2, N), 7.0, dtype=torch.float16, device="cuda")
    ops.linear(w, x, M, out)
    planes = torch.full((8, M, N), 7.0, dtype=torch.float32, device="cuda")
    n = ops.linear_partial(ops.make_linear([p], K, 128), x, M, planes)
    torch.cuda.synchronize()
    ops.check()
    want = x[:M].float() @ wd.float().T
    # fp32 sums in another order: 1e-5; stored in fp16: half a unit, 2^-11
    assert _rel(planes[:n].double().sum(0), want) < 1e-5
    assert _rel(out[:M], want + bias.float()) < 5e-4
    assert (out[M:] == 7).all() and (planes[n:] == 7).all()


@pytest.mark.parametrize("kind", ["int4", "int8"])
@pytest.mark.parametrize("M,I,K", [(66, 64, 256), (130, 200, 640), (512, 9728, 384)])
def test_pair_swiglu(ops, kind, M, I, K):
    (g, gd), (u, ud) = _part(kind, I, K, 1), _part(kind, I, K, 2)
    w = ops.make_linear([g, u], K, 128, swiglu=True)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    out = torch.full((M + 1, I), 7.0, dtype=torch.float16, device="cuda")
    ops.linear_swiglu(w, x, M, out)
    torch.cuda.synchronize()
    ops.check()
    want = ref.swiglu(x.float() @ gd.float().T, x.float() @ ud.float().T)
    assert _rel(out[:M], want) < 5e-4 and (out[M:] == 7).all()


@pytest.mark.parametrize("ks", [1, 2, 3, 5, 8])
def test_pair_planes_on_request(ops, ks):
    M, N, K = 97, 512, 1408
    p, wd = _part("int4", N, K, 3)
    w = ops.make_linear([p], K, 128)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    planes = torch.zeros(8, M, N, dtype=torch.float32, device="cuda")
    n = ops.linear_partial(w, x, M, planes, k_split=ks)
    torch.cuda.synchronize()
    ops.check()
    assert n == native.gemm_w4_splits(M, N, K, ks) and n <= ks
    assert _rel(planes[:n].double().sum(0), x.float() @ wd.float().T) < 1e-5


@pytest.mark.parametrize("ks", [2, 4])
@pytest.mark.parametrize("M,N,K,epilogue", [(200, 1024, 2048, 0), (300, 2048, 1152, 0), (513, 2048, 640, 1)])
def test_cluster_along_k_on_request(ops, ks, M, N, K, epilogue):
    """An explicit split of an epilogue that needs the whole sum: wide CTAs in a cluster along K (csrc/gemm_w4.cu)."""
    assert native.gemm_w4_plan(M, N, K, epilogue, ks)[2:] == (ks, 0)
    if epilogue == 1:
        (g, gd), (u, ud) = _part("int4", N // 2, K, 1), _part("int4", N // 2, K, 2)
        w, cols = ops.make_linear([g, u], K, 128, swiglu=True), N // 2
    else:
        p, wd = _part("int4", N, K, 3)
        w, cols = ops.make_linear([p], K, 128), N
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    out = torch.full((M + 1, cols), 7.0, dtype=torch.float16, device="cuda")
    native.gemm_w4(w.data, x, M, None, out, M, N, K, cols, epilogue, ks, ops.status.ptr)
    torch.cuda.synchronize()
    ops.check()
    want = ref.swiglu(x.float() @ gd.float().T, x.float() @ ud.float().T) if epilogue == 1 else x.float() @ wd.float().T
    assert _rel(out[:M], want) < 5e-4 and (out[M:] == 7).all()


# Narrow layers of up to 256 tokens run in the wide CTA of csrc/gemm_w4.cu; these send them to the paired kernel, where the edges
# of its tiles are.
@pytest.fixture
def pairs_only():
    native.gemm_w4_set_mode(8)
    yield
    native.gemm_w4_set_mode(0)


@pytest.mark.parametrize("M,N,K", [(65, 256, 128), (77, 384, 640), (160, 1000, 1152), (129, 100, 256), (256, 1920, 384)])
def test_pair_narrow_int4(ops, pairs_only, M, N, K):
    assert native.gemm_w4_plan(M, N, K, 0)[3] == native.gemm_w4_plan(M, N, K, 2)[3] == 2
    test_pair_epilogues(ops, "int4", M, N, K)


@pytest.mark.parametrize("M,I,K", [(66, 64, 256), (130, 200, 640), (255, 832, 128)])
def test_pair_narrow_swiglu_int4(ops, pairs_only, M, I, K):
    assert native.gemm_w4_plan(M, 2 * I, K, 1)[3] == 2
    test_pair_swiglu(ops, "int4", M, I, K)
