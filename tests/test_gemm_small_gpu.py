"""The register-streamed INT4 GEMM for up to 8 tokens (csrc/gemm_w4_small.cu) against float64 products of the stored weights: token
counts, half tiles, K ranges with fewer groups than warps, all epilogues."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from zse_b200.ops import native


@pytest.fixture(scope="module")
def ops():
    from zse_b200.ops.backend import CudaOps
    o = CudaOps("cuda")
    yield o
    o.check()


def _part(N, K, seed):
    """(part as files hold it, its weights q * s + z in float64)."""
    rng = np.random.default_rng(seed)
    s = (0.002 + 0.004 * rng.random((N, K // 128))).astype(np.float16)
    z = (-8 * s * (0.8 + 0.4 * rng.random(s.shape))).astype(np.float16)
    q = rng.integers(0, 16, (N, K), dtype=np.uint8)
    w = q.reshape(N, -1, 128).astype(np.float64) * s[..., None].astype(np.float64) + z[..., None].astype(np.float64)
    return ({"dtype": "int4", "data": q[:, 0::2] | (q[:, 1::2] << 4), "scales": s, "zeros": z, "shape": (N, K)},
            torch.from_numpy(w.reshape(N, K)).cuda())


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


# fewer and more items than SMs, more than two an SM; rows that end inside a half tile; one K group, fewer groups than warps
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (1, 3584, 3584), (2, 200, 640), (7, 4608, 3584), (8, 19456, 256), (5, 384, 2048),
                                   (6, 20480, 384), (8, 5120, 13824), (3, 1000, 1152)])
def test_small_epilogues(ops, M, N, K):
    p, wd = _part(N, K, N + K)
    bias = (torch.randn(N, device="cuda") * 0.1).half()
    x = (torch.randn(M + 3, K, device="cuda") * 0.5).half()
    x[:, 5] = 3e-5                                            # fp16 subnormals among the activations
    out = torch.full((M + 2, N), 7.0, dtype=torch.float16, device="cuda")
    ops.linear(ops.make_linear([p], K, 128, bias), x, M, out)
    planes = torch.full((8, M, N), 7.0, dtype=torch.float32, device="cuda")
    n = ops.linear_partial(ops.make_linear([p], K, 128), x, M, planes)
    torch.cuda.synchronize()
    ops.check()
    want = x[:M].double() @ wd.T
    # exact products, fp32 sums: 1e-5; stored in fp16: half a unit, 2^-11
    assert _rel(planes[:n].double().sum(0), want) < 1e-5
    assert _rel(out[:M], want + bias.double()) < 5e-4
    assert (out[M:] == 7).all() and (planes[n:] == 7).all()


@pytest.mark.parametrize("M,I,K", [(1, 64, 128), (3, 200, 640), (8, 18944, 512), (5, 9728, 384)])
def test_small_swiglu(ops, M, I, K):
    (g, gd), (u, ud) = _part(I, K, 1), _part(I, K, 2)
    w = ops.make_linear([g, u], K, 128, swiglu=True)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    out = torch.full((M + 1, I), 7.0, dtype=torch.float16, device="cuda")
    ops.linear_swiglu(w, x, M, out)
    torch.cuda.synchronize()
    ops.check()
    want = torch.nn.functional.silu(x.double() @ gd.T) * (x.double() @ ud.T)
    assert _rel(out[:M], want) < 5e-4 and (out[M:] == 7).all()


@pytest.mark.parametrize("ks", [1, 2, 3, 8])
def test_small_planes_on_request(ops, ks):
    M, N, K = 5, 512, 1408
    p, wd = _part(N, K, 3)
    w = ops.make_linear([p], K, 128)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    planes = torch.zeros(8, M, N, dtype=torch.float32, device="cuda")
    n = ops.linear_partial(w, x, M, planes, k_split=ks)
    torch.cuda.synchronize()
    ops.check()
    assert n == native.gemm_w4_splits(M, N, K, ks) and n <= ks
    assert _rel(planes[:n].double().sum(0), x.double() @ wd.T) < 1e-5


@pytest.mark.parametrize("M,nh,nkv,K", [(1, 2, 1, 256), (6, 28, 4, 640), (8, 40, 8, 384)])
def test_small_qkv_rope(ops, M, nh, nkv, K):
    N, bs = (nh + 2 * nkv) * 128, 16
    p, wd = _part(N, K, 9)
    bias = (torch.randn(N, device="cuda") * 0.1).half()
    w = ops.make_linear([p], K, 128, bias)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    ang = torch.arange(64, device="cuda")[:, None] * 10000.0 ** (-torch.arange(64, device="cuda") / 64)
    table = torch.stack([ang.cos(), ang.sin()], -1).float().contiguous()
    pos = torch.randint(0, 64, (M,), dtype=torch.int32, device="cuda")
    slots = torch.randperm(4 * bs, device="cuda")[:M].to(torch.int64)
    slots[0] = -1
    kv = torch.full((4, 2, nkv, bs, 128), 7.0, dtype=torch.float16, device="cuda")
    qkv = torch.full((M, N), 7.0, dtype=torch.float16, device="cuda")
    native.gemm_w4_dec_qkv_rope(w.data, x, M, w.bias, qkv, N, M, K, nh, nkv, kv, bs, pos, slots, table, 64, ops.dec_ws,
                                ops.status.ptr)
    torch.cuda.synchronize()
    ops.check()
    y = (x.double() @ wd.T + bias.double()).view(M, nh + 2 * nkv, 128)
    c, s = table[pos.long(), :, 0].double()[:, None], table[pos.long(), :, 1].double()[:, None]
    a, b = y[:, : nh + nkv, :64], y[:, : nh + nkv, 64:]
    turned = torch.cat([a * c - b * s, b * c + a * s], -1)
    assert _rel(qkv[:, : nh * 128], turned[:, :nh].reshape(M, -1)) < 5e-4
    for m in range(1, M):
        blk, off = divmod(int(slots[m]), bs)
        assert _rel(kv[blk, 0, :, off], turned[m, nh:]) < 6e-4 and _rel(kv[blk, 1, :, off], y[m, nh + nkv:]) < 6e-4
    assert int((kv != 7).any(-1).any(2).any(1).sum()) == M - 1      # nothing else was written


@pytest.mark.parametrize("M,N,K", [(1, 256, 640), (2, 4864, 256), (8, 200, 2176)])
def test_small_infinite_activation(ops, M, N, K):
    """An infinite activation times a weight that is not zero is infinite, of the product's sign: 65504 where outputs are fp16."""
    p, _ = _part(N, K, K)
    q = np.stack([p["data"] & 15, p["data"] >> 4], -1).reshape(N, -1, 128)
    w = (q * p["scales"][..., None].astype(np.float32) + p["zeros"][..., None].astype(np.float32)).astype(np.float16).reshape(N, K)
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    at = [(37 * m + 5) % K for m in range(M)]
    for m in range(0, M, 2):                                  # the other tokens are finite
        x[m, at[m]] = float("inf") if m % 4 == 0 else float("-inf")
    out = torch.zeros(M, N, dtype=torch.float16, device="cuda")
    ops.linear(ops.make_linear([p], K, 128), x, M, out)
    planes = torch.zeros(8, M, N, dtype=torch.float32, device="cuda")
    n = ops.linear_partial(ops.make_linear([p], K, 128), x, M, planes)
    torch.cuda.synchronize()
    ops.check()
    want = x.double() @ torch.from_numpy(w).cuda().double().T
    for m in range(M):
        if m % 2:
            assert torch.isfinite(out[m]).all() and _rel(planes[:n, m].double().sum(0), want[m]) < 5e-4
            continue
        col = torch.from_numpy(w[:, at[m]]).cuda().float()
        sign = torch.sign(col) * torch.sign(x[m, at[m]].float())
        ok = col != 0
        assert int(ok.sum()) > N // 2 and torch.equal(out[m][ok].float(), 65504 * sign[ok])
        assert torch.equal(planes[:n, m].sum(0)[ok], float("inf") * sign[ok])


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K", [(1024, 8192), (200, 6400), (3584, 14336)])
def test_narrow_and_deep_layers(ops, M, N, K):
    """Layers that the register-streamed kernel leaves to a cluster along K; the planes of the same layers are its own."""
    assert native.gemm_w4_plan(M, N, K, 0)[3] != -1 and native.gemm_w4_plan(M, N, K, 2)[3] == -1
    p, wd = _part(N, K, 5)
    bias = (torch.randn(N, device="cuda") * 0.1).half()
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    out = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    ops.linear(ops.make_linear([p], K, 128, bias), x, M, out)
    torch.cuda.synchronize()
    ops.check()
    # weights and the result rounded to fp16: 2^-11 each at most
    assert _rel(out[:M], x.double() @ wd.T + bias.double()) < 1e-3 and (out[M:] == 7).all()
