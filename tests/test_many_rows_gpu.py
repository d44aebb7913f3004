"""Row kernels of passes of many rows (csrc/elementwise.cu, csrc/gemma.cu) against the kernels that passes of few rows take: the
same call on all rows at once and in slices below the line between them.  The arithmetic of an element is the same in both; sums of
squares are added in another order, so a result may move by one unit of fp16 (2^-10 of its size)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -10


@pytest.fixture(scope="module")
def ops():
    from zse_b200.ops.backend import CudaOps
    o = CudaOps("cuda")
    yield o
    o.check()


def _close(a, b, floor):
    a, b = a.float(), b.float()
    return bool(((a - b).abs() <= UNIT * b.abs() + floor).all())


@pytest.mark.parametrize("H", [8, 128, 3584, 5120, 8192, 5124])
@pytest.mark.parametrize("planes,addend", [(0, False), (1, False), (3, True), (9, False)])
def test_add_rmsnorm(ops, H, planes, addend):
    M, step = 595, 119
    g = torch.Generator(device="cuda").manual_seed(H + planes)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    res, part, w = rnd(M, H), rnd(max(planes, 1), M, H), (1 + 0.1 * rnd(H)).half()
    add = rnd(M, H).half() if addend else None
    r1, o1 = res.clone(), torch.empty(M, H, dtype=torch.float16, device="cuda")
    ops.add_rmsnorm(r1, part, planes, add, w, o1, M, 1e-6)
    r2, o2 = res.clone(), torch.empty_like(o1)
    for i in range(0, M, step):
        ops.add_rmsnorm(r2[i:i + step], part[:, i:i + step].contiguous(), planes, None if add is None else add[i:i + step], w,
                        o2[i:i + step], step, 1e-6)
    torch.cuda.synchronize()
    assert torch.equal(r1, r2) and _close(o1, o2, 1e-7)


@pytest.mark.parametrize("H", [8, 2304, 3584, 8192])
@pytest.mark.parametrize("scaled,out", [(False, True), (True, True), (False, False)])
def test_post_norm(ops, H, scaled, out):
    M, step = 600, 200
    g = torch.Generator(device="cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, res, wp, wn = rnd(M, H).half(), rnd(M, H), (0.1 * rnd(H)).half(), (1 + 0.1 * rnd(H)).half()
    sc = torch.tensor([0.75], dtype=torch.float16, device="cuda") if scaled else None
    r1, o1 = res.clone(), torch.zeros(M, H, dtype=torch.float16, device="cuda")
    ops.norm_add_rmsnorm(x, wp, r1, sc, wn, o1 if out else None, M, 1e-6)
    r2, o2 = res.clone(), torch.zeros_like(o1)
    for i in range(0, M, step):
        ops.norm_add_rmsnorm(x[i:i + step], wp, r2[i:i + step], sc, wn, o2[i:i + step] if out else None, step, 1e-6)
    torch.cuda.synchronize()
    assert (r1 - r2).abs().max() < 1e-5 and _close(o1, o2, 1e-5)      # the residual is fp32: sums of squares in another order


@pytest.mark.parametrize("hd,nh,nkv", [(96, 32, 32), (160, 32, 8), (80, 32, 32), (48, 60, 15), (512, 5, 1), (16, 3, 1)])
@pytest.mark.parametrize("M", [1, 33])
def test_rotation_of_heads_that_leave_threads_over(ops, hd, nh, nkv, M):
    """hd / 16 threads a head: where that does not divide the CTA, and there are more heads than fit it at once."""
    bs, half = 16, hd // 2
    g = torch.Generator(device="cuda").manual_seed(hd + M)
    qkv = torch.randn(M, (nh + 2 * nkv) * hd, device="cuda", generator=g).half()
    pos = torch.randint(0, 64, (M,), dtype=torch.int32, device="cuda", generator=g)
    slots = torch.randperm(64, device="cuda", generator=g)[:M].to(torch.int64)
    freqs = 1e4 ** (-torch.arange(half, device="cuda").float() / half)
    kv = torch.full((4, 2, nkv, bs, hd), 7.0, dtype=torch.float16, device="cuda")
    x = qkv.double().view(M, nh + 2 * nkv, hd)
    ops.rope_kv_write(qkv, kv, pos, slots, freqs, M, nh, nkv, hd, bs)
    torch.cuda.synchronize()
    ang = pos.double()[:, None] * freqs.double()
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[:, : nh + nkv, :half], x[:, : nh + nkv, half:]
    turned = torch.cat([a * c - b * s, b * c + a * s], -1)
    # one rounding to fp16, and angles of up to 64 in fp32 (64 * 2^-24) times what is rotated
    close = lambda got, want: bool(((got.double() - want).abs() <= UNIT / 2 * want.abs() + 1e-4).all())
    assert close(qkv.view(M, -1, hd)[:, : nh + nkv], turned)
    blk, off = slots // bs, slots % bs
    assert close(kv[blk, 0, :, off], turned[:, nh:]) and close(kv[blk, 1, :, off], x[:, nh + nkv:])
    assert int((kv != 7).any(-1).any(2).any(1).sum()) == M


@pytest.mark.parametrize("hd,nh,nkv,k_is_v,norm_v", [(256, 16, 8, False, False), (8, 3, 1, False, False), (64, 4, 2, True, True),
                                                     (512, 8, 1, False, True), (200, 2, 2, False, False)])
def test_head_norms(ops, hd, nh, nkv, k_is_v, norm_v):
    M, bs, step = 300, 16, 150
    g = torch.Generator(device="cuda").manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    qkv = rnd(M, (nh + (1 if k_is_v else 2) * nkv) * hd).half()
    pos = torch.randint(0, 30000, (M,), dtype=torch.int32, device="cuda", generator=g)
    slots = torch.randperm(320, device="cuda", generator=g)[:M].to(torch.int64)
    slots[7] = -1
    freqs = 1e4 ** (-torch.arange(hd // 2, device="cuda").float() / (hd // 2))
    freqs[hd // 4:] = 0                                               # a part that does not rotate
    qw, kw = (1 + 0.1 * rnd(hd)).half(), (1 + 0.1 * rnd(hd)).half()
    got = []
    for n in (M, step):
        q, kv = qkv.clone(), torch.full((20, 2, nkv, bs, hd), 7.0, dtype=torch.float16, device="cuda")
        for i in range(0, M, n):
            ops.headnorm_rope_kv_write(q[i:i + n], kv, pos[i:i + n], slots[i:i + n], freqs, qw, kw, norm_v, k_is_v, 1e-6, n, nh,
                                       nkv, hd, bs)
        got.append((q, kv))
    torch.cuda.synchronize()
    assert _close(got[0][0], got[1][0], 2e-3) and _close(got[0][1], got[1][1], 2e-3)   # a unit of what a rotation adds up
    assert torch.equal(got[0][1] == 7, got[1][1] == 7)


def test_pairs_that_do_not_rotate_pass_infinities_through(ops):
    """Frequency 0: an infinite or NaN partner does not reach the other element of the pair."""
    hd, nh, nkv, bs, M, step = 64, 2, 1, 16, 300, 150
    qkv = torch.randn(M, (nh + 2 * nkv) * hd, device="cuda").half()
    qkv[::3, 20], qkv[1::3, 20 + hd // 2], qkv[2::3, hd + 25] = float("inf"), float("nan"), float("-inf")
    qkv[::2, 2 * hd + 30] = float("inf")
    pos = torch.arange(M, dtype=torch.int32, device="cuda")
    slots = torch.arange(M, device="cuda")
    freqs = 1e4 ** (-torch.arange(hd // 2, device="cuda").float() / (hd // 2))
    freqs[hd // 4:] = 0
    got = []
    for n in (M, step):
        q, kv = qkv.clone(), torch.zeros(20, 2, nkv, bs, hd, dtype=torch.float16, device="cuda")
        for i in range(0, M, n):
            ops.headnorm_rope_kv_write(q[i:i + n], kv, pos[i:i + n], slots[i:i + n], freqs, None, None, False, False, 1e-6, n, nh,
                                       nkv, hd, bs)
        got.append((q, kv))
    torch.cuda.synchronize()
    still = torch.arange(hd, device="cuda") % (hd // 2) >= hd // 4
    heads = qkv[:, : nh * hd].view(M, nh, hd)[:, :, still].float()
    heads = torch.nan_to_num(heads, nan=-65504.0).clamp(-65504, 65504)        # (what the clamp before the store makes of them)
    for q, kv in got:
        assert torch.equal(q[:, : nh * hd].view(M, nh, hd)[:, :, still].float(), heads)
    assert _close(got[0][1], got[1][1], 2e-3)


@pytest.mark.parametrize("M,I", [(1, 8), (3, 14336), (70, 264), (5, 2056), (4, 20)])
@pytest.mark.parametrize("gelu", [False, True])
def test_glu(ops, M, I, gelu):
    gu = (torch.randn(M, 2 * I, device="cuda") * 2).half()
    out = torch.full((M + 1, I), 7.0, dtype=torch.float16, device="cuda")
    ops.glu(gu, out, M, I, gelu)
    torch.cuda.synchronize()
    a, b = gu[:, :I].double(), gu[:, I:].double()
    want = (torch.nn.functional.gelu(a, approximate="tanh") if gelu else torch.nn.functional.silu(a)) * b
    assert ((out[:M].double() - want).abs() <= 2 * UNIT * want.abs() + 1e-4).all() and (out[M:] == 7).all()
