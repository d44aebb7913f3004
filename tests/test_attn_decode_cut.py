"""Decode attention over sequences of unequal length (csrc/attention.cu): equal shares of 16-token tiles for every CTA, items cut
anywhere.  The arithmetic of the cut on the CPU; results against float64 on the GPU, for every head size, group size and bound on
the pieces, with windows, soft caps, dropped blocks and empty sequences."""
import math
import random

import pytest
import torch


def _per(total, longest, ctas, splits):
    return max(4, -(-total // ctas), (longest + splits - 3) // (splits - 2))


def test_no_item_is_cut_into_more_pieces_than_scratch_holds():
    rnd = random.Random(1)
    for _ in range(3000):
        nkv, splits, ctas = rnd.choice([1, 2, 4, 8]), rnd.randint(3, 16), rnd.choice([148, 296, 592])
        lens = [rnd.choice([0, 1, rnd.randint(1, 40), rnd.randint(1, 2000)]) for _ in range(rnd.randint(1, 40))]
        per, start, used = _per(sum(lens) * nkv, max(lens), ctas, splits), 0, 0
        for n in lens:
            for _ in range(nkv if n else 0):
                pieces = (start + n - 1) // per - start // per + 1
                assert 1 <= pieces <= splits - 1
                start += n
                used = (start - 1) // per + 1
        assert used <= ctas


def _case(S, nh, nkv, hd, bs, lens, seed=0, holes=0.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    blocks = [-(-n // bs) for n in lens]
    kv = torch.randn(sum(blocks) + 3, 2, nkv, bs, hd, device="cuda", generator=g).half()
    q = torch.randn(S, nh * hd, device="cuda", generator=g).half()
    order = torch.randperm(sum(blocks) + 3, generator=torch.Generator().manual_seed(seed)).tolist()
    bt = torch.full((S, max(blocks + [1]) + 1), -1, dtype=torch.int32)
    rnd = random.Random(seed)
    for s, n in enumerate(blocks):
        for i in range(n):
            blk = order.pop()
            bt[s, i] = -1 if i + 1 < n and rnd.random() < holes else blk      # (the last block is never dropped)
    return q, kv, bt.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")


def _want(q, kv, bt, lens, nh, nkv, hd, bs, scale, softcap, window):
    out = torch.zeros(q.shape[0], nh, hd, dtype=torch.float64, device="cuda")
    for s, n in enumerate(lens.tolist()):
        if n == 0:
            continue
        table = bt[s, : -(-n // bs)].long()
        k, v = (kv[table.clamp(min=0), i].double().transpose(1, 2).reshape(-1, nkv, hd)[:n] for i in range(2))
        pos = torch.arange(n, device="cuda")
        seen = (table >= 0).repeat_interleave(bs)[:n] & (pos >= n - window if window else pos >= 0)
        k, v = (t.repeat_interleave(nh // nkv, 1) for t in (k, v))
        x = torch.einsum("hd,nhd->hn", q[s].view(nh, hd).double(), k) * scale
        x = torch.tanh(x / softcap) * softcap if softcap else x
        out[s] = torch.einsum("hn,nhd->hd", torch.softmax(x.masked_fill(~seen, -math.inf), -1), v)
    return out.view(q.shape[0], -1)


@pytest.mark.gpu
@pytest.mark.parametrize("hd,nh,nkv,bs,softcap,window", [(128, 28, 4, 16, 0, 0), (128, 40, 8, 32, 0, 0), (128, 16, 1, 48, 0, 0),
                                                         (128, 4, 4, 16, 0, 200), (256, 16, 8, 16, 50.0, 300), (256, 9, 1, 32, 0, 0),
                                                         (64, 12, 1, 64, 30.0, 0), (64, 14, 2, 16, 0, 0)])
@pytest.mark.parametrize("splits", [1, 2, 7, 16])
@pytest.mark.parametrize("lens", [[1], [517], [0, 3, 3000, 16, 0, 129, 700, 17], [40 * i % 901 for i in range(70)], [5000, 16, 15]])
def test_decode_attention(hd, nh, nkv, bs, softcap, window, splits, lens):
    from zse_b200.ops.backend import CudaOps
    ops, S = CudaOps("cuda"), len(lens)
    q, kv, bt, ln = _case(S, nh, nkv, hd, bs, lens, seed=len(lens) + hd, holes=0.2 if bs == 32 else 0.0)
    out = torch.full((S, nh * hd), 7.0, dtype=torch.float16, device="cuda")
    scratch = torch.full((S * nh * splits * (hd + 2),), float("nan"), device="cuda")
    ops.attn_decode(q, kv, bt, ln, out, S, nh, nkv, hd, bs, hd ** -0.5, scratch, splits, softcap=softcap, window=window)
    torch.cuda.synchronize()
    ops.check()
    want = _want(q, kv, bt, ln, nh, nkv, hd, bs, hd ** -0.5, softcap, window)
    # probabilities and the result in fp16 (2^-11 each), keys and values exact
    assert float((out.double() - want).norm() / want.norm()) < 1.2e-3
    assert (out[ln == 0] == 0).all() and torch.isfinite(out).all()


@pytest.mark.gpu
@pytest.mark.parametrize("splits,lens", [(64, [4096, 30]), (33, [9000]), (34, [9000, 1]), (16, [(7 * i) % 90 for i in range(300)]),
                                         (5, [900] + [0] * 2100 + [50])])
def test_many_pieces_and_many_sequences(splits, lens):
    """More pieces than a warp has lanes, more sequences than one window of 32, sequences of nothing in between."""
    test_decode_attention(128, 8, 2, 16, 0, 0, splits, lens)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[3000], [1, 0, 16, 17, 700]])
def test_two_pieces_are_two(lens):
    """num_splits = 2: half of every sequence in each record, whatever its length; the records add up to the output."""
    from zse_b200.ops.backend import CudaOps
    nh, nkv, hd, bs = 8, 2, 128, 16
    ops, S = CudaOps("cuda"), len(lens)
    q, kv, bt, ln = _case(S, nh, nkv, hd, bs, lens)
    out = torch.full((S, nh * hd), 7.0, dtype=torch.float16, device="cuda")
    scratch = torch.full((S, nh, 2, hd + 2), float("nan"), device="cuda")
    ops.attn_decode(q, kv, bt, ln, out, S, nh, nkv, hd, bs, hd ** -0.5, scratch, 2)
    torch.cuda.synchronize()
    ops.check()
    o, m, l = scratch[..., :hd].double(), scratch[..., hd].double(), scratch[..., hd + 1].double()
    for s, n in enumerate(lens):
        assert bool((l[s, :, 0] > 0).all()) == (n > 0) and bool((l[s, :, 1] > 0).all()) == (n > 16)
    f = torch.where(l > 0, torch.exp2(m - m.amax(2, keepdim=True)), 0.0)
    merged = (o * f[..., None]).sum(2) / (l * f).sum(2).clamp(min=1e-30)[..., None]
    assert (out.view(S, nh, hd).double() - merged).abs().max() <= 2.0 ** -11 * merged.abs().max() + 1e-6
