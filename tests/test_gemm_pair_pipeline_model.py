"""Host model of the barrier protocol of the paired quantised GEMM (csrc/gemm_pair.cu).

Two CTAs, each with a weight loader, an activation loader and four dequantisation groups (two of their four warps stand for
all) that also run the epilogues; one MMA issuer for both.  Coroutines under a random scheduler; copies complete in any
order (``late``: now and then one is overtaken by all that were issued after it), MMA commits in issue order, their arrivals
in the two CTAs at different times.  Every parity test is checked against the phase it stands for, every ring slot, operand
slot and the accumulator against refills while somebody needs them, and every run has to end.  No GPU is involved.
"""
import os
import random
import re

import pytest

from test_attention_tc_pipeline_model import Bar

WARPS = 2


def run(units, SW, S, seed, late=False):
    """``units``: K chunks of each unit in turn; ``SW``, ``S``: weight ring, operand slots."""
    rnd = random.Random(seed)
    total = sum(units)
    owner = [j for j, n in enumerate(units) for _ in range(n)]         # unit of every chunk
    two = lambda n, count: [[Bar(count) for _ in range(n)] for _ in range(2)]
    w_full, w_empty, done = two(SW, 1), two(SW, WARPS), two(S, 1)
    acc_full = [Bar(1), Bar(1)]
    x_full = [Bar(3) for _ in range(S)]              # the leader's arrival and the bytes of both CTAs
    a_ready = [Bar(2 * WARPS) for _ in range(S)]
    acc_empty = Bar(8 * WARPS)
    w_slot = [[None] * SW for _ in range(2)]
    x_slot = [[None] * S for _ in range(2)]
    operand = [[None] * S for _ in range(2)]
    acc = [None]                                     # unit whose sums the accumulator holds
    copies, commits, arrivals, finished = [], [], [], []

    def wait(bar, parity, want):
        while not bar.test(parity, want):
            yield

    def w_loader(c):
        s, ph = 0, 1
        for u in range(total):
            if u >= SW:
                yield from wait(w_empty[c][s], ph, u // SW - 1)
            w_slot[c][s] = u
            copies.append(w_full[c][s])
            s += 1
            if s == SW:
                s, ph = 0, ph ^ 1
            yield

    def x_loader(c):
        for u in range(total):
            s = u % S
            if u >= S:
                yield from wait(done[c][s], (u // S - 1) & 1, u // S - 1)
            x_slot[c][s] = u
            if c == 0:
                x_full[s].arrive()
            yield
            copies.append(x_full[s])

    def issuer():
        u = 0
        for j, n in enumerate(units):
            if j > 0:
                yield from wait(acc_empty, (j - 1) & 1, j - 1)
            acc[0] = j
            for _ in range(n):
                s = u % S
                yield from wait(x_full[s], (u // S) & 1, u // S)
                yield from wait(a_ready[s], (u // S) & 1, u // S)
                assert all(x_slot[c][s] == u and operand[c][s] == u for c in range(2))
                commits.append([done[0][s], done[1][s]])
                u += 1
                yield
            commits.append(list(acc_full))

    def group(c, g, w):
        sw, wph, slot, sph, first, nxt, epi = g, 0, g, 1, 0, g, 0

        def finish():
            nonlocal epi
            yield from wait(acc_full[c], epi & 1, epi)
            assert acc[0] == epi, "the accumulator was overwritten"
            yield
            acc_empty.arrive()
            epi += 1
            yield

        for j, n in enumerate(units):
            while nxt < first + n:
                yield from wait(w_full[c][sw], wph, nxt // SW)
                assert w_slot[c][sw] == nxt
                if nxt >= S:
                    yield from wait(done[c][slot], sph, nxt // S - 1)
                assert slot == nxt % S
                operand[c][slot] = nxt
                yield
                assert w_slot[c][sw] == nxt
                w_empty[c][sw].arrive()
                yield
                a_ready[slot].arrive()
                sw += 4
                if sw >= SW:
                    sw, wph = sw - SW, wph ^ 1
                slot += 4
                if slot >= S:
                    slot, sph = slot - S, sph ^ 1
                nxt += 4
                while epi < j:
                    yield from finish()
            first += n
        while epi < len(units):
            yield from finish()
        finished.append((c, g, w))

    agents = ([w_loader(c) for c in range(2)] + [x_loader(c) for c in range(2)] + [issuer()]
              + [group(c, g, w) for c in range(2) for g in range(4) for w in range(WARPS)])
    live = list(range(len(agents)))
    for _ in range(2000000):
        if not live and not copies and not commits and not arrivals:
            break
        r = rnd.random()
        if r < 0.12 and commits:
            arrivals.append(commits.pop(0))
        elif r < 0.24 and arrivals:
            pair = arrivals[0]
            pair.pop(rnd.randrange(len(pair))).arrive()
            if not pair:
                arrivals.pop(0)
        elif r < 0.4 and copies:
            i = rnd.randrange(len(copies))
            if not late or i > 0 or rnd.random() < 0.003:
                copies.pop(i).arrive()
        elif live:
            i = rnd.choice(live)
            try:
                next(agents[i])
            except StopIteration:
                live.remove(i)
    else:
        raise AssertionError("the roles did not finish: a wait never came true")
    assert len(finished) == 8 * WARPS and owner[-1] == len(units) - 1


@pytest.mark.parametrize("SW,S", [(4, 4), (8, 4), (8, 5), (12, 6), (16, 7)])
@pytest.mark.parametrize("units", [[1], [3], [4, 4], [1, 1, 1, 1, 1], [2, 3, 2, 3], [5, 5, 5], [7, 6, 7], [12, 11], [28]])
def test_pair_protocol(units, SW, S):
    for seed in range(8):
        run(units, SW, S, seed)


@pytest.mark.parametrize("SW,S", [(4, 4), (8, 5), (8, 6), (16, 7)])
def test_a_late_copy_is_not_taken_for_another(SW, S):
    for seed in range(20):
        run([9, 2, 9, 9], SW, S, seed, late=True)


def test_the_kernel_has_the_depths_that_are_modelled():
    text = open(os.path.join(os.path.dirname(__file__), "..", "csrc", "gemm_pair.cu")).read()
    assert re.search(r"kPairMaxSlots = 7;", text) and re.search(r"kPairMaxSW = 16;", text) and "/ chunk / 4 * 4" in text
