"""Decode-form sequences of very different lengths, cut in proportion to them: the work list on the CPU, and on the GPU the
same attention as with equal splits."""
import random

import numpy as np
import pytest
import torch

from mashbox_b200.parts import attention as A
from tests import test_attention_plan as T


def longest(dec, lengths, window=None):
    """key tiles of a plan's longest block (one new token a sequence)"""
    t = lambda n: -(-n // 64) - (max(0, n - window) // 64 if window else 0)
    return max(-(-t(lengths[s]) // ns) for s, m, _, ns in dec if m == 0)


@pytest.mark.parametrize("lengths", [[700, 64], [512, 2048], [128, 512], [600, 600, 600, 1500], [64, 192], [3545, 67], [64] * 15 + [480],
                                     [200, 300, 100, 500, 64, 96, 400, 128], [4096, 64] * 32])
def test_short_batches_keep_the_plan_whose_splits_meet_cheaply(lengths):
    """measured slower when cut in proportion: the longest block gets hardly shorter, and its splits meet through global memory"""
    p, dec, pre, part_base, part_tok = T.plan(lengths, [1] * len(lengths))
    q, even, *_ = T.plan(lengths, [1] * len(lengths), dict(attention_uneven_splits=False))
    assert not p["uneven"] and p["cluster"] == q["cluster"] and np.array_equal(dec, even)
    T.check_cover(p, dec, pre, part_base, part_tok, lengths, [1] * len(lengths))


@pytest.mark.parametrize("lengths", [[4096] + [256] * 7, [16384, 128], [128, 300, 700, 1500, 3000, 4096] * 6 + [2000], [4096] + [300] * 40,
                                     [12995, 130, 82], [4096] + [64] * 63])
def test_batches_that_would_wait_for_one_block_are_cut_in_proportion(lengths):
    new = [1] * len(lengths)
    p, dec, pre, part_base, part_tok = T.plan(lengths, new)
    q, even, *_ = T.plan(lengths, new, dict(attention_uneven_splits=False))
    assert p["uneven"] and not p["cluster"] and not q["uneven"]
    T.check_cover(p, dec, pre, part_base, part_tok, lengths, new)
    assert longest(dec, lengths) < longest(even, lengths)


def test_the_cut_stays_while_the_sequences_grow():
    """37 requests of 190 to 4,400 tokens, whose equal splits would change from two to three on the way"""
    r = random.Random(3)
    start = [int(round(np.exp(r.uniform(np.log(128), np.log(4096))))) for _ in range(37)]
    for t in range(0, 300, 10):
        p, dec, *_ = T.plan([n + t for n in start] + [1] * 3, [1] * 40, heads=24)
        assert p["uneven"] and len(dec) == 96


def test_random_batches():
    """log-spread lengths: never a longer block than in the plan of equal splits where the device is not crowded, as many places
    in the partial buffers as decode-form tokens, and a work list that grows with the sequences changes its length seldom"""
    rng = random.Random(3)
    used = 0
    for _ in range(400):
        S, kv = rng.randint(2, 70), rng.choice([2, 4, 8])
        lengths = [int(64 * 256 ** rng.random()) for _ in range(S)]
        new = [1] * S if rng.random() < 0.7 else [min(n, rng.choice([1, 1, 4, 700])) for n in lengths]
        window, G = rng.choice([None, None, 1000]), 32 // kv
        p, dec, pre, part_base, part_tok = T.plan(lengths, new, kv=kv, window=window)
        T.check_cover(p, dec, pre, part_base, part_tok, lengths, new, G)
        if not p["uneven"]:
            continue
        used += 1
        assert len(part_tok) == sum(q for q in new if q * G <= 16) and len(dec) == A.listed_items(int((dec[:, 1] == 0).sum()))
        if sum(-(-n // 64) for n in lengths) * kv < 16 * 296 and new == [1] * S and window is None:
            _, even, *_ = T.plan(lengths, new, dict(attention_uneven_splits=False), kv=kv)
            assert longest(dec, lengths) + 6 <= longest(even, lengths)
    assert used > 60
    sizes = {len(T.plan([4096 + t] + [256 + t] * 7, [1] * 8)[1]) for t in range(1000)}
    assert len(sizes) <= 3


def test_splits_in_proportion():
    for tiles, items in (([64, 2, 2, 30], 111), ([1] * 40 + [128], 111), ([5, 6, 200] * 30, 180)):
        n = A.uneven_splits(tiles, items, 32)
        assert sum(n) <= items and all(1 <= x <= min(32, max(1, -(-t // 4))) for x, t in zip(n, tiles))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["C", "D"])
def test_uneven_splits_give_the_logits_of_equal_ones(name, tmp_path):
    """heads of 128 and of 64; five requests of 3 to 900 tokens decode side by side, alone and beside a prompt's portion: the
    sums over the keys are cut elsewhere, float32 all the same, so the logits agree to a few roundings of bfloat16"""
    from mashbox_b200.engine.engine import Engine
    from tests import helpers as H
    folder = H.make_folder(str(tmp_path), name, H.store_for("bfloat16"))
    lens, outs, used = [900, 3, 65, 640, 130], [], []
    for uneven in (True, False):
        eng = Engine.from_folder(folder, dtype="bfloat16", device="cuda:0", page_size=16, max_tokens=4096, max_requests=8,
                                 max_context=1024, options=dict(attention_uneven_splits="always" if uneven else False))
        r = np.random.default_rng(1)
        vocab = eng.runner.model.head.vocab if hasattr(eng.runner.model.head, "vocab") else 256
        ids = [r.integers(0, min(vocab, 256), n + 8).tolist() for n in lens]
        for i, n in enumerate(lens):
            eng.runner.cache.admit(i)
            eng.runner.step([(i, ids[i][:n], [])])
        got = []
        for t in range(4):
            step = [(i, ids[i][n + t:n + t + 1], [0]) for i, n in enumerate(lens)]
            if t == 3:
                eng.runner.cache.admit("p")
                step.append(("p", ids[0][:77], [76]))
            ctx = eng.runner.prepare(step)
            plan = next(v for k, v in ctx.memo.items() if k[0] == "attention")
            used.append(plan["uneven"])
            got.append(eng.runner.launch(ctx, step).float().cpu().clone())
        eng.runner.check()
        outs.append(torch.cat(got))
    assert used == [True] * 4 + [False] * 4
    err = float((outs[0] - outs[1]).norm() / outs[1].norm())
    assert err < 1e-2, err
