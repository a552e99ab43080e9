"""Decode-form sequences of very different lengths, cut in proportion to them: the work list on the CPU, and on the GPU the
same attention as with equal splits."""
import random

import numpy as np
import pytest
import torch

from mashbox_b200.parts import attention as A
from tests import test_attention_plan as T


def test_every_key_tile_once_and_as_many_items_as_the_sequences_say():
    rng = random.Random(3)
    used = 0
    for _ in range(300):
        S, kv = rng.randint(2, 70), rng.choice([2, 4, 8])
        lengths = [rng.choice([1, 2, 63, 64, 65, 500, 4096, 20000]) for _ in range(S)]
        new = [1] * S if rng.random() < 0.5 else [min(n, rng.choice([1, 1, 4, 700])) for n in lengths]
        p, dec, pre, part_base, part_tok = T.plan(lengths, new, kv=kv, window=rng.choice([None, None, 1000]))
        rows = [s for s, _, _, _ in dec]
        real = [tuple(r) for r in dec if r[1] == 0]
        decoding = [s for s, q in enumerate(new) if q * (32 // kv) <= 16]
        if not p["uneven"]:
            continue
        T.check_cover(p, dec, pre, part_base, part_tok, lengths, new, 32 // kv)
        by = {s: [(sp, ns) for t, _, sp, ns in real if t == s] for s in decoding}
        assert all(by[s] == [(i, len(by[s])) for i in range(len(by[s]))] and 1 <= len(by[s]) <= 32 for s in decoding)
        if len(dec) > len(real):
            used += 1
            assert len(dec) == max(2 * len(decoding), -(-3 * 296 // kv)) and len(part_tok) == sum(new[s] for s in decoding)
            assert all(r[1] * 16 >= 1 << 20 and r[3] == 1 for r in dec[len(real):])
            # the splits of a sequence stand side by side (the merge counts them from the first)
            assert all(rows[i] == s for s in decoding for i in range(rows.index(s), rows.index(s) + len(by[s])))
    assert used > 30


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
                                 max_context=1024, options=dict(attention_uneven_splits=uneven))
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
