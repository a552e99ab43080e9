"""Which steps of the linear-attention layers run the chunk form (ops.linear_chunks_shortest, parts/base.py: plan_chunks), on the
CPU: by the lengths of the step's sequences, since a record of a few tokens costs as much as one of 32."""
import random
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from mashbox_b200 import ops
from mashbox_b200.parts.base import StepInputs, Workspace, chunked_recurrence, plan_chunks

# heads, dim, vdim of the benchmark's smallest decoders
SIZES = {"delta": (16, 128, 128), "channels": (24, 128, 128), "heads": (48, 128, 64), "wkv": (16, 128, 128), "fixed": (16, 128, 128)}


def context(lengths, dtype=torch.bfloat16, rows=2112):
    calls = []
    fake = SimpleNamespace(CHUNKS=ops.CHUNKS, linear_chunks_shortest=ops.linear_chunks_shortest, linear_chunks_slots=ops.linear_chunks_slots,
                           linear_chunks_floats=lambda H, dim, vdim, mode: H * 4, linear_chunks=lambda *a, **k: calls.append(k))
    ctx = SimpleNamespace(dtype=dtype, ops=fake, q_len=lengths, N=sum(lengths), S=len(lengths), memo={}, inputs=StepInputs(None),
                          ws=Workspace("cpu", rows), dev=lambda name: None)
    return ctx, calls


@pytest.mark.parametrize("mode", SIZES)
def test_by_the_lengths_of_the_sequences(mode):
    H, dim, vdim = SIZES[mode]
    at = lambda *lengths: ops.linear_chunks_shortest(list(lengths), H, dim, vdim, mode)
    assert at(2048) and at(*[1000] + [1] * 63) and at(*[512] * 4) and at(128)
    # measured slower than the scan: short sequences, however many (fixed decays, 16 of 33 tokens: 87 us against 59)
    assert not at(*[31] * 10) and not at(*[33] * 16) and not at(*[48] * 16) and not at(*[2] * 300) and not at(*[63] * 30)
    assert not at(65) and not at(*[1] * 2000)
    # a sequence that is hardly long enough beside short ones, which take a scan of their own
    assert not at(100, *[20] * 10) and not at(96, *[1] * 8)
    # beside a long one, sequences of 32 tokens and more go with it: no scan for them alone
    assert at(1531, 300, 37) == 32 and at(*[1000] + [50] * 8) == 32
    assert at(*[1000] + [33] * 8) == (48 if mode == "delta" else 32)
    # sizes that the kernels do not take
    assert not ops.linear_chunks_shortest([2048], H, 256, vdim, mode) and not ops.linear_chunks_shortest([2048], H, dim, 30, mode)


@pytest.mark.parametrize("mode", SIZES)
def test_every_sequence_once_and_the_scratch_holds_the_chunks(mode):
    H, dim, vdim = SIZES[mode]
    rng = random.Random(1)
    for _ in range(300):
        lengths = [rng.choice([1, 1, 31, 32, 33, 63, 64, 79, 80, 95, 96, 159, 160, 161, 500]) for _ in range(rng.randint(1, 40))]
        ctx, calls = context(lengths)
        plan_chunks(ctx, mode, H, dim, vdim)
        ran = chunked_recurrence(ctx, mode, *[None] * 6, H, H, dim, vdim)
        if not ran:
            assert not calls and ops.linear_chunks_shortest(lengths, H, dim, vdim, mode) == 0
            continue
        shortest, rest, scratch = calls[0]["shortest"], calls[0]["rest"], calls[0]["scratch"]
        long = [n for n in lengths if n >= shortest]
        assert shortest in (32, 48) and max(long) >= min(ops.CHUNKS[mode]) and rest == (len(long) < len(lengths))
        assert sum(-(-n // 32) for n in long) * H * 4 <= scratch.numel()


def test_the_decision_is_part_of_a_captured_steps_shape():
    """the same number of tokens and sequences, long and short: other arrays, so another graph"""
    seen = {}
    for lengths in ([1000, 24], [512, 512], [24, 1000]):
        ctx, _ = context(lengths)
        plan_chunks(ctx, "delta", 16, 128, 128)
        plan_chunks(ctx, "delta", 16, 128, 128)                    # another layer of these sizes
        seen[tuple(lengths)] = ctx.inputs.signature()
        assert len(ctx.inputs.arrays) == 1
    assert seen[1000, 24] == seen[24, 1000] != seen[512, 512]
    ctx, calls = context([1024], dtype=torch.float32)              # one order of sums in every cut
    plan_chunks(ctx, "delta", 16, 128, 128)
    assert not chunked_recurrence(ctx, "delta", *[None] * 6, 16, 16, 128, 128) and not calls
    assert all(len(a) == 0 for a in ctx.inputs.arrays.values())


def test_one_scratch_for_all_layers():
    """two kinds of layers share one buffer, which the largest step does not make grow"""
    ctx, calls = context([300, 200])
    for mode, H in (("channels", 24), ("heads", 48)):
        plan_chunks(ctx, mode, H, 128, 64)
        assert chunked_recurrence(ctx, mode, *[None] * 6, H, H, 128, 64)
    assert len(ctx.ws.buffers) == 1
    made = ctx.ws.generation
    for lengths in ([64] * 33, [2112], [80] * 26, [500] * 4 + [1] * 60):
        step, _ = context(lengths)
        step.ws = ctx.ws
        for mode, H in (("channels", 24), ("heads", 48)):
            plan_chunks(step, mode, H, 128, 64)
            assert chunked_recurrence(step, mode, *[None] * 6, H, H, 128, 64) or max(lengths) < 80
    assert ctx.ws.generation == made and len(ctx.ws.buffers) == 1
