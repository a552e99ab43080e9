"""The float32 product's working memory: a step takes it from the runner's workspace, made once for the largest step."""
import threading

import pytest
import torch

from tests import gpu_harness as G
from tests import helpers as H


def test_the_buffer_is_a_threads_own_and_is_put_back():
    from mashbox_b200 import ops
    now = lambda: getattr(ops._float32_planes, "buffer", None)
    one, two, seen = object(), object(), []
    with ops.float32_planes(one):
        t = threading.Thread(target=lambda: seen.append(now()))
        t.start()
        t.join()
        with pytest.raises(ValueError):
            with ops.float32_planes(two):
                seen.append(now())
                raise ValueError
        assert now() is one
    assert seen == [None, two] and now() is None


@pytest.mark.gpu
def test_float32_products_of_a_step_allocate_nothing(tmp_path):
    """the first step of any size makes the buffers for the largest; after that a step asks the allocator for no more than the two
    lists of block-table entries that changed, where its products are nine and more"""
    from mashbox_b200.engine.engine import Engine
    folder = H.make_folder(tmp_path, "C", "float32")
    eng = Engine.from_folder(folder, dtype="float32", device=G.DEV, page_size=16, max_tokens=2048, max_requests=4,
                             max_tokens_per_step=600, options={"no_graphs": True})
    run = eng.runner
    short, long, more = H.prompts_for("C", (5, 500, 590), seed=4)
    for name in ("a", "b", "c"):
        eng.cache.admit(name)
    run.step([("a", short, [4])])
    size = run.ws.buffers[("float32_planes", (), torch.bfloat16)].numel()
    run.step([("b", long, [499])])
    run.check()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    run.step([("c", more, [589])])
    run.step([("a", [7], [0]), ("b", [9], [0])])
    assert torch.cuda.memory_stats()["allocation.all.allocated"] <= before + 4
    assert run.ws.buffers[("float32_planes", (), torch.bfloat16)].numel() == size
    run.check()


@pytest.mark.gpu
def test_slabs_in_a_buffer_give_the_same_bits(monkeypatch):
    from mashbox_b200 import ops
    g = torch.Generator().manual_seed(1)
    a, w = torch.randn(700, 260, generator=g).to(G.DEV), torch.randn(100, 260, generator=g).to(G.DEV)
    whole, asked = ops.linear(a, w), []

    def buffer(rows, most, Kp):
        asked.append((rows, most, Kp))
        return torch.full((3 * rows * Kp + 8,), float("nan"), dtype=torch.bfloat16, device=G.DEV)
    monkeypatch.setattr(ops, "F32_SPLIT_PLANE", 300 * 264)
    with ops.float32_planes(buffer):
        assert torch.equal(ops.linear(a, w), whole)
    assert asked == [(300, 300, 264)]
