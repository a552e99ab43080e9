"""-m gpu: both heights of the tiles of the routed experts' products (gemm_experts.cu): the same bits, and blocks that go through
many tiles, against float64."""
import pytest
import torch

from tests import gpu_harness as G

pytestmark = pytest.mark.gpu


def check(rows, D, F, weigh, most):
    import mashbox_b200.ops as ops
    E, N = len(rows), sum(rows)
    g = torch.Generator().manual_seed(N)
    r = lambda *s: torch.randn(*s, generator=g).to(G.DEV)
    h, wts = r(N, D).bfloat16(), torch.rand(N, 1, generator=g).to(G.DEV)
    wgu, wd = (r(E, 2 * F, D) * D ** -0.5).bfloat16(), (r(E, D, F) * F ** -0.5).bfloat16()
    ids = torch.cat([torch.full((n,), e) for e, n in enumerate(rows)])[torch.randperm(N, generator=g)].int().to(G.DEV)[:, None]
    T = ops.moe_tc5_tiles(N, 1, E)
    e = lambda *s, t=torch.bfloat16: torch.full(s, float("nan"), dtype=t, device=G.DEV)
    out, buf, act, y = e(N, D), e(128 * T, D), e(128 * T, F), e(128 * T, D, t=torch.float32)
    scale = e(128 * T, t=torch.float32) if weigh == "input" else None
    ops.moe_tc5(h, ids, wts, wgu, wd, out, buf, act, y, torch.zeros(N + T, dtype=torch.int32, device=G.DEV), 7.0, 1.702, 1.0,
                row_scale=scale, most=most)
    ops.check_error_word(ops.error_word(out.device))
    want = torch.zeros(N, D, dtype=torch.float64, device=G.DEV)
    for x in range(E):
        n = (ids[:, 0] == x).nonzero()[:, 0]
        if n.numel():
            s = wts[n].double()
            gu = h[n].double() @ wgu[x].double().T * (s if scale is not None else 1)
            a, u = gu[:, :F].clamp(max=7.0), gu[:, F:].clamp(-7.0, 7.0)
            want[n] = (a * torch.sigmoid(1.702 * a) * (u + 1)) @ wd[x].double().T * (1 if scale is not None else s)
    # gate, up, their gated product and the result are rounded to bf16 (2^-9 each, the gate's slope at most 1.1 beside it)
    assert float((out.double() - want).norm() / want.norm()) < 4 * 2.0 ** -9
    assert float((out.double() - want).abs().max()) < 0.05 * float(want.abs().max())
    return out


@pytest.mark.parametrize("rows,D,F", [
    ([1, 15, 16, 17, 0, 63, 64, 65], 64, 136), ([127, 128, 129, 255, 0, 0, 256, 257], 200, 264), ([513, 0, 1, 300], 1024, 72),
    ([0] * 2100 + [40, 0, 90], 72, 24)])
@pytest.mark.parametrize("most", [(256, 256), (128, 128), (256, 128), (128, 256)])
def test_both_heights_of_a_tile_give_the_same_bits(rows, D, F, most):
    assert torch.equal(check(rows, D, F, "output", most), check(rows, D, F, "output", None))


# a block goes through three units and more, wide ones and narrow ones in turn: the accumulators change hands in both parities and
# the ring of stages (K has 5 blocks of 64) runs on from unit to unit.  48 tiles of 256 rows x 11 of W's, in either product
@pytest.mark.parametrize("D,F", [(264, 1288), (2568, 264)])
@pytest.mark.parametrize("most", [(256, 256), (128, 128)])
@pytest.mark.parametrize("weigh", ["output", "input"])
def test_a_block_goes_through_many_units(D, F, most, weigh):
    check([256, 1, 130, 17] * 12, D, F, weigh, most)
