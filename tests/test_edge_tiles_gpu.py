"""Tiles on an edge: the general attention looks at every key's place only in tiles that some row sees in part, the grouped
tcgen05 product deals out only tiles that hold rows."""
import math

import pytest
import torch

from tests.gpu_harness import DEV
from tests.plain import lorozen as plain
from tests.test_lorozen_gpu import Step, WindowCase, dev
from tests.test_sufopel_gpu import kernel_close

pytestmark = pytest.mark.gpu
TILE = 64                       # keys of a tile


class CappedCase(WindowCase):
    def scores(self, s, cap):
        return cap * torch.tanh(s / cap) if cap else s

    def want(self, scale, cap=None):
        out = []
        for q, k, v, n, ql in zip(self.q, self.k, self.v, self.lengths, self.q_lens):
            ok = plain.visible(n, dict(size=self.window) if self.window else None)[n - ql:]
            G = self.H // self.KV
            s = self.scores(torch.einsum("ihd,jhd->hij", q[n - ql:], k.repeat_interleave(G, 1)) * scale, cap)
            w = torch.softmax(s.masked_fill(~ok[None], -math.inf), -1)
            out.append(torch.einsum("hij,jhd->ihd", w, v.repeat_interleave(G, 1)).reshape(ql, -1))
        return torch.cat(out)

    def run(self, scale, cap=None, **options):
        from mashbox_b200.parts.attention import PagedAttention
        core = PagedAttention(self.H, self.KV, self.DK, self.window, scale, vdim=self.DV, softcap=cap)
        assert core.general
        step = Step(self.dtype, self.lengths, self.q_lens, self.page, self.pages, options)
        core.prepare(step)
        step.inputs.upload()
        rows = dev(torch.cat([q[n - ql:].reshape(ql, -1) for q, n, ql in zip(self.q, self.lengths, self.q_lens)]), self.dtype)
        out = torch.full((step.N, self.H * self.DV), float("nan"), device=DEV, dtype=torch.bfloat16)
        core.attend(step, rows, rows.stride(0), out, self.table, self.kpool, self.vpool)
        assert int(step.err.item()) == 0
        return out


@pytest.mark.parametrize("H,KV,DK,DV", [(4, 1, 128, 64), (2, 2, 32, 64), (6, 2, 192, 128)])
@pytest.mark.parametrize("cap", [None, 30.0])
def test_a_key_on_a_tiles_edge_is_seen_or_not(H, KV, DK, DV, cap):
    """windows that begin on the first key of a tile, one before and one after, and a last key that is a tile's last, one before and
    one after; the loud key stands on either side of each; decoded tokens, a few, and blocks of rows whose windows begin in
    different tiles"""
    for window in (None, TILE - 1, TILE, TILE + 1, 2 * TILE):
        for n in (2 * TILE, 2 * TILE + 1, 3 * TILE - 1, 4 * TILE + 2):
            q = n - 1
            first = max(0, q - window + 1) if window else 0
            keys = {q, q - 1, first, first - 1, n // TILE * TILE, n // TILE * TILE - 1, (first // TILE + 1) * TILE - 1}
            for kpos in sorted(k for k in keys if 0 <= k <= q):
                seen = first <= kpos
                for ql in (1, 3, TILE + 7):
                    case = CappedCase("bfloat16", H, KV, DK, DV, window, [n, 40], [ql, 1], 16, [(0, q, kpos)], seed=kpos, amount=7.0)
                    got, want = case.run(1.0, cap), case.want(1.0, cap)
                    kernel_close(got, want, "bfloat16", f"window {window} n {n} key {kpos} {ql} queries cap {cap}", 3e-2)
                    assert (float(want[ql - 1].view(H, DV)[:, 0].abs().min()) > 2.0) == seen


@pytest.mark.parametrize("rows", [[128], [0, 0, 1], [129, 0, 127], [128, 128, 0, 5], [1] * 20, [300, 0, 0, 700, 1, 128, 256, 127, 513]])
def test_experts_whose_rows_end_on_a_tiles_edge(rows):
    """rows of every expert: none, one, whole tiles, one more and one fewer, the first and the last expert among those with none;
    more tiles than the device has SMs and fewer"""
    from mashbox_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(len(rows))
    E, N, D, F, bf = len(rows) + 1, max(128, sum(rows)), 64, 1032, torch.bfloat16
    rows = rows + [N - sum(rows)]
    ids = torch.cat([torch.full((r,), e) for e, r in enumerate(rows)])[torch.randperm(N, generator=torch.Generator().manual_seed(1))]
    ids = ids.to(DEV, torch.int32)[:, None].contiguous()
    new = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=DEV) * scale).to(bf)
    h, wgu, wd = new(N, D), new(E, 2 * F, D, scale=D ** -0.5), new(E, D, F, scale=F ** -0.5)
    wts = torch.rand(N, 1, generator=g, device=DEV)
    T = ops.moe_tc5_tiles(N, 1, E)
    out = torch.full((N, D), float("nan"), device=DEV, dtype=bf)
    buf, act = torch.empty(128 * T, D, device=DEV, dtype=bf), torch.empty(128 * T, F, device=DEV, dtype=bf)
    y, scratch = torch.empty(128 * T, D, device=DEV), torch.empty(N + T, dtype=torch.int32, device=DEV)
    ops.moe_tc5(h, ids, wts, wgu, wd, out, buf, act, y, scratch, 1e30, 1.0, shift=0.0)
    ops.check_error_word(ops.error_word(DEV))
    want = torch.empty(N, D, device=DEV, dtype=torch.float64)
    for e in range(E):
        at = (ids[:, 0] == e).nonzero()[:, 0]
        z = h[at].double() @ wgu[e].double().T
        gate, up = z[:, :F].to(bf).double(), z[:, F:].to(bf).double()
        want[at] = (gate * torch.sigmoid(gate) * up).to(bf).double() @ wd[e].double().T * wts[at].double()
    kernel_close(out, want.cpu(), "bfloat16", f"rows {rows}", 1e-2)
