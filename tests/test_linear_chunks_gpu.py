"""The chunk form of the linear-attention recurrences: every kind against the recurrence in float64, token by token, and
against the token-by-token kernels -- on the edges of chunks, across portions, in slots and groups of their own."""
import numpy as np
import pytest
import torch

from tests.gpu_harness import DEV, i32

pytestmark = pytest.mark.gpu

KINDS = ("delta", "channels", "heads", "wkv", "fixed")


def recurrence(kind, q, k, v, g, beta, S):
    """float64; q, k (T, H, dim), v (T, H, vdim), g broadcast to (T, H, dim), beta (T, H), S (H, dim, vdim) -> o, S"""
    out = []
    for t in range(q.shape[0]):
        u = v[t]
        if kind == "wkv":
            out.append(torch.einsum("hiv,hi->hv", S, q[t]) + beta[t][:, None] * v[t])
        S = g[t][:, :, None] * S
        if kind == "delta":
            u = beta[t][:, None] * (v[t] - torch.einsum("hiv,hi->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        if kind != "wkv":
            out.append(torch.einsum("hiv,hi->hv", S, q[t]))
    return torch.stack(out), S


def inputs(kind, seed, T, H, G, dim, vdim, decays):
    r = torch.Generator().manual_seed(seed)
    n = lambda *s: torch.randn(*s, generator=r)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k, v = unit(n(T, G, dim)) * dim ** -0.5, unit(n(T, G, dim)), n(T, H, vdim)
    if decays == "slow":
        z = 0.9 + 0.0999 * torch.rand(T, H, dim, generator=r)
    else:                       # from one token to the next almost everything goes, or nothing, or exactly everything
        z = torch.rand(T, H, dim, generator=r).pow(8)
        z[torch.rand(T, H, dim, generator=r) < 0.1] = 0.0
        z[torch.rand(T, H, dim, generator=r) < 0.1] = 1.0
    if kind == "heads":
        z = z[:, :, :1]
    if kind == "fixed":
        z = z[:1, :, :1].clamp(min=1e-3)
    beta = torch.rand(T, H, generator=r) if kind == "delta" else n(T, H)
    return q, k, v, z, beta


def launch(ops, kind, chunks, q, k, v, z, beta, o, state, seq, H, G, dim, vdim):
    dev = lambda x: x.reshape(x.shape[0], -1).contiguous().to(DEV)
    q, k, v, b = dev(q), dev(k), dev(v), dev(beta)
    g = z.reshape(-1).contiguous().to(DEV) if kind == "fixed" else dev(z)
    if chunks:
        ops.linear_chunks(kind, q, k, v, g, o, state, seq, H, G, dim, vdim, beta=b if kind in ("delta", "wkv") else None)
    elif kind == "delta":
        ops.delta_rule(q, k, v, g, b, o, state, seq, H, G, dim, vdim)
    elif kind == "fixed":
        ops.retention(q, k, v, g, o, state, seq, H, dim, vdim)
    else:
        ops.gated_scan(q, k, v, g, o, state, seq, H, G, dim, vdim, kind == "heads", bonus=b if kind == "wkv" else None)


@pytest.mark.parametrize("decays", ("slow", "any"))
@pytest.mark.parametrize("H,G,dim,vdim", [(2, 2, 128, 128), (4, 1, 128, 64), (6, 3, 64, 40), (3, 3, 4, 4), (2, 1, 68, 20),
                                          (1, 1, 100, 36)])
@pytest.mark.parametrize("kind", KINDS)
def test_chunks_follow_the_recurrence_across_portions(kind, H, G, dim, vdim, decays):
    """Portions of 1 to 200 tokens of three sequences side by side.  The bar on the error: sums of up to dim + 200 products of
    float32, 2^-24 each, of terms no larger than a few times the result; and no more than twice the scan's own error beside
    that of a single rounding."""
    from mashbox_b200 import ops
    if kind == "fixed":
        G = H                   # retention has a key and a query per head
    cuts = [[1, 31, 32, 33, 64, 100], [200, 1, 40, 20], [2, 63, 65, 96, 35]]
    T = 261
    seqs = [inputs(kind, 100 * i + dim, T, H, G, dim, vdim, decays) for i in range(3)]
    rep = lambda x: x.repeat_interleave(H // G, 1).double()
    want = []
    for q, k, v, z, beta in seqs:
        g = z.double().expand(T, H, dim)
        want.append(recurrence(kind, rep(q), rep(k), v.double(), g, beta.double(), torch.zeros(H, dim, vdim, dtype=torch.float64)))
    decay = seqs[0][3]
    if kind == "fixed":         # one decay per head for all sequences
        want = [recurrence(kind, rep(q), rep(k), v.double(), decay.double().expand(T, H, dim), beta.double(),
                           torch.zeros(H, dim, vdim, dtype=torch.float64)) for q, k, v, z, beta in seqs]
    pad, n, slots, errors = 8, H * dim * vdim, [3, 0, 4], {}
    for chunks in (False, True):
        state = torch.zeros(5, pad + n + 4, device=DEV)
        at, got = [0, 0, 0], [[], [], []]
        for step in range(max(len(c) for c in cuts)):
            live = [s for s in range(3) if step < len(cuts[s])]
            lens = [cuts[s][step] for s in live]
            cat = [torch.cat([seqs[s][j][at[s]:at[s] + m] for s, m in zip(live, lens)]) for j in (0, 1, 2)]
            z = decay if kind == "fixed" else torch.cat([seqs[s][3][at[s]:at[s] + m] for s, m in zip(live, lens)])
            beta = torch.cat([seqs[s][4][at[s]:at[s] + m] for s, m in zip(live, lens)])
            o = torch.full((sum(lens), H * vdim), float("nan"), device=DEV)
            seq = (i32(np.concatenate([[0], np.cumsum(lens)[:-1]])), i32(lens), i32([slots[s] for s in live]))
            launch(ops, kind, chunks, *cat, z, beta, o, state[:, pad:pad + n], seq, H, G, dim, vdim)
            lo = 0
            for s, m in zip(live, lens):
                got[s].append(o[lo:lo + m].double().cpu())
                lo, at[s] = lo + m, at[s] + m
        assert float(state[:, :pad].abs().max()) == 0.0 and float(state[:, pad + n:].abs().max()) == 0.0
        assert float(state[1].abs().max()) == 0.0 and float(state[2].abs().max()) == 0.0
        err = []
        for s in range(3):
            o = torch.cat(got[s]).reshape(at[s], H, vdim)
            w = want[s][0][:at[s]]
            err.append(float((o - w).norm() / w.norm()))
            assert float((o - w).abs().max()) <= 1e-5 * float(w.abs().max()), (kind, chunks, s)
            if at[s] == T:
                S = state[slots[s], pad:pad + n].double().cpu().view((H, vdim, dim) if kind == "fixed" else (H, dim, vdim))
                S = S.transpose(1, 2) if kind == "fixed" else S
                err.append(float((S - want[s][1]).norm() / want[s][1].norm()))
        errors[chunks] = max(err)
    print(kind, H, G, dim, vdim, decays, "scan %.2e chunks %.2e" % (errors[False], errors[True]))
    assert errors[True] <= 2 * errors[False] + 2.0 ** -24
    ops.check_error_word(ops.error_word(DEV))


@pytest.mark.parametrize("kind", KINDS)
def test_a_bad_value_does_not_reach_earlier_tokens(kind):
    """an infinity among one token's values leaves every token before it, and other columns and heads, as they were"""
    from mashbox_b200 import ops
    H, dim, vdim, T, bad = 2, 64, 32, 70, 45
    q, k, v, z, beta = inputs(kind, 5, T, H, H, dim, vdim, "slow")
    outs = []
    for x in (None, float("inf")):
        w = v.clone()
        if x is not None:
            w[bad, 1, 3] = x
        o = torch.empty(T, H * vdim, device=DEV)
        launch(ops, kind, True, q, k, w, z, beta, o, torch.zeros(1, H * dim * vdim, device=DEV), (i32([0]), i32([T]), i32([0])), H,
               H, dim, vdim)
        outs.append(o.view(T, H, vdim))
    same = torch.ones(T, H, vdim, dtype=torch.bool, device=DEV)
    same[bad:, 1, 3] = False
    assert torch.equal(outs[0][same], outs[1][same]) and not torch.isfinite(outs[1][bad, 1, 3])


@pytest.mark.parametrize("lens", [[33] * 40, [32] * 33 + [1] * 31, [31] * 10, [1000] + [1] * 63, [5, 31, 32, 63, 64, 65, 2]])
@pytest.mark.parametrize("kind", ("delta", "channels", "fixed"))
def test_many_sequences_side_by_side(kind, lens):
    """as many chunks as the scratch has room for, steps with long and short sequences, steps of short ones alone; sequences in
    slots in reverse order: against the token-by-token kernels (float32 sums in another order)"""
    from mashbox_b200 import ops
    H, dim, vdim, N = 2, 64, 32, sum(lens)
    q, k, v, z, beta = inputs(kind, len(lens), N, H, H, dim, vdim, "slow")
    start = torch.randn(len(lens), H * dim * vdim, generator=torch.Generator().manual_seed(1)) * 0.1
    seq = (i32(np.concatenate([[0], np.cumsum(lens)[:-1]])), i32(lens), i32(list(range(len(lens)))[::-1]))
    outs = []
    for chunks in (False, True):
        o, state = torch.full((N, H * vdim), float("nan"), device=DEV), start.to(DEV)
        launch(ops, kind, chunks, q, k, v, z, beta, o, state, seq, H, H, dim, vdim)
        outs.append((o.double(), state.double()))
    for a, b in zip(*outs):
        assert float((a - b).norm() / a.norm()) < 1e-6 and torch.isfinite(b).all()
    ops.check_error_word(ops.error_word(DEV))


@pytest.mark.parametrize("shortest", (32, 64, 160))
@pytest.mark.parametrize("kind", KINDS)
def test_sequences_below_the_shortest_are_the_scans(kind, shortest):
    """lengths on both sides of the line; those below it get the bits of the scan over them alone, and without `rest` are left
    as they are"""
    from mashbox_b200 import ops
    H, dim, vdim, lens = 2, 64, 32, [31, 32, 63, 64, 159, 160, 161, 1, 300]
    N = sum(lens)
    q, k, v, z, beta = inputs(kind, shortest, N, H, H, dim, vdim, "slow")
    dev = lambda x: x.reshape(x.shape[0], -1).contiguous().to(DEV)
    g = z.reshape(-1).contiguous().to(DEV) if kind == "fixed" else dev(z)
    start = torch.randn(len(lens), H * dim * vdim, generator=torch.Generator().manual_seed(1)) * 0.1
    seq = (i32(np.concatenate([[0], np.cumsum(lens)[:-1]])), i32(lens), i32(list(range(len(lens)))))
    outs = []
    for form in ("scan", "chunks", "no rest"):
        o, state = torch.full((N, H * vdim), 7.0, device=DEV), start.to(DEV)
        if form == "scan":
            launch(ops, kind, False, q, k, v, z, beta, o, state, seq, H, H, dim, vdim)
        else:
            ops.linear_chunks(kind, dev(q), dev(k), dev(v), g, o, state, seq, H, H, dim, vdim,
                              beta=dev(beta) if kind in ("delta", "wkv") else None, shortest=shortest,
                              rest=None if form == "chunks" else False)
        outs.append((o, state))
    (so, ss), (co, cs), (no, ns) = outs
    lo = 0
    for s, n in enumerate(lens):
        rows, short = slice(lo, lo + n), n < shortest
        for a, b in ((so[rows], co[rows]), (ss[s], cs[s])):
            assert float((a - b).norm() / a.norm()) < 1e-6         # float32 sums in another order
        assert bool((no[rows] == 7.0).all()) == short and torch.equal(ns[s].cpu(), start[s]) == short
        if not short:
            assert torch.equal(no[rows], co[rows]) and torch.equal(ns[s], cs[s])
        lo += n
    ops.check_error_word(ops.error_word(DEV))


@pytest.mark.parametrize("kind", ("channels", "heads", "wkv"))
def test_decoded_tokens_beside_a_prompt_run_as_without_it(kind):
    """the scan of the short sequences lays the state out as it does in a step of theirs alone: the same bits"""
    from mashbox_b200 import ops
    H, dim, vdim, lens = 2, 128, 64, [200, 1, 2, 1]
    N, n = sum(lens), H * dim * vdim
    q, k, v, z, beta = inputs(kind, 9, N, H, H, dim, vdim, "slow")
    start = (torch.randn(4, n, generator=torch.Generator().manual_seed(1)) * 0.1).to(DEV)
    both, alone = start.clone(), start.clone()
    o, p = torch.empty(N, H * vdim, device=DEV), torch.empty(4, H * vdim, device=DEV)
    launch(ops, kind, True, q, k, v, z, beta, o, both, (i32([0, 200, 201, 203]), i32(lens), i32([0, 1, 2, 3])), H, H, dim, vdim)
    launch(ops, kind, False, *(x[200:] for x in (q, k, v, z, beta)), p, alone, (i32([0, 1, 3]), i32(lens[1:]), i32([1, 2, 3])), H, H,
           dim, vdim)
    assert torch.equal(o[200:], p) and torch.equal(both[1:], alone[1:])


def test_sizes_that_the_chunk_form_does_not_take():
    from mashbox_b200 import ops
    assert ops.linear_chunks_supports(2000, 3, 128, 64, "delta") and not ops.linear_chunks_supports(160, 80, 128, 64, "delta")
    for dim, vdim in ((132, 64), (130, 64), (62, 64), (64, 30)):
        assert not ops.linear_chunks_supports(2000, 3, dim, vdim, "delta")
