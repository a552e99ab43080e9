"""-m gpu: the tiles of the float32 product and the tiled form of the plain attention.  Both promise more than closeness:
an output is the same chain of float32 operations in every tile and in both forms, so the bars are equalities."""
import pytest
import torch

from tests import gpu_harness as G

pytestmark = pytest.mark.gpu


def ops():
    import mashbox_b200.ops as K
    return K


# one size for every tile the product chooses by size, on the edges of its rows, columns and stages of 16; K no multiple of 4
# and an operand off a 16-byte boundary (the second below) take single loads
@pytest.mark.parametrize("N,M,Kd,off", [(130, 16384, 48, 0), (129, 37890, 36, 0), (64, 9473, 20, 0), (33, 9472, 18, 0),
                                        (32, 9472, 64, 1), (17, 9409, 16, 0), (16, 65, 4, 0), (1, 1000, 1030, 0), (5, 3, 1, 0),
                                        (200, 130, 100, 0)])
def test_gemm_f32_tiles_give_the_bits_of_a_row_alone(N, M, Kd, off):
    K = ops()
    g = torch.Generator().manual_seed(N + M)
    a = torch.randn(N * Kd + off, generator=g).to(G.DEV)[off:].view(N, Kd)
    w = torch.randn(M * Kd + off, generator=g).to(G.DEV)[off:].view(M, Kd)
    out = torch.full((N, M + 5), 7.0, device=G.DEV)[:, :M]
    K.linear(a, w, out=out)
    exact = a.double() @ w.double().T
    # Kd roundings of partial sums of at most sum |a||w|, each 2^-24
    bound = (a.abs().double() @ w.abs().double().T) * Kd * 2.0 ** -24 + 1e-30
    assert bool(((out.double() - exact).abs() <= bound).all())
    for n in sorted({0, N // 2, N - 1}):
        assert torch.equal(K.linear(a[n:n + 1], w)[0], out[n])
    assert bool((out._base[:, M:] == 7.0).all())


@pytest.mark.parametrize("N", [17, 32, 33, 64, 65, 128, 129, 192, 193])
def test_gemm_f32_many_columns(N):
    """more than 592 tiles of 64 columns: the rows decide the tile"""
    test_gemm_f32_tiles_give_the_bits_of_a_row_alone(N, 37889, 20, 0)


def test_gemm_f32_takes_more_rows_than_the_smallest_tile_could():
    K = ops()
    N, M, Kd = 16 * 65535 + 17, 5, 3
    a, w = torch.randn(N, Kd, device=G.DEV), torch.randn(M, Kd, device=G.DEV)
    out = K.linear(a, w)
    bound = (a.abs().double() @ w.abs().double().T) * Kd * 2.0 ** -24 + 1e-30
    assert bool(((out.double() - a.double() @ w.double().T).abs() <= bound).all())


# (lengths, tokens of the step): runs that fill tiles, straddle them, are too short for the tiled form, stand on their edges
@pytest.mark.parametrize("H,KV,HD,HDV,page,lengths,q_lens", [
    (32, 8, 64, 64, 16, [100, 40, 33], [100, 1, 33]),
    (8, 1, 128, 128, 8, [70, 1, 1, 260], [67, 1, 1, 3]),
    (7, 7, 20, 12, 4, [65, 64, 63], [65, 64, 63]),
    (6, 2, 40, 40, 16, [300, 90, 4, 31], [44, 85, 4, 31]),
    (16, 2, 256, 256, 16, [50], [50])])
@pytest.mark.parametrize("extras", [False, True])
def test_tiled_attention_gives_the_bits_of_the_plain_form(H, KV, HD, HDV, page, lengths, q_lens, extras):
    K = ops()
    seqs = G.PagedSequences(lengths, q_lens, H, KV, HD, page, torch.float32, seed=HD).round().build()
    vpool = seqs.vpool[..., :HDV].contiguous()
    sinks = torch.randn(H, device=G.DEV) if extras else None
    gate = torch.randn(seqs.N, H, device=G.DEV) if extras else None
    cap = 5.0 if extras else None
    err = K.new_error_word(G.DEV)
    scale = HD ** -0.5

    def run(lo, hi):
        out = torch.full((hi - lo, H * HDV), 7.0, device=G.DEV)
        K.attention_general(seqs.q_dev[lo:hi], H * HD, out, seqs.positions[lo:hi], seqs.tok_row[lo:hi], seqs.table, seqs.kpool,
                            vpool, H, KV, HD, HDV, page, seqs.num_pages, None, scale, err, cap, sinks,
                            gate[lo:hi] if extras else None)
        return out
    whole = run(0, seqs.N)
    alone = torch.cat([run(n, n + 1) for n in range(seqs.N)])            # one token a call is the plain form
    K.check_error_word(err)
    assert torch.isfinite(whole).all() and torch.equal(whole, alone)
    if not extras and HD == HDV:
        want = seqs.reference(scale)
        assert float((whole.double().cpu() - want).abs().max()) < 1e-5 * float(want.abs().max())
    # a page that is missing is reported by the tiled form too, and its keys are left out as the plain form leaves them out
    bad = seqs.table.clone()
    bad[seqs.rows[0], 0] = -1
    table, seqs.table = seqs.table, bad
    whole = run(0, seqs.N)
    with pytest.raises(Exception, match="block table does not hold"):
        K.check_error_word(err)
    assert torch.equal(whole, torch.cat([run(n, n + 1) for n in range(seqs.N)]))
    seqs.table = table
    err.zero_()


@pytest.mark.parametrize("order", ["gaps", "reversed", "shuffled", "whole"])
def test_tokens_in_any_order_are_all_computed(order):
    """The tiled form takes runs of neighbours that are one sequence's tokens in order; every other token is the plain form's --
    also one whose neighbours beyond another sequence's token would continue it ("gaps": three tokens, one of another sequence,
    three tokens, each at the place its position asks for)."""
    K = ops()
    H, KV, HD, page = 8, 2, 64, 16
    seqs = G.PagedSequences([120, 60], [120, 60], H, KV, HD, page, torch.float32, seed=3).round().build()
    places = list(range(seqs.N))
    if order == "gaps":
        places = [120 + j // 4 if j % 4 == 3 else j for j in range(120)]
    elif order == "reversed":
        places = places[::-1]
    elif order == "shuffled":
        places = torch.randperm(seqs.N, generator=torch.Generator().manual_seed(1)).tolist()
    err, at = K.new_error_word(G.DEV), torch.tensor(places, device=G.DEV)

    def run(at):
        out = torch.full((len(at), H * HD), 7.0, device=G.DEV)
        K.attention_simple(seqs.q_dev[at].contiguous(), H * HD, out, seqs.positions[at].contiguous(), seqs.tok_row[at].contiguous(),
                           seqs.table, seqs.kpool, seqs.vpool, H, KV, HD, page, seqs.num_pages, None, HD ** -0.5, err)
        return out
    alone = torch.cat([run(at[n:n + 1]) for n in range(len(places))])
    assert torch.equal(run(at), alone)
    K.check_error_word(err)
