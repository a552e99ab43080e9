"""-m gpu: the float32 product on the tensor cores (gemm_f32_tc5.cu): every tile and cut of K gives the same bits, and they lie
no further from 64 bits than one chain of fused multiply-adds does."""
import pytest
import torch

from tests import gpu_harness as G

pytestmark = pytest.mark.gpu
TILES = [(tile, cluster) for tile in (16, 32, 64, 128, 256) for cluster in (1, 4)]


def ops():
    import mashbox_b200.ops as K
    return K


def chain(a, w):
    """the product of the FMA units, whatever the matrix"""
    K = ops()
    N, Kd = a.shape
    out = torch.empty(N, w.shape[0], device=G.DEV)
    f = K._fn("gemm_f32", "mb_gemm_f32", [K.c_void_p] * 3 + [K.c_int] * 4 + [K.c_void_p])
    K._check(f(K._p(a), K._p(w), K._p(out), N, w.shape[0], Kd, w.shape[0], K._stream()), "gemm_f32")
    return out


def operands(N, M, Kd, kind="normal", seed=0, off=0):
    g = torch.Generator().manual_seed(seed + N + M + Kd)
    make = {"normal": lambda *s: torch.randn(*s, generator=g), "positive": lambda *s: torch.rand(*s, generator=g),
            "wide": lambda *s: torch.randn(*s, generator=g) * torch.exp(4 * torch.randn(*s, generator=g)),
            "tiny": lambda *s: 1e-17 * torch.randn(*s, generator=g)}[kind]
    return make(N * Kd + off).to(G.DEV)[off:].view(N, Kd), make(M, Kd).to(G.DEV)


# rows on the edges of every tile; columns on the edges of 128; K with quarters of one block, empty quarters (5 blocks: two each),
# a block that is not full, and no multiple of 8; rows of a off a 16-byte boundary
@pytest.mark.parametrize("N,M,Kd,off", [(1, 64, 128, 0), (16, 128, 160, 0), (17, 129, 132, 1), (33, 200, 1028, 0), (65, 127, 516, 0),
                                        (129, 256, 2048, 0), (257, 300, 640, 3), (300, 65, 8192, 0)])
def test_every_tile_gives_the_same_bits(N, M, Kd, off):
    K = ops()
    a, w = operands(N, M, Kd, off=off)
    assert K.f32_split_supports(w)
    first = K.linear(a, w)
    exact = a.double() @ w.double().T
    # dropped parts 2^-21 of a product; a block of 32 k: twelve sums cut off at 2^-23 of its products; K / 32 + 4 rounded sums
    bound = (a.abs().double() @ w.abs().double().T) * (8 + 24 + Kd / 32 + 4) * 2.0 ** -24
    assert bool(((first.double() - exact).abs() <= bound).all())
    for tile, cluster in TILES:
        out = torch.full((N, M + 5), 7.0, device=G.DEV)
        K.linear_f32_split(a, w, out[:, :M], tile=tile, cluster=cluster)
        assert torch.equal(out[:, :M], first), (tile, cluster)
        assert bool((out[:, M:] == 7.0).all())
    for n in sorted({0, N // 2, N - 1}):
        assert torch.equal(K.linear(a[n:n + 1], w)[0], first[n])
    K.check_error_word(K.error_word(a.device))


@pytest.mark.parametrize("kind", ["normal", "positive", "wide", "tiny"])
@pytest.mark.parametrize("Kd", [128, 512, 2048, 8192])
def test_no_further_from_64_bits_than_a_chain(kind, Kd):
    K = ops()
    a, w = operands(64, 512, Kd, kind)
    exact = a.double() @ w.double().T
    err = lambda x: float((x.double() - exact).norm() / exact.norm())
    # where single products decide the sums ("wide"), a chain is exact but for its last bit: here the last bit may be cut off
    assert err(K.linear(a, w)) <= max(err(chain(a, w)), 2.0 ** -23)


def test_infinities_and_nan_are_those_of_the_chain():
    K = ops()
    a, w = operands(40, 130, 256)
    a[3, 7], a[5, 9], a[9, 20], a[11, 4] = float("inf"), float("nan"), float("-inf"), 3.4e38
    w[100, 3], w[60, 7], w[61, 9] = float("-inf"), 0.0, 0.0
    a[12] = 0.0
    want = chain(a, w)
    for tile, cluster in TILES:
        got = K.linear_f32_split(a, w, torch.empty(40, 130, device=G.DEV), tile=tile, cluster=cluster)
        odd = ~torch.isfinite(want)
        assert bool(odd.any()) and torch.equal(torch.isfinite(got), ~odd)
        assert torch.equal(torch.nan_to_num(got[odd], nan=1.0), torch.nan_to_num(want[odd], nan=1.0))


def test_rows_in_slabs(monkeypatch):
    K = ops()
    a, w = operands(700, 100, 256)
    whole = K.linear(a, w)
    monkeypatch.setattr(K, "F32_SPLIT_PLANE", 1)
    assert torch.equal(K.linear(a, w), whole)
