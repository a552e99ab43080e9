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


def worst(x, exact):
    """the largest error of an element over that element, where the result is a normal number"""
    at = exact.abs() >= 2.0 ** -125
    return float(((x.double() - exact).abs()[at] / exact.abs()[at]).max())


def of_bits(n, g):
    """values of [1, 2) with all their bits drawn"""
    return (0x3f800000 + torch.randint(0, 1 << 23, (n,), generator=g, dtype=torch.int32)).view(torch.float32).to(G.DEV)


# Where few products decide a result: rows that are one value throughout (every product of a result has the same parts left over;
# 0x3f80ff80 is the worst of all mantissas for parts that are left out), rows of one value and zeros, rows of one value among others
# that are 2^-34 of it together.  The chain rounds a product once, 2^-24; the bar beside its worst element is that and the parts of 2^-7, which an
# accumulator may cut off at 2^-23 of them.
@pytest.mark.parametrize("kind", ["constant", "the worst constant", "one-hot", "dominant"])
@pytest.mark.parametrize("Kd", [128, 512, 2048])
@pytest.mark.parametrize("tile,cluster", [(0, 0), (64, 1), (64, 4), (256, 1)])
def test_few_products_are_as_exact_as_in_a_chain(kind, Kd, tile, cluster):
    K = ops()
    N, M = 48, 192
    g = torch.Generator().manual_seed(Kd)
    if kind == "constant":
        a, w = of_bits(N, g)[:, None].repeat(1, Kd), of_bits(M, g)[:, None].repeat(1, Kd)
    elif kind == "the worst constant":
        x = torch.tensor([0x3f80ff80], dtype=torch.int32).view(torch.float32).to(G.DEV)
        a, w = x.repeat(N, Kd), x.repeat(M, Kd)
    else:
        w = of_bits(M * Kd, g).view(M, Kd)
        a = torch.zeros(N, Kd, device=G.DEV) if kind == "one-hot" else of_bits(N * Kd, g).view(N, Kd) * 2.0 ** -34 / Kd
        a[torch.arange(N), torch.randint(0, Kd, (N,), generator=g)] = of_bits(N, g)
    exact = a.double() @ w.double().T
    got = K.linear_f32_split(a, w, torch.empty(N, M, device=G.DEV), tile=tile, cluster=cluster)
    assert worst(got, exact) <= max(worst(chain(a, w), exact), 2.0 ** -24) * (1 + 2.0 ** -6)


@pytest.mark.parametrize("kind", ["normal", "positive", "wide", "tiny"])
@pytest.mark.parametrize("Kd", [128, 512, 2048, 8192, 16384])
def test_the_worst_element_is_no_further_off_than_a_chains(kind, Kd):
    """measured by the sum of the products' magnitudes; and sums that many products make, by themselves"""
    K = ops()
    a, w = operands(64, 512, Kd, kind, seed=5)
    exact, size = a.double() @ w.double().T, a.abs().double() @ w.abs().double().T
    got, old = K.linear(a, w), chain(a, w)
    assert float(((got - exact).abs() / size).max()) <= float(((old - exact).abs() / size).max())
    if kind != "wide":
        assert float((got - exact).norm()) <= max(float((old - exact).norm()), 2.0 ** -24 * float(exact.norm()))


@pytest.mark.parametrize("p", [-96, -109, -112, -118, -124, -130, -140, -149])
@pytest.mark.parametrize("side", ["a", "w", "both"])
def test_tiny_operands_keep_all_their_bits(p, side):
    """operands down to the smallest subnormal, beside ones that bring the products back among the normal numbers"""
    K = ops()
    N, M, Kd = 24, 70, 256
    g = torch.Generator().manual_seed(-p)
    tiny = lambda n: torch.ldexp(of_bits(n, g).double(), torch.tensor(p, device=G.DEV)).float()
    big = lambda n: of_bits(n, g) * 2.0 ** min(-p, 100)
    a = (tiny(N * Kd) if side != "w" else big(N * Kd)).view(N, Kd)
    w = (tiny(M * Kd) if side != "a" else big(M * Kd)).view(M, Kd)
    a[:, 1::2] *= -1.0
    exact = a.double() @ w.double().T
    # the last bit of a result that is itself subnormal; a chain may lose it at every k, the quarters of K here at their ends
    err = lambda x: float(((x.double() - exact).abs() - 4 * 2.0 ** -149).clamp(min=0).norm() / exact.norm().clamp(min=2.0 ** -149))
    assert err(K.linear_f32_split(a, w, torch.empty(N, M, device=G.DEV))) <= max(err(chain(a, w)), 2.0 ** -24)


@pytest.mark.parametrize("cluster", [1, 4])
def test_it_is_float32_arithmetic(cluster):
    """1 + 2^-p is a float32 number down to p = 23: as a sum of two products, and as one operand"""
    K = ops()
    w = torch.zeros(64, 128, device=G.DEV)
    w[:, 0] = w[:, 70] = 1.0
    a = torch.zeros(48, 128, device=G.DEV)
    for p in range(24):
        a[p, 0], a[p, 70] = 1.0, 2.0 ** -p
        a[24 + p, 0] = 1.0 + 2.0 ** -p
    out = K.linear_f32_split(a, w, torch.empty(48, 64, device=G.DEV), cluster=cluster)
    assert torch.equal(out, (a[:, :1] + a[:, 70:71]).expand(48, 64))


@pytest.mark.parametrize("N,M,Kd,off", [(130, 130, 260, 1), (70, 64, 132, 0), (300, 200, 2052, 3)])
def test_many_results_that_are_not_finite(N, M, Kd, off):
    """more columns of a tile than go through a chain at a time, whole rows and single results, finite ones between them"""
    K = ops()
    a, w = operands(N, M, Kd, off=off)
    a[5:70:2, 3] = float("nan")
    a[1:60:7, 0] = float("inf")
    a[:, 9] *= 1e30
    w[3, 9], w[10, 9], w[40, 0] = 3e38, 1e20, 0.0
    want = chain(a, w)
    odd = ~torch.isfinite(want)
    assert bool(odd.any()) and not bool(odd.all())
    first = None
    for tile, cluster in TILES:
        got = K.linear_f32_split(a, w, torch.empty(N, M, device=G.DEV), tile=tile, cluster=cluster)
        assert torch.equal(torch.nan_to_num(got[odd], nan=1.0), torch.nan_to_num(want[odd], nan=1.0))
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        first = got if first is None else first
        assert torch.equal(torch.nan_to_num(got, nan=1.0), torch.nan_to_num(first, nan=1.0))
    K.check_error_word(K.error_word(a.device))


def test_a_prompt_of_nan_costs_a_few_products():
    """509 x 16384 x 2048 of finite numbers takes 0.25 ms; with a thread for every chain NaN took 70"""
    K = ops()
    a, w = operands(509, 16384, 2048)
    out = torch.empty(509, 16384, device=G.DEV)

    def took(a):
        K.linear(a, w, out=out)
        best = float("inf")
        for _ in range(3):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            K.linear(a, w, out=out)
            end.record()
            end.synchronize()
            best = min(best, begin.elapsed_time(end))
        return best
    plain = took(a)
    assert took(torch.full_like(a, float("nan"))) < 40 * plain and bool(torch.isnan(out).all())


@pytest.mark.parametrize("N,M,Kd,split", [(33, 512, 128, False), (5, 2048, 192, False), (300, 161, 252, False), (7, 160, 128, True),
                                          (20, 161, 256, True), (9, 63, 512, False), (9, 64, 258, False)])
def test_short_matrices_stay_on_the_fma_units(N, M, Kd, split):
    """where the tensor cores' two launches cost more (ops.f32_split_supports): the same bits as the FMA units' product"""
    K = ops()
    a, w = operands(N, M, Kd)
    assert K.f32_split_supports(w) == split
    want = K.linear_f32_split(a, w, torch.empty(N, M, device=G.DEV)) if split else chain(a, w)
    assert torch.equal(K.linear(a, w), want)
