"""The two-SM GEMM (csrc/kernels/gemm_pair.cu) against f32 products: edges of its 256-row tiles, of the tile widths that its plan picks, of
K blocks and of the K split inside a cluster."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(M, N, K, seed=0, ldx=0, ldw=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.empty(M, ldx or K, dtype=torch.bfloat16, device="cuda").normal_(generator=g)[:, :K]
    w = torch.empty(N, ldw or K, dtype=torch.bfloat16, device="cuda").normal_(0, 0.05, generator=g)[:, :K]
    return x, w


def _close(got, want, K):
    # bf16 results: half a unit in the last place (2^-9 of the value).  f32 results: the tensor core cuts off what an addition of 16 products
    # leaves below the accumulator's last place, half a unit (2^-24) on average and always downwards, so K / 16 additions lose up to K / 16 * 2^-24
    tol = 2.0 ** -8 if got.dtype == torch.bfloat16 else (K / 16 + 8) * 2.0 ** -24
    assert not torch.isnan(got).any()
    err = (got.double() - want).norm() / want.norm()
    assert err < tol, err
    assert (got.double() - want).abs().max() < 8 * tol * want.abs().max()


SHAPES = [(129, 64, 64), (217, 3840, 4096), (217, 8192, 3840), (256, 32, 8), (257, 40, 72), (300, 8, 2048), (384, 2112, 7168), (511, 1000, 520),
          (513, 257 * 8, 192), (701, 3840, 1024), (1024, 3840, 8192), (2050, 4104, 264), (4096, 16, 3840), (4096, 48, 15360)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("f32", [False, True])
def test_pair_matches_f32(M, N, K, f32):
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K)
    want = x.double() @ w.double().t()
    got = K_.linear_f32(x, w) if f32 else K_.linear(x, w)
    _close(got, want, K)
    assert torch.equal(got, K_.linear_f32(x, w) if f32 else K_.linear(x, w))          # no sum whose order depends on timing
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,N,K", [(130, 48, 128), (217, 15360, 256), (400, 1040, 3840), (1000, 120, 4096)])
@pytest.mark.parametrize("act", ["geglu", "swiglu"])
def test_pair_glu(M, N, K, act):
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, 2 * N, K)
    gu = x.double() @ w.double().t()
    gate = torch.nn.functional.gelu(gu[:, :N], approximate="tanh") if act == "geglu" else torch.nn.functional.silu(gu[:, :N])
    got = K_.linear_glu(x, w, act)
    _close(got, gate * gu[:, N:], K)
    out = torch.zeros(M, N + 24, dtype=torch.bfloat16, device="cuda")                 # a row view: nothing beside it is touched
    K_.linear_glu(x, w, act, out=out[:, 8:8 + N])
    assert torch.equal(out[:, 8:8 + N], got) and not out[:, :8].any() and not out[:, 8 + N:].any()
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,N,K", [(200, 500, 640), (1030, 264, 4096)])
def test_pair_bias_views_and_activation(M, N, K):
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K, ldx=K + 16, ldw=K + 8)
    bias = torch.randn(N, device="cuda")
    want = x.double() @ w.double().t()
    _close(K_.linear(x, w, bias), want + bias.double(), K)
    _close(K_.linear_f32(x, w, alpha=0.25), 0.25 * want, K)
    cols = N - 13
    acted = want.clone()
    acted[:, :cols] = torch.nn.functional.silu(want[:, :cols])
    _close(K_.linear_act(x, w, "silu", cols), acted, K)
    out = torch.zeros(M, N + 3, dtype=torch.bfloat16, device="cuda")                  # rows that no 16-byte store can take
    K_.gemm(x, w, out=out[:, 1:1 + N])
    _close(out[:, 1:1 + N], want, K)
    assert not out[:, 0].any() and not out[:, 1 + N:].any()
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,N,K", [(3, 128, 7168), (33, 384, 4096), (100, 96, 15360), (217, 3840, 4096), (300, 128, 7168), (16, 1536, 15360)])
def test_f32_sums_are_as_exact_as_sixteen_slices(M, N, K):
    """Router logits and partial sums: an addition in the tensor core loses half a unit (2^-24 of the sum so far) on average, always downwards.  A sum
    that grows to its value over K / 16 / 16 additions therefore loses half of that many units at most; the f32 additions of the slices lose less than 8."""
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K, seed=3)
    want = x.double() @ w.double().t()
    err = (K_.linear_f32(x, w).double() - want).norm() / want.norm()
    assert err < (K / 16 / 16 / 2 + 8) * 2.0 ** -24, err


@pytest.mark.parametrize("M", [1, 3, 33, 100, 128])
@pytest.mark.parametrize("N,K", [(1100, 4096), (40, 2568), (2112, 7168), (129, 15360), (384, 3840)])
def test_few_rows(M, N, K):
    """Products of at most 128 rows whose K is cut: the weights are the row operand."""
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K, seed=M)
    want = x.double() @ w.double().t()
    for f in (K_.linear, K_.linear_f32):
        got = f(x, w)
        _close(got, want, K)
        assert torch.equal(got, f(x, w))
    bias = torch.randn(N, device="cuda")
    _close(K_.linear(x, w, bias), want + bias.double(), K)
    cols = N - 13
    acted = want.clone()
    acted[:, :cols] = torch.nn.functional.silu(want[:, :cols])
    _close(K_.linear_act(x, w, "silu", cols), acted, K)
    assert K_.last_status() == 0


@pytest.mark.parametrize("bn", [32, 64, 96, 224, 256])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("swap", [False, True])
def test_every_width_and_split(bn, splits, swap):
    """Widths, splits (also a last part of K of one block, and a last block that is cut) and both operand orders, at sizes that leave partial tiles."""
    from mary_b200.ops import cuda as K_
    for M, N, K in ((70, 300, 64 * (5 * (splits - 1) + 1)), (300, 264, 64 * 9 * splits - 24)):
        x, w = _problem(M, N, K, seed=bn + splits)
        want = x.double() @ w.double().t()
        for f32 in (False, True):
            _close(K_.gemm_pair(x, w, bn, splits, swap=swap, f32=f32), want, K)
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,N,K", [(257, 128, 15360), (300, 40, 7168), (129, 33, 2112), (70, 3840, 256), (2050, 1032, 136)])
def test_f32_rows(M, N, K):
    """f32 results: clusters of 16, stores of 16 columns, rows that end inside a box or that no 16-byte store can take, a bias."""
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K, seed=7)
    want = x.double() @ w.double().t()
    for pad in (0, 4, 3):
        out = torch.zeros(M, N + pad, device="cuda")
        K_.gemm(x, w, out=out[:, :N], epi="f32")
        _close(out[:, :N], want, K)
        assert not out[:, N:].any()
    bias = torch.randn(N, device="cuda")
    _close(K_.gemm(x, w, bias=bias, epi="f32"), want + bias.double(), K)
    assert K_.last_status() == 0


@pytest.mark.parametrize("bn", [64, 96, 224, 256])
@pytest.mark.parametrize("splits", [1, 2, 4])
def test_every_width_and_split_of_glu(bn, splits):
    from mary_b200.ops import cuda as K_
    if bn % (16 * splits):
        pytest.skip("columns of a CTA")
    x, w = _problem(300, 2 * 264, 2112, seed=bn)
    gu = x.double() @ w.double().t()
    _close(K_.gemm_pair(x, w, bn, splits, glu="swiglu"), torch.nn.functional.silu(gu[:, :264]) * gu[:, 264:], 2112)
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,N,K", [(257, 64, 8), (300, 1000, 1024), (384, 2112, 2048), (701, 512, 512), (8192, 128, 3072), (1024, 1024, 3080), (257, 96, 1024)])
def test_short_products_of_many_rows(M, N, K):
    """Around the line between the one-SM and the two-SM kernel (tiles of one wave, K blocks against tiles)."""
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, N, K, seed=5)
    want = x.double() @ w.double().t()
    for f in (K_.linear, K_.linear_f32):
        _close(f(x, w), want, K)
        assert torch.equal(f(x, w), f(x, w))
    assert K_.last_status() == 0


@pytest.mark.parametrize("M,F,K,two", [(257, 8192, 1024, True), (2048, 512, 1536, True), (2048, 512, 1544, False), (2040, 512, 1024, False), (256, 8192, 1024, False)])
@pytest.mark.parametrize("act", ["geglu", "swiglu", "situ"])
def test_short_glu_products_take_two_launches(M, F, K, two, act):
    from mary_b200.ops import cuda as K_
    x, w = _problem(M, 2 * F, K, seed=11)
    got, parts = K_.linear_glu(x, w, act), K_.glu(K_.gemm(x, w), act)
    assert torch.equal(got, parts) == two                                              # fused, gate and up are not rounded to bf16 in between
    assert (got.double() - parts.double()).norm() / parts.double().norm() < 2.0 ** -7   # two more roundings of 2^-9
    out = torch.zeros(M, F + 24, dtype=torch.bfloat16, device="cuda")
    K_.linear_glu(x, w, act, out=out[:, 8:8 + F])
    assert torch.equal(out[:, 8:8 + F], got) and not out[:, :8].any() and not out[:, 8 + F:].any()
    out.zero_()
    K_.linear_glu(x, w, act, out=out[:, 1:1 + F])                                      # rows that no 16-byte store can take
    assert (out[:, 1:1 + F].double() - got.double()).norm() / got.double().norm() < 2.0 ** -7 and not out[:, 0].any() and not out[:, 1 + F:].any()
    assert K_.last_status() == 0
