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
