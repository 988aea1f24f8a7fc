"""The soft-capped cross-entropy kernels at the edges of the cluster form: rows of one to eight CTAs, parts that end early, caps beyond the fixed
reference, arguments on both sides of the series, labels outside the vocabulary."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [8, 2048, 4088, 4096, 32768, 32776, 65544, 131080, 262144, 400008, 600000])
@pytest.mark.parametrize("cap,std", [(30.0, 1.2), (30.0, 15.0), (50.0, 30.0), (0.0, 8.0)])
def test_softcap_cross_entropy(V, cap, std):
    from mary_b200.ops import train_ops as T
    from mary_b200.ops.cuda import _p, _stream, check, last_status, lib
    rows, scale = 5, 0.125
    g = torch.Generator(device="cuda").manual_seed(V)
    lg = torch.empty(rows, V + 8, dtype=torch.bfloat16, device="cuda").normal_(0, std, generator=g)
    labels = torch.tensor([0, V - 1, V // 2, -1, V], device="cuda")
    z = lg[:, :V].double()
    t = torch.tanh(z / cap) if cap else z
    z = cap * t if cap else z
    want_loss = torch.logsumexp(z, 1) - z.gather(1, labels.clamp(0, V - 1)[:, None])[:, 0]
    p = torch.softmax(z, 1)
    hot = torch.zeros_like(p).scatter_(1, labels.clamp(0, V - 1)[:, None], 1.0)
    want = scale * (p - hot) * (1 - t * t if cap else 1.0)
    want_loss[3:], want[3:] = 0.0, 0.0
    loss = torch.empty(rows, device="cuda")
    rest = lg[:, V:].clone()
    check(lib().mary_softcap_ce(_p(lg), lg.stride(0), _p(labels), rows, V, cap, scale, _p(loss), _stream()), "softcap_ce")
    # f32 sums of V exponentials whose arguments (up to 2 cap or 10 std, in units of ln 2) carry a rounding of 2^-24 each
    assert (loss.double() - want_loss).abs().max() < 2e-5 * max(1.0, float(want_loss.abs().max()))
    # gradients: rounded to bf16; an exponential is exact to 2^-21 at these arguments
    assert ((lg[:, :V].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-7 * scale).all()
    assert torch.equal(lg[:, V:], rest) and last_status() == 0


@pytest.mark.parametrize("V", [8184, 8192, 16384, 51200, 51208, 409600, 409608, 524288])
@pytest.mark.parametrize("rows", [1, 19, 40, 300])
def test_softcap_cross_entropy_by_rows(V, rows):
    """The edges of the rule that picks the form and the cluster: values per CTA, rows for few and for all SMs."""
    from mary_b200.ops import train_ops as T                                      # noqa: F401  (declares the launcher)
    from mary_b200.ops.cuda import _p, _stream, check, last_status, lib
    if rows * V > 2.5e7:
        rows = max(1, int(2.5e7 // V))
    g = torch.Generator(device="cuda").manual_seed(V + rows)
    lg = torch.empty(rows, V, dtype=torch.bfloat16, device="cuda").normal_(0, 3.0, generator=g)
    labels = torch.randint(0, V, (rows,), device="cuda", generator=g)
    t = torch.tanh(lg.double() / 30.0)
    z = 30.0 * t
    want_loss = torch.logsumexp(z, 1) - z.gather(1, labels[:, None])[:, 0]
    want = (torch.softmax(z, 1) - torch.zeros_like(z).scatter_(1, labels[:, None], 1.0)) * (1.0 - t * t)
    loss = torch.empty(rows, device="cuda")
    check(lib().mary_softcap_ce(_p(lg), V, _p(labels), rows, V, 30.0, 1.0, _p(loss), _stream()), "softcap_ce")
    assert (loss.double() - want_loss).abs().max() < 2e-5 * want_loss.abs().max()
    assert ((lg.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-7).all()
    assert last_status() == 0


@pytest.mark.parametrize("V", [4096, 32768, 151936])
@pytest.mark.parametrize("cap", [0.0, 30.0, 50.0])
@pytest.mark.parametrize("at,n", [(0, 8), (8, 8), (3000, 1), (0, 4096)])
def test_a_nan_logit_reaches_the_loss(V, cap, at, n):
    """Whole vectors of NaN, also the first that a thread reads; the other rows keep their loss, and an infinite logit is at the cap."""
    from mary_b200.ops import train_ops as T                                      # noqa: F401
    from mary_b200.ops.cuda import _p, _stream, check, lib
    lg = torch.empty(3, V, dtype=torch.bfloat16, device="cuda").normal_(0, 2.0, generator=torch.Generator(device="cuda").manual_seed(1))
    if cap:
        lg[2, 5], lg[2, 9] = float("inf"), float("-inf")
    labels = torch.tensor([7, 11, 13], device="cuda")
    z = lg.double()
    z = cap * torch.tanh(z / cap) if cap else z
    want = torch.logsumexp(z, 1) - z.gather(1, labels[:, None])[:, 0]
    lg[1, at:at + n] = float("nan")
    loss = torch.empty(3, device="cuda")
    check(lib().mary_softcap_ce(_p(lg), V, _p(labels), 3, V, cap, 1.0, _p(loss), _stream()), "softcap_ce")
    assert torch.isnan(loss[1]) and (loss.double() - want)[[0, 2]].abs().max() < 2e-5 * want.abs().max()
