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
