"""The router against 64-bit scores, on both sides of the line between one CTA and one warp per token (256 tokens, 256 experts, groups): every number of
experts per lane, biases, renormalisation, equal logits, counts and the flag of a non-finite logit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(lg, k, mode, bias, scale, renorm):
    z = lg.double()
    s = torch.softmax(z, -1) if mode == "softmax" else torch.sigmoid(z)
    sel = s + (bias.double() if bias is not None else 0.0)
    idx = torch.sort(sel, dim=-1, descending=True, stable=True).indices[:, :k]
    w = s.gather(1, idx)
    return sel, idx, (w / w.sum(-1, keepdim=True) if renorm else w) * scale


@pytest.mark.parametrize("T", [255, 256, 1000])
@pytest.mark.parametrize("E,k", [(8, 2), (32, 1), (33, 8), (100, 8), (128, 8), (129, 6), (256, 8), (257, 8), (384, 8)])
@pytest.mark.parametrize("mode,biased,renorm", [("softmax", False, True), ("softmax", True, False), ("sigmoid", True, True), ("sigmoid", False, False)])
def test_router(T, E, k, mode, biased, renorm):
    from mary_b200.ops import cuda as K
    g = torch.Generator(device="cuda").manual_seed(T * E)
    wide = torch.empty(T, E + 5, device="cuda").normal_(0, 1.5, generator=g)
    lg = wide[:, :E]
    bias = torch.empty(E, device="cuda").normal_(0, 0.1, generator=g) if biased else None
    counts, flag = torch.zeros(E, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    idx, w = K.router_topk(lg, k, mode, bias, 1, 1, 2.5, renorm, counts, flag)
    sel, want_i, want_w = _want(lg, k, mode, bias, 2.5, renorm)
    # scores carry a few roundings of f32 and the fast exponential's 2^-21: two experts closer than that may change places
    at = sel.gather(1, idx.long())
    assert (at - sel.gather(1, want_i)).abs().max() < 4e-6
    assert (idx.long() == want_i).float().mean() > 0.999
    same = (idx.long() == want_i).all(1)
    assert ((w.double() - want_w).abs()[same] <= 8e-6 * want_w[same] + 1e-7).all()
    assert torch.equal(counts.long(), torch.bincount(idx.long().flatten(), minlength=E)) and flag.item() == 0
    assert (torch.sort(idx, 1).values.diff(dim=1) > 0).all()                     # no expert twice


@pytest.mark.parametrize("T", [200, 300])
@pytest.mark.parametrize("mode", ["softmax", "sigmoid"])
def test_router_ties_masked_experts_and_bad_logits(T, mode):
    from mary_b200.ops import cuda as K
    lg = torch.zeros(T, 128, device="cuda")                                      # all equal: the lower index wins
    idx, w = K.router_topk(lg, 8, mode)
    assert torch.equal(idx, torch.arange(8, device="cuda", dtype=torch.int32).expand(T, 8)) and (w - 0.125).abs().max() < 1e-6
    lg[:, :100] = torch.finfo(torch.float32).min                                 # experts masked by the lowest value are never taken
    idx, w = K.router_topk(lg, 8, mode)
    assert torch.equal(idx, torch.arange(100, 108, device="cuda", dtype=torch.int32).expand(T, 8)) and (w - 0.125).abs().max() < 1e-6
    for bad in (float("nan"), float("inf"), float("-inf")):
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        lg[T // 2, 3] = bad
        K.router_topk(lg, 8, mode, flag=flag)
        assert flag.item() == 1
