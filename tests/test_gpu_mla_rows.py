"""The row kernels around latent attention in their vector forms: head counts that leave groups unfilled, projections of every register depth, the rows
that fall back, and slots outside the cache."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _meta(T, slots=None):
    return SimpleNamespace(positions=torch.arange(5, 5 + T, dtype=torch.int32, device="cuda"),
                           slot_mapping=torch.randperm(T, device="cuda") if slots is None else slots)


def _turn(x, pos, inv):
    a = pos.double()[:, None] * inv.double()[None]
    c, s = a.cos(), a.sin()
    while c.dim() < x.dim():
        c, s = c[:, None], s[:, None]
    x1, x2 = x[..., :32], x[..., 32:]
    return torch.cat([x1 * c - x2 * s, x1 * s + x2 * c], -1)


@pytest.mark.parametrize("H", [1, 3, 16, 17, 64])
@pytest.mark.parametrize("T", [1, 37])
def test_query_rotation_and_shared_key_dims(H, T):
    from mary_b200.ops import cuda as K
    inv = 10000.0 ** (-torch.arange(32, device="cuda").float() / 32)
    m = _meta(T)
    for off in (0, 1):                             # rows that no 8-byte access can take fall back
        store = torch.randn(T * H * 192 + 1, device="cuda").bfloat16()
        qb = store[off:off + T * H * 192].view(T, H * 192)
        was = qb.clone().view(T, H, 192)
        K.mla_q_rope_inplace(qb, inv, m, H)
        got = qb.view(T, H, 192)
        assert torch.equal(got[..., :128], was[..., :128])
        # one bf16 rounding; the angles (up to 42) come from the fast sine, exact to 2^-21 of a turn there
        assert ((got[..., 128:].double() - _turn(was[..., 128:].double(), m.positions, inv)).abs() <= 2.0 ** -8 * 6).all()
    rows = torch.randn(T, 576, device="cuda").bfloat16()
    uk, uv = torch.randn(H * 128, 512, device="cuda").bfloat16() * 0.05, torch.randn(H * 128, 512, device="cuda").bfloat16() * 0.05
    k, v = K.mla_expand_kv(rows, uk, uv, H)
    want = (rows[:, :512].double() @ uk.double().t()).view(T, H, 128)
    assert (k[..., :128].double() - want).norm() / want.norm() < 2.0 ** -8
    assert torch.equal(k[..., 128:], rows[:, None, 512:].expand(T, H, 64))
    assert (v.double() - (rows[:, :512].double() @ uv.double().t()).view(T, H, 128)).norm() / v.double().norm() < 2.0 ** -8
    assert K.last_status() == 0


@pytest.mark.parametrize("T,H", [(64, 64), (65, 64), (300, 17), (4100, 1), (64, 128), (241, 17)])
def test_query_rotation_of_many_heads(T, H):
    """Around 4096 heads in all, from where a warp walks 16 heads: groups that are left unfilled."""
    test_query_rotation_and_shared_key_dims(H, T)


@pytest.mark.parametrize("q_lora", [8, 64, 1536, 1544, 6144, 6152, 36])
def test_prep_norms_and_appends(q_lora):
    from mary_b200.ops import cuda as K
    T = 21
    inv = 10000.0 ** (-torch.arange(32, device="cuda").float() / 32)
    x = torch.randn(T, q_lora + 576, device="cuda").bfloat16()
    wq, wk = (torch.randn(n, device="cuda").bfloat16() * 0.1 + 1 for n in (q_lora, 512))
    cache = torch.zeros(4, 16, 576, dtype=torch.bfloat16, device="cuda")
    slots = torch.randperm(64, device="cuda")[:T]
    slots[3] = 64
    m = _meta(T, slots)
    qa = K.mla_prep(x, q_lora, wq, wk, inv, m, cache, 1e-6)
    rms = lambda v, w: v.double() * torch.rsqrt(v.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()  # noqa: E731
    want = rms(x[:, :q_lora], wq)
    assert ((qa.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
    assert K.last_status() == 6                    # the slot outside the cache is reported ...
    keep = torch.arange(T, device="cuda") != 3     # ... and nothing else is lost
    got = cache.view(64, 576)[slots[keep]].double()
    lat = rms(x[keep, q_lora:q_lora + 512], wk)
    assert ((got[:, :512] - lat).abs() <= 2.0 ** -8 * lat.abs() + 1e-6).all()
    assert ((got[:, 512:] - _turn(x[keep, q_lora + 512:].double(), m.positions[keep], inv)).abs() <= 2.0 ** -8 * 6).all()
    assert cache.view(64, 576).abs().sum(1).count_nonzero() == T - 1
