"""The row kernels of the decoders (norms, head norm + rotation + append) over their forms: one to three chunks of 8 values per thread, every vector width of
the head kernel, one and four heads per warp with groups left unfilled, rows that no vector access can take, slots outside the cache."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rms(x, w=None, eps=1e-6):
    y = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _near(got, want, ulps=1.0):
    """Within ``ulps`` roundings to bf16 (2^-8 of the value at most) and what f32 sums leave."""
    assert not torch.isnan(got).any()
    assert ((got.double() - want).abs() <= ulps * 2.0 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("H", [8, 264, 4088, 4096, 4104, 8192, 8200, 12280, 12288])
@pytest.mark.parametrize("T", [1, 5, 700])
@pytest.mark.parametrize("f32", [False, True])
def test_norms(H, T, f32):
    from mary_b200.ops import cuda as K
    g = torch.Generator(device="cuda").manual_seed(H + T)
    rn = lambda *s, std=1.0, mean=0.0: torch.empty(*s, device="cuda").normal_(mean, std, generator=g)  # noqa: E731
    x = rn(T, H, std=2.0) if f32 else rn(T, H, std=2.0).bfloat16()
    w, w2, h = rn(H, std=0.2, mean=1.0).bfloat16(), rn(H, std=0.2, mean=1.0).bfloat16(), rn(T, H).bfloat16()
    _near(K.rmsnorm(x, w), _rms(x, w))
    _near(K.rmsnorm(x), _rms(x))
    wide = torch.zeros(T, H + 16, dtype=x.dtype, device="cuda")
    wide[:, 8:8 + H] = x
    _near(K.rmsnorm(wide[:, 8:8 + H], w), _rms(x, w))
    res = h.clone()
    y, res = K.add_rmsnorm(x, res, w)
    assert torch.equal(res, (h.float() + x.float()).bfloat16())
    _near(y, _rms(res, w))
    for nxt in (w2, None):
        xo, hn = K.norm_add_norm(x, w, h.clone(), nxt, 1e-6, 0.5)
        # the branch's rounding to bf16 may fall the other way where the f32 sum of squares does: one unit of it, then the sum's own rounding
        want = (h.double() + _rms(x, w)) * 0.5
        assert ((hn.double() - want).abs() <= 2.0 ** -8 * (want.abs() + 0.5 * _rms(x, w).abs()) + 1e-5).all()
        if nxt is not None:
            _near(xo, _rms(hn, w2))
    assert K.last_status() == 0


@pytest.mark.parametrize("D", [64, 128, 256, 512, 96])
@pytest.mark.parametrize("heads,kv,T", [(4, 1, 3), (3, 2, 2500), (16, 8, 600), (5, 0, 2100), (1, 1, 3000)])
@pytest.mark.parametrize("norm", [False, True])
def test_head_norm_rotation_append(D, heads, kv, T, norm):
    from mary_b200.ops import cuda as K
    g = torch.Generator(device="cuda").manual_seed(D + T)
    for off in (0, 1):                                       # one element off: rows that no vector access can take
        n = T * (heads + 2 * kv) * D
        qkv = torch.empty(n + off, device="cuda").normal_(0, 2, generator=g).bfloat16()[off:].view(T, -1)
        qn, kn = (torch.empty(D, device="cuda").normal_(1, 0.2, generator=g).bfloat16() if norm else None for _ in range(2))
        inv = 10000.0 ** (-torch.arange(D // 2, device="cuda").float() * 2 / D)
        pages = (T + 15) // 16 + 1
        slots = torch.randperm(pages * 16, device="cuda", generator=g)[:T]
        bad = kv > 0 and T > 3
        if bad:
            slots[3] = pages * 16                            # outside the cache: reported, nothing written
        m = SimpleNamespace(positions=torch.randint(0, 60, (T,), device="cuda", dtype=torch.int32, generator=g), slot_mapping=slots)
        kc, vc = (torch.zeros(pages, 16, max(kv, 1), D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        q = K.qk_norm_rope_append(qkv, heads, kv, D, qn, kn, norm, inv, m, kc, vc, 1e-6)
        x = qkv.double().view(T, heads + 2 * kv, D)
        rnd = lambda v: v.bfloat16().double()                # noqa: E731  (normed heads are rounded before they turn)
        parts = [x[:, :heads], x[:, heads:heads + kv], x[:, heads + kv:]]
        if norm:
            parts = [rnd(_rms(parts[0], qn)), rnd(_rms(parts[1], kn)), rnd(_rms(parts[2]))]
        a = m.positions.double()[:, None] * inv.double()
        c, s = a.cos()[:, None], a.sin()[:, None]
        turn = lambda v: torch.cat([v[..., :D // 2] * c - v[..., D // 2:] * s, v[..., :D // 2] * s + v[..., D // 2:] * c], -1)  # noqa: E731
        # a normed value's rounding may fall the other way (2^-8 of it, carried by the turn), then the result's own; the fast sine is exact to 2^-21 of a turn
        close = lambda got, want: ((got.double() - want).abs() <= 2.0 ** -8 * (want.abs() + 8.0)).all()  # noqa: E731
        assert close(q, turn(parts[0]))
        keep = torch.arange(T, device="cuda") != 3 if bad else torch.ones(T, dtype=torch.bool, device="cuda")
        if kv:
            assert close(kc.view(-1, kv, D)[slots[keep]], turn(parts[1])[keep]) and close(vc.view(-1, kv, D)[slots[keep]], parts[2][keep])
            assert kc.view(-1, kv * D).abs().sum(1).count_nonzero() == int(keep.sum())
        assert K.last_status() == (6 if bad else 0)
