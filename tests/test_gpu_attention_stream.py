"""The streaming decode attention (csrc/kernels/attention_stream.cu) against 64-bit attention: head widths, rows per kv head, both cache types, key
ranges that end inside a group, splits that stay empty, windows, the cap, and pages of every size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(q_lens, kv_lens, page, seed):
    from mary_b200.runtime.batch import BatchMeta
    need = [-(-n // page) for n in kv_lens]
    order = np.random.default_rng(seed).permutation(sum(need) + 3).astype(np.int32)
    table = np.zeros((len(need), max(need)), np.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return BatchMeta.build(q_lens, kv_lens, table, page, "cuda"), table, sum(need) + 3


def _exact(q, k, v, table, q_lens, kv_lens, page, scale, window, cap):
    out, at = torch.empty(q.shape, dtype=torch.float64, device="cuda"), 0
    g = q.shape[1] // k.shape[2]
    for s, (m, n) in enumerate(zip(q_lens, kv_lens)):
        p = np.arange(n)
        slots = torch.from_numpy(table[s, p // page].astype(np.int64) * page + p % page).cuda()
        ks, vs = (t.reshape(-1, *t.shape[2:])[slots].repeat_interleave(g, 1) for t in (k, v))
        x = torch.einsum("thd,lhd->htl", q[at:at + m].double(), ks) * scale
        if cap:
            x = cap * torch.tanh(x / cap)
        pos = torch.arange(n - m, n, device="cuda")[:, None]
        keys = torch.arange(n, device="cuda")[None]
        hide = (keys > pos) | ((pos - keys >= window) if window else torch.zeros_like(keys > pos))
        out[at:at + m] = torch.einsum("htl,lhd->thd", torch.softmax(x.masked_fill(hide[None], -torch.inf), -1), vs)
        at += m
    return out


CASES = [  # D, q heads, kv heads, q_lens, kv_lens, page, window, cap
    (256, 16, 8, [1], [1], 16, 0, 0.0), (256, 2, 1, [1, 1, 1], [777, 64, 65], 16, 0, 0.0), (256, 16, 8, [1] * 5, [1024, 1025, 1500, 31, 33], 16, 1024, 0.0), (256, 8, 8, [2, 1], [500, 40], 16, 64, 30.0), (256, 4, 4, [1], [2049], 64, 0, 0.0),
    (256, 4, 4, [2, 4, 1], [700, 4, 129], 32, 100, 0.0), (256, 4, 1, [1, 1], [333, 2100], 64, 0, 30.0), (128, 8, 8, [1, 1], [257, 15], 16, 0, 0.0),
    (128, 8, 2, [2, 2, 1], [300, 2, 900], 16, 128, 0.0), (128, 8, 1, [1, 1], [513, 8], 16, 0, 0.0), (64, 4, 2, [1, 3], [100, 1000], 16, 0, 50.0),
    (64, 8, 1, [1], [4097], 64, 0, 0.0), (64, 4, 4, [8], [200], 16, 33, 0.0)]


@pytest.mark.parametrize("case", CASES, ids=str)
@pytest.mark.parametrize("q8", [False, True])
@pytest.mark.parametrize("nsplit,warps", [(None, None), (1, 4), (4, 8), (8, 4)])
def test_stream_attention(case, q8, nsplit, warps):
    from mary_b200.ops import cuda as K
    from mary_b200.runtime.kv_cache import Q8Pages
    D, Hq, Hkv, q_lens, kv_lens, page, window, cap = case
    if not q8 and (D != 256 or max(q_lens) * Hq // Hkv > 2):
        pytest.skip("bf16 shapes of the tensor-core kernel")
    meta, table, pages = _batch(q_lens, kv_lens, page, 1)
    g = torch.Generator(device="cuda").manual_seed(2)
    k, v = (torch.empty(pages, page, Hkv, D, dtype=torch.bfloat16, device="cuda").normal_(0.2, 1.0, generator=g) for _ in range(2))
    q = torch.empty(sum(q_lens), Hq, D, dtype=torch.bfloat16, device="cuda").normal_(0, 0.3, generator=g)
    scale = 3.0 * D ** -0.5
    if q8:
        kc, vc = Q8Pages(pages, page, Hkv, D, "cuda"), Q8Pages(pages, page, Hkv, D, "cuda")
        for t, r in ((kc, k), (vc, v)):
            t.codes, t.sz = Q8Pages.quantize(r)
        k64, v64 = (t.codes.double() * t.sz[..., :1].double() + t.sz[..., 1:].double() for t in (kc, vc))
    else:
        kc, vc, k64, v64 = k, v, k.double(), v.double()
    got = K.attention_stream(q, kc, vc, meta, scale, window, cap, nsplit, warps).double()
    want = _exact(q, k64, v64, table, q_lens, kv_lens, page, scale, window, cap)
    # one rounding to bf16 (2^-9 of the value), f32 everywhere before it (the cap's tangent: 2^-10 of a score of at most 3 standard deviations)
    assert (got - want).norm() / want.norm() < (2.0 ** -8 if cap == 0 else 2.0 ** -7)
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -8 * want.abs().max()).all()
    assert K.last_status() == 0


def test_stream_attention_strided_cache():
    """Caches that are slices of a wider store (token and page strides of their own, different for K and V)."""
    from mary_b200.ops import cuda as K
    meta, table, pages = _batch([1, 1], [400, 123], 16, 3)
    store = torch.randn(pages, 2, 16, 2, 2, 256, device="cuda").bfloat16()
    k, v = store[:, 0, :, 0], store[:, 1, :, 1]
    wide = torch.randn(pages, 20, 2, 256, device="cuda").bfloat16()[:, :16]
    q = torch.randn(2, 4, 256, device="cuda").bfloat16()
    for vc in (v, wide):
        got = K.attention_stream(q, k, vc, meta, 0.1).double()
        want = _exact(q, k.double(), vc.double(), table, [1, 1], [400, 123], 16, 0.1, 0, 0.0)
        assert (got - want).norm() / want.norm() < 2.0 ** -8


def test_more_query_blocks_than_a_grid_has_rows():
    """70000 sequences of one to three keys over an 8-bit cache."""
    from mary_b200 import ops
    from mary_b200.runtime.batch import BatchMeta
    from mary_b200.runtime.kv_cache import Q8Pages
    from mary_b200.ops import cuda as K
    S = 70000
    kv = np.arange(S, dtype=np.int32) % 3 + 1
    meta = BatchMeta.build(np.ones(S, dtype=np.int32), kv, np.arange(S, dtype=np.int32)[:, None], 4, "cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    kc, vc = Q8Pages(S, 4, 1, 64, "cuda"), Q8Pages(S, 4, 1, 64, "cuda")
    for t in (kc, vc):
        t.codes, t.sz = Q8Pages.quantize(torch.empty(S, 4, 1, 64, device="cuda").normal_(0, 1, generator=g))
    q = torch.empty(S, 1, 64, dtype=torch.bfloat16, device="cuda").normal_(0, 0.3, generator=g)
    got = ops.paged_attention(q, kc, vc, meta, 0.5)
    k64, v64 = ((t.codes.double() * t.sz[..., :1].double() + t.sz[..., 1:].double())[:, :, 0] for t in (kc, vc))
    x = torch.einsum("sd,std->st", q[:, 0].double(), k64) * 0.5
    x = x.masked_fill(torch.arange(4, device="cuda")[None] >= torch.from_numpy(kv).cuda()[:, None], -torch.inf)
    want = torch.einsum("st,std->sd", torch.softmax(x, -1), v64)
    assert (got[:, 0].double() - want).norm() / want.norm() < 2.0 ** -8
    assert K.last_status() == 0
