"""Prefill-sized expert batches: the quantiser's conversion against the comparison rule over all bf16 values and scales, the routing plan over its
cluster sizes, and the 128-token GEMM tiles at their edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_quantiser_codes_every_value_at_every_scale():
    """Blocks [largest, 15 values below it]: every bf16 magnitude from the largest down to 2^-6 of it, for every largest magnitude from below the smallest
    scale to beyond the largest, both signs."""
    from mary_b200.ops import cuda_moe
    from mary_b200.ops import reference as ref
    first, last = (torch.tensor([v]).bfloat16().view(torch.int16).item() for v in (2.0 ** -8, 4096.0))
    for lo in range(first, last, 256):
        big = torch.arange(lo, min(lo + 256, last), dtype=torch.int32)
        below = big[:, None] - torch.arange(0, 7 * 128 - 1 - (7 * 128 - 1) % 15, dtype=torch.int32)[None]      # 59 blocks of 15
        v = below.clamp_min(0).view(big.numel(), -1, 15)
        sign = (torch.arange(v.numel()).view(v.shape) % 2).int() * 0x8000
        v = torch.cat([big[:, None, None].expand(-1, v.shape[1], 1), v | sign], 2).reshape(big.numel(), -1)
        pad = (-v.shape[1]) % 64
        v = torch.nn.functional.pad(v, (0, pad)).to(torch.int16).view(torch.bfloat16).cuda()
        codes, sf = cuda_moe.quantize_nvfp4(v)
        want_codes, want_sf = ref.quantize_nvfp4(v)
        assert torch.equal(sf, want_sf) and torch.equal(codes, want_codes)


def test_quantiser_special_values():
    from mary_b200.ops import cuda_moe
    x = torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda")
    x[1, :3] = torch.tensor([float("inf"), float("-inf"), 1.0])
    x[2, :4] = torch.tensor([6.0, float("nan"), -0.0, -0.01])
    x[3, :2] = float("nan")
    codes, sf = cuda_moe.quantize_nvfp4(x)
    nib = torch.stack([codes & 15, codes >> 4], -1).view(4, 64)
    assert not nib[0].any() and not sf[0].any()
    assert nib[1, :3].tolist() == [7, 15, 0] and nib[2, 0] == 7 and nib[2, 1] & 7 == 0 and nib[2, 2:4].tolist() == [8, 8]
    assert not nib[3].any() and not sf[3].any()


@pytest.mark.parametrize("n,k,E,nt", [(1, 1, 1, 32), (4095, 3, 7, 32), (4096, 8, 128, 32), (4104, 8, 385, 128), (8192, 8, 128, 128), (16385, 5, 1000, 128),
                                      (32768, 8, 128, 128), (70000, 4, 4096, 64)])
def test_plan_places_every_entry_once(n, k, E, nt):
    from mary_b200.ops import cuda_moe
    n = n // k * k
    idx = torch.randint(-1, E, (n // k, k), dtype=torch.int32, generator=torch.Generator().manual_seed(n)).cuda()
    plan = cuda_moe.moe_plan(idx, E, nt)
    flat = idx.flatten().long()
    rows = plan.row_of.long()
    counts = torch.bincount(flat[flat >= 0], minlength=E)
    padded = (counts + nt - 1) // nt * nt
    off = torch.cumsum(padded, 0) - padded
    assert torch.equal(plan.counts.long(), counts)
    assert plan.meta.tolist() == [int(padded.sum()) // nt, int(padded.sum())]
    assert (rows[flat < 0] == -1).all()
    ok = flat >= 0
    r, e = rows[ok], flat[ok]
    assert r.unique().numel() == r.numel() and (r >= off[e]).all() and (r < off[e] + counts[e]).all()
    src = torch.full((plan.max_rows,), -1, dtype=torch.int64, device="cuda")
    src[r] = (torch.arange(n, device="cuda") // k)[ok]
    assert torch.equal(plan.src_of.long(), src)
    tiles = plan.tiles[:plan.meta[0].item()].long()
    assert (tiles[:, 1] == torch.arange(tiles.shape[0], device="cuda") * nt).all() and (tiles[:, 3] == torch.arange(tiles.shape[0], device="cuda")).all()
    assert torch.equal(torch.zeros(E, dtype=torch.int64, device="cuda").index_add_(0, tiles[:, 0], tiles[:, 2]), counts)


@pytest.mark.parametrize("n,k,E,nt", [(8, 8, 8, 32), (1023, 3, 16, 32), (1024, 8, 128, 32), (1032, 8, 385, 128), (4096, 1, 4096, 32), (4097, 1, 3, 128)])
def test_plan_at_the_edges_of_a_lone_cta(n, k, E, nt):
    test_plan_places_every_entry_once(n, k, E, nt)


@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (127, 1, 1), (129, 2, 1), (260, 3, 2), (1000, 5, 2)])
def test_token_tiles_of_128_equal_those_of_32(T, E, k):
    """The same products through both epilogues: plain rows, and quantised for the next GEMM."""
    from mary_b200.ops import cuda, cuda_moe
    from mary_b200.ops.moe import NVFP4Experts
    H, F = 512, 768
    ex = NVFP4Experts.random(E, H, F, "cuda", std=0.05, seed=T)
    x = torch.randn(T, H, device="cuda", generator=torch.Generator("cuda").manual_seed(T)).bfloat16()
    idx, w = cuda.router_topk(torch.randn(T, E, device="cuda", generator=torch.Generator("cuda").manual_seed(T + 1)), k, "softmax")
    a, b = (cuda_moe.experts_forward(x, idx, w, ex, None, nt) for nt in (128, 32))
    assert torch.equal(a, b) and a.float().norm() > 0
    plan = cuda_moe.moe_plan(idx, E, 128)
    xq, sfx = cuda_moe.quantize_entries(x, plan, k, identity=False)
    h = cuda_moe.grouped_gemm(ex.w13_q, ex.w13_sf, ex.w13_s2, xq, sfx, plan, F, H, E, ex.act)       # bf16 rows, quantised by the stand-alone kernel
    hq, sfh = cuda_moe.quantize_entries(h, plan, k, identity=True)
    y = cuda_moe.grouped_gemm(ex.w2_q, ex.w2_sf, ex.w2_s2, hq, sfh, plan, H, F, E, None)
    assert torch.equal(cuda_moe.unpermute(y, plan, w, T, k), a)
    assert cuda.last_status() == 0
