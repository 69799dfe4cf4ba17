"""GPU: causal attention of blocks that go to the tcgen05 kernel (256 or 128 query rows per CTA, steps of 128 positions) against an f64
softmax over the same 16-bit inputs: remainders of tiles and steps, one tile and two tiles per CTA, one and two numbers per probability."""
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


def inputs(torch, orc, nh, nkv, hd, S, start, seed):
    q = dev(orc.to_act16(orc.fill_normal(S * nh * hd, seed, 1)), torch.float16).view(S, nh * hd)
    kc, vc = (dev(orc.to_act16(orc.fill_normal(nkv * (start + S + 3) * hd, seed, 2 + i)), torch.float16).view(nkv, start + S + 3, hd) for i in range(2))
    kc[:, start + S:] = float("nan")  # positions behind the block must not be touched
    vc[:, start + S:] = float("nan")
    return q, kc, vc


def reference(torch, q, kc, vc, nh, nkv, hd, S, start):
    L = start + S
    s = torch.einsum("skgd,kld->skgl", q.double().view(S, nkv, nh // nkv, hd), kc[:, :L].double()) * hd ** -0.5
    seen = torch.arange(L, device="cuda")[None, :] <= torch.arange(start, L, device="cuda")[:, None]
    s = s.masked_fill(~seen[:, None, None, :], float("-inf"))
    return torch.einsum("skgl,kld->skgd", s.softmax(-1), vc[:, :L].double()).reshape(S, nh * hd)


@pytest.mark.parametrize("nh,nkv,hd,S,start", [
    (32, 8, 128, 416, 0),    # 13 whole tiles of 32 positions, the last step a quarter full
    (32, 8, 128, 417, 95),   # a tile of a single position; 512 positions: whole steps
    (32, 8, 128, 1217, 320),  # two tiles per CTA, an odd number of tiles, one position in the last; 1537 positions: a step of a single one
    (32, 8, 128, 800, 800),  # two tiles per CTA and fewer than two waves of them
    (24, 8, 128, 300, 700),  # three heads: 42 positions (126 rows) per tile, two numbers per probability
    (24, 8, 128, 1600, 0),   # the same, two tiles per CTA
    (40, 8, 64, 330, 200),   # five heads: 24 positions (120 rows)
    (32, 8, 64, 1250, 1),    # heads of 64, two tiles per CTA
    (20, 20, 128, 900, 10),  # one head per KV head: tiles of 128 positions, whose steps differ by one
    (40, 40, 64, 1100, 0),   # the same in pairs
    (64, 1, 64, 230, 300),   # 64 heads: two positions per tile
    # on both sides of the lines to the form with tiles of 64 rows: 448 / 449 positions, 512 / 513, and 56 / 64 tiles with heads of 64
    (32, 8, 128, 224, 224), (32, 8, 128, 224, 225), (32, 8, 128, 256, 2304), (32, 8, 128, 289, 0),
    (32, 8, 64, 310, 202), (32, 8, 64, 310, 203), (32, 8, 64, 224, 900), (32, 8, 64, 225, 900), (16, 4, 64, 608, 600), (16, 4, 64, 608, 0),
])
def test_against_f64(cuda, orc, nh, nkv, hd, S, start):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    q, kc, vc = inputs(torch, orc, nh, nkv, hd, S, start, 891)
    got = ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, start + S + 3, hd ** -0.5)
    # f16 probabilities (2^-11 relative each, so 2^-11 of the largest |v| at most), their f32 sums and one f16 rounding of the result
    bound = (2.0 ** -10 + 2.0 ** -11) * vc[:, :start + S].double().abs().max().item()
    assert (got.double() - reference(torch, q, kc, vc, nh, nkv, hd, S, start)).abs().max().item() < bound
    assert torch.equal(got, ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, start + S + 3, hd ** -0.5))


def test_growing_scores(cuda, orc):
    """Every step has larger scores than the one before: each rescales the sums so far."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    nh, nkv, hd, S, start = 32, 8, 128, 512, 300
    q, kc, vc = inputs(torch, orc, nh, nkv, hd, S, start, 893)
    q[:] = 0.25
    kc[:, :start + S] = (torch.arange(start + S, device="cuda") * 0.02)[None, :, None].half()
    got = ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, start + S + 3, hd ** -0.5)
    bound = (2.0 ** -10 + 2.0 ** -11) * vc[:, :start + S].double().abs().max().item()
    assert (got.double() - reference(torch, q, kc, vc, nh, nkv, hd, S, start)).abs().max().item() < bound


@pytest.mark.parametrize("nh,nkv,hd,S,start", [(32, 8, 128, 420, 21), (24, 8, 128, 600, 0), (32, 8, 64, 1250, 64), (32, 8, 128, 1301, 0), (64, 8, 128, 208, 0), (64, 8, 128, 360, 0)])
def test_infinities_do_not_reach_earlier_rows(cuda, orc, nh, nkv, hd, S, start):
    """An infinity and a NaN in v, and a NaN in k, at positions inside the block: rows that do not see them keep their bits, rows that
    do are not finite where they have to be."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    q, kc, vc = inputs(torch, orc, nh, nkv, hd, S, start, 895)
    run = lambda: ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, start + S + 3, hd ** -0.5).view(S, nkv, -1, hd)
    clean = run()
    inf, nan, key = S // 3, S // 2, S - 1  # rows of the block
    vc[:, start + inf, 3] = float("inf")
    vc[:, start + nan, hd - 1] = float("nan")
    kc[:, start + key] = float("nan")
    got = run()
    assert torch.equal(got[:inf], clean[:inf])
    assert torch.equal(got[inf:key, ..., 4:hd - 1], clean[inf:key, ..., 4:hd - 1]) and torch.equal(got[inf:nan, ..., hd - 1], clean[inf:nan, ..., hd - 1])
    assert not torch.isfinite(got[inf:key, ..., 3]).any() and not torch.isfinite(got[nan:key, ..., hd - 1]).any()
    assert torch.equal(run().view(torch.int16), got.view(torch.int16))
    out = q.clone()  # in place: a tile that is computed once more still finds its queries
    ck.attn_prefill_causal(out, kc, vc, start, nh, nkv, hd, start + S + 3, hd ** -0.5, out=out)
    assert torch.equal(out.view(torch.int16).view_as(got), got.view(torch.int16))


@pytest.mark.parametrize("nh,nkv,hd,L,score", [(32, 8, 128, 65536, 17.3), (32, 8, 64, 131072, 18.0), (16, 16, 128, 65536, 17.3), (24, 8, 128, 65536, 17.3)])
def test_one_dominating_key(cuda, orc, nh, nkv, hd, L, score):
    """One position far above all others, whose equal probabilities (2^-25 of the largest, where f16 has one bit or none) count together in the sum."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    S = 640
    q = torch.full((S, nh * hd), 0.5, dtype=torch.float16, device="cuda")
    kc, vc = (torch.zeros((nkv, L, hd), dtype=torch.float16, device="cuda") for _ in range(2))
    kc[:, 0, :16] = score * hd ** 0.5 / 8
    vc[:, 0] = dev(orc.to_act16(orc.fill_normal(nkv * hd, 897, 1)), torch.float16).view(nkv, hd)
    got = ck.attn_prefill_causal(q, kc, vc, L - S, nh, nkv, hd, L, hd ** -0.5).double().view(S, nkv, nh // nkv, hd)
    others = torch.arange(L - S, L, dtype=torch.float64, device="cuda")[:, None, None, None]  # positions that a row sees behind the first
    want = vc[None, :, None, 0].double() / (1 + others * torch.exp(-8 * hd ** -0.5 * kc[0, 0, 0].double()))
    # one f16 rounding of the result, the f32 exponentials, the roundings of the f32 sums of up to 1024 steps
    assert ((got - want).abs() <= (2.0 ** -11 + 2.0 ** -14) * want.abs() + 2.0 ** -25).all()
