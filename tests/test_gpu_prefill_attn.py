"""GPU: the tiled causal attention of a block of new positions against an f64 softmax over the same 16-bit inputs, at
the edges of its tiles (64 query rows, 64 positions per step) and with the positions of a tile split over a cluster."""
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,hd,S,start", [
    (32, 8, 128, 32, 32),    # 32 positions x 4 heads per KV head, 64 positions in all
    (32, 8, 128, 33, 31),    # one position more than two tiles
    (24, 8, 128, 43, 0),     # 3 heads per KV head: 21 positions (63 rows) per tile, one position in the third
    (24, 8, 128, 8, 1013),   # few rows behind a longer prefix
    (8, 8, 64, 129, 64),     # one head per KV head, a tile of a single row
    (5, 1, 64, 70, 250),     # odd group
    (16, 1, 128, 64, 5),     # more heads per KV head than the decode kernels take
    (64, 2, 128, 300, 700),  # several tiles, split in two or four
    (32, 8, 128, 38, 2050),  # three tiles per KV head, the last of six positions, four CTAs each
    (32, 8, 128, 16, 500),   # a short block: the streaming kernel, row by row
    (32, 8, 128, 33, 3000),  # few rows, but too much K/V to read row by row
])
def test_tiled_causal_attention(cuda, orc, nh, nkv, hd, S, start):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    max_seq, G = start + S + 3, nh // nkv
    q = dev(orc.to_act16(orc.fill_normal(S * nh * hd, 881, 1)), torch.float16).view(S, nh * hd)
    kc = dev(orc.to_act16(orc.fill_normal(nkv * max_seq * hd, 881, 2)), torch.float16).view(nkv, max_seq, hd)
    vc = dev(orc.to_act16(orc.fill_normal(nkv * max_seq * hd, 881, 3)), torch.float16).view(nkv, max_seq, hd)
    kc[:, start + S:] = float("nan")  # positions behind the block must not be touched
    vc[:, start + S:] = float("nan")
    got = ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, max_seq, hd ** -0.5)
    L = start + S
    qd = q.double().view(S, nkv, G, hd)
    s = torch.einsum("skgd,kld->skgl", qd, kc[:, :L].double()) * hd ** -0.5
    seen = torch.arange(L, device="cuda")[None, :] <= torch.arange(start, L, device="cuda")[:, None]
    s = s.masked_fill(~seen[:, None, None, :], float("-inf"))
    want = torch.einsum("skgl,kld->skgd", s.softmax(-1), vc[:, :L].double()).reshape(S, nh * hd)
    # f16 probabilities (2^-11 relative each, so 2^-11 of the largest |v| at most) and one f16 rounding of the result,
    # plus f32 scores and sums (2^-16 of a score of at most ~60 in the exponent)
    bound = (2.0 ** -10 + 2.0 ** -11) * vc[:, :L].double().abs().max().item()
    assert (got.double() - want).abs().max().item() < bound


@pytest.mark.parametrize("nh,nkv,hd,S,start", [(32, 8, 128, 40, 21), (24, 8, 128, 130, 0), (8, 8, 64, 129, 64), (64, 2, 128, 300, 700),
                                               (32, 8, 128, 16, 5), (5, 1, 64, 70, 250)])
def test_infinities_do_not_reach_earlier_rows(cuda, orc, nh, nkv, hd, S, start):
    """An infinity and a NaN in v, and a NaN in k, at positions inside the block: rows that do not see them keep their bits, rows that
    do are not finite where they have to be."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    max_seq = start + S
    q = dev(orc.to_act16(orc.fill_normal(S * nh * hd, 885, 1)), torch.float16).view(S, nh * hd)
    kc, vc = (dev(orc.to_act16(orc.fill_normal(nkv * max_seq * hd, 885, 2 + i)), torch.float16).view(nkv, max_seq, hd) for i in range(2))
    clean = ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, max_seq, hd ** -0.5).view(S, nkv, -1, hd)
    inf, nan, key = S // 3, S // 2, S - 1  # rows of the block
    vc[:, start + inf, 3] = float("inf")
    vc[:, start + nan, hd - 1] = float("nan")
    kc[:, start + key] = float("nan")
    got = ck.attn_prefill_causal(q, kc, vc, start, nh, nkv, hd, max_seq, hd ** -0.5).view(S, nkv, -1, hd)
    assert torch.equal(got[:inf], clean[:inf])
    assert torch.equal(got[inf:key, ..., 4:hd - 1], clean[inf:key, ..., 4:hd - 1]) and torch.equal(got[inf:nan, ..., hd - 1], clean[inf:nan, ..., hd - 1])
    assert not torch.isfinite(got[inf:key, ..., 3]).any() and not torch.isfinite(got[nan:key, ..., hd - 1]).any()
