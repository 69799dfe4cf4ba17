"""GPU: the streaming decode attention against an f64 softmax over the same 16-bit inputs: every group size, lengths around its
16-position tiles, its slices per CTA and its 128-position and 1280-position limits, one and several sequences, few enough for
clusters and too many, with a cache row of the new token that holds NaN before the call."""
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,hd,max_seq,lens", [
    (8, 8, 64, 40, [40, 1, 16, 17]),
    (10, 5, 128, 128, [128]),
    (24, 8, 128, 129, [129, 128, 113, 2]),
    (16, 4, 64, 1281, [1281]),
    (5, 1, 128, 1100, [1024, 15, 1100]),
    (12, 2, 64, 2500, [2047, 2500]),
    (7, 1, 64, 1500, [1500]),
    (64, 8, 128, 3000, [3000]),                         # clusters of eight, two stages per warp
    (32, 8, 128, 300, [1 + 37 * i % 300 for i in range(40)]),  # four warps per unit
    (16, 16, 64, 70, [1 + 11 * i % 70 for i in range(33)]),
])
def test_streaming_decode_attention(cuda, orc, nh, nkv, hd, max_seq, lens):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    B, G = len(lens), nh // nkv
    f16 = torch.float16
    q = dev(orc.to_act16(orc.fill_normal(B * nh * hd, 891, 1)), f16).view(B, nh * hd)
    k = dev(orc.to_act16(orc.fill_normal(B * nkv * hd, 891, 2)), f16).view(B, nkv * hd)
    v = dev(orc.to_act16(orc.fill_normal(B * nkv * hd, 891, 3)), f16).view(B, nkv * hd)
    kc = dev(orc.to_act16(orc.fill_normal(B * nkv * max_seq * hd, 891, 4)), f16).view(B, nkv, max_seq, hd)
    vc = dev(orc.to_act16(orc.fill_normal(B * nkv * max_seq * hd, 891, 5)), f16).view(B, nkv, max_seq, hd)
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    for b, n in enumerate(lens):
        kc[b, :, n - 1:] = float("nan")
        vc[b, :, n - 1:] = float("nan")
    d_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
    d_pos = d_len - 1
    kc0, vc0 = kc.clone(), vc.clone()
    got = ck.attn_decode_fused_batch(q, k, v, kc, vc, cos, sin, d_pos, d_len, nh, nkv, hd, max_seq, hd ** -0.5)
    for b, n in enumerate(lens):
        q1, k1 = q[b].clone().view(nh, hd), k[b].clone().view(nkv, hd)
        ck.rope_decode_dyn_inplace(q1, k1, cos, sin, nh, nkv, hd, d_pos[b:b + 1].data_ptr())
        kc0[b, :, n - 1], vc0[b, :, n - 1] = k1, v[b].view(nkv, hd)
        s = torch.einsum("kgd,kld->kgl", q1.double().view(nkv, G, hd), kc0[b, :, :n].double()) * hd ** -0.5
        want = torch.einsum("kgl,kld->kgd", s.softmax(-1), vc0[b, :, :n].double()).reshape(-1)
        # f16 probabilities (2^-11 of the largest |v| at most), one f16 rounding of the result, f32 scores in the exponent
        bound = (2.0 ** -10 + 2.0 ** -11) * vc0[b, :, :n].double().abs().max().item()
        assert (got[b].double() - want).abs().max().item() < bound, f"sequence {b}"
        # the plain form on the same cache, one row: same bits where neither splits a row and both take eight warps per unit
        # (below 64 units and up to 128 positions), within the same bound otherwise
        one = torch.empty((nh, hd), dtype=f16, device="cuda")
        ck.flash_decode_dyn_into(q1, kc0[b], vc0[b], one, nh, nkv, d_len[b:b + 1].data_ptr(), hd, hd ** -0.5, max_seq)
        if max_seq <= 128 and B * nkv < 64:
            assert torch.equal(one.view(-1), got[b])
        assert (one.view(-1).double() - want).abs().max().item() < bound
    assert torch.equal(torch.nan_to_num(kc, nan=77.0), torch.nan_to_num(kc0, nan=77.0))
    assert torch.equal(torch.nan_to_num(vc, nan=77.0), torch.nan_to_num(vc0, nan=77.0))


@pytest.mark.parametrize("cuda_core", [False, True])
@pytest.mark.parametrize("nh,nkv,hd,max_seq,pos", [(24, 8, 128, 1000, 777), (32, 8, 128, 1280, 130), (8, 8, 64, 129, 0), (16, 2, 64, 300, 299),
                                                   (32, 8, 128, 4096, 777), (16, 4, 64, 64, 33)])
def test_rows_never_written_do_not_reach_the_output(cuda, orc, nh, nkv, hd, max_seq, pos, cuda_core):
    """One sequence: the cache from the position on holds NaN before the call, in caches for each of the kernels; the last tile of
    16 positions is cut at the new row."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    f16, G = torch.float16, nh // nkv
    q, k, v = (dev(orc.to_act16(orc.fill_normal(h * hd, 893, i)), f16).view(h, hd) for i, h in enumerate((nh, nkv, nkv)))
    kc, vc = (dev(orc.to_act16(orc.fill_normal(nkv * max_seq * hd, 893, 4 + i)), f16).view(nkv, max_seq, hd) for i in range(2))
    kc[:, pos:], vc[:, pos:] = float("nan"), float("nan")
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    d_pos = torch.tensor([pos], dtype=torch.int32, device="cuda")
    d_len = d_pos + 1
    got = torch.empty((nh, hd), dtype=f16, device="cuda")
    prev = ck.set_attn_decode_kernel(cuda_core)
    try:
        ck.attn_decode_fused(q, k, v, kc, vc, cos, sin, d_pos.data_ptr(), d_len.data_ptr(), got, nh, nkv, hd, max_seq, hd ** -0.5)
    finally:
        ck.set_attn_decode_kernel(prev)
    q1, k1 = q.clone(), k.clone()
    ck.rope_decode_dyn_inplace(q1, k1, cos, sin, nh, nkv, hd, d_pos.data_ptr())
    assert torch.equal(kc[:, pos], k1) and torch.equal(vc[:, pos], v)
    s = torch.einsum("kgd,kld->kgl", q1.double().view(nkv, G, hd), kc[:, :pos + 1].double()) * hd ** -0.5
    want = torch.einsum("kgl,kld->kgd", s.softmax(-1), vc[:, :pos + 1].double()).reshape(nh, hd)
    # f16 probabilities (2^-11 of the largest |v| at most), one f16 rounding of the result, f32 scores in the exponent
    bound = (2.0 ** -10 + 2.0 ** -11) * vc[:, :pos + 1].double().abs().max().item()
    assert (got.double() - want).abs().max().item() < bound


@pytest.mark.parametrize("B,max_seq", [(1, 2000), (3, 300), (40, 100)])
def test_a_nan_score_gives_nan(cuda, orc, B, max_seq):
    """A NaN in a key that a sequence sees, as in a softmax: NaN for the query heads of that KV head, the others keep their bits."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    nh, nkv, hd, f16 = 12, 4, 64, torch.float16
    mk = lambda sid, *shape: dev(orc.to_act16(orc.fill_normal(int(torch.tensor(shape).prod()), 899, sid)), f16).view(*shape)
    q, k, v, kc, vc = mk(1, B, nh * hd), mk(2, B, nkv * hd), mk(3, B, nkv * hd), mk(4, B, nkv, max_seq, hd), mk(5, B, nkv, max_seq, hd)
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    d_len = torch.full((B,), max_seq, dtype=torch.int32, device="cuda")
    run = lambda: ck.attn_decode_fused_batch(q, k, v, kc, vc, cos, sin, d_len - 1, d_len, nh, nkv, hd, max_seq, hd ** -0.5).view(B, nkv, 3, hd).clone()
    clean = run()
    kc[B // 2, 1, max_seq // 3, 7] = float("nan")
    got = run()
    assert torch.isnan(got[B // 2, 1]).all()
    got[B // 2, 1] = clean[B // 2, 1]
    assert torch.equal(got, clean)


@pytest.mark.parametrize("nh,nkv,hd,max_seq,lens,S", [
    (24, 8, 128, 700, [700], 0),                          # the latency kernel
    (21, 3, 64, 1280, [1111], 0),
    (12, 2, 64, 2500, [2500], 0),                         # the streaming kernel over clusters
    (24, 8, 128, 4000, [4000, 1733, 901], 0),
    (10, 2, 128, 900, [900 - 7 * i for i in range(80)], 0),  # four warps per unit
    (24, 8, 128, 1000, [1], 300),                         # blocks of positions: in tiles, the positions split over a cluster or not
    (5, 1, 64, 3000, [1], 70),
    (16, 1, 128, 600, [1], 200),
    (24, 8, 128, 500, [1], 3),                            # row by row
])
def test_probabilities_of_the_other_group_sizes_keep_32_bits(cuda, orc, nh, nkv, hd, max_seq, lens, S):
    """Group sizes other than 1, 2, 4 and 8: what is left of the error is the rounding of the result to f16 (2.0e-4 of its 2-norm); one f16
    number per probability would add as much again (2.9e-4 in all)."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    B, G, f16 = len(lens), nh // nkv, torch.float16
    mk = lambda sid, *shape: dev(orc.to_act16(orc.fill_normal(int(torch.tensor(shape).prod()), 897, sid)), f16).view(*shape)
    kc, vc = mk(4, B, nkv, max_seq, hd), mk(5, B, nkv, max_seq, hd)
    if S:
        start = max_seq - S
        q = mk(1, S, nh * hd)
        got = ck.attn_prefill_causal(q, kc[0], vc[0], start, nh, nkv, hd, max_seq, hd ** -0.5).view(S, nkv, G, hd)
        seen = torch.arange(max_seq, device="cuda")[None, :] <= torch.arange(start, max_seq, device="cuda")[:, None]
        s = torch.einsum("skgd,kld->skgl", q.double().view(S, nkv, G, hd), kc[0].double()) * hd ** -0.5
        want = torch.einsum("skgl,kld->skgd", s.masked_fill(~seen[:, None, None, :], float("-inf")).softmax(-1), vc[0].double())
    else:
        q, k, v = mk(1, B, nh * hd), mk(2, B, nkv * hd), mk(3, B, nkv * hd)
        cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
        cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
        d_len = torch.tensor(lens, dtype=torch.int32, device="cuda")
        d_pos = d_len - 1
        got = torch.empty((B, nh * hd), dtype=f16, device="cuda")
        if B == 1:
            ck.attn_decode_fused(q, k, v, kc, vc, cos, sin, d_pos.data_ptr(), d_len.data_ptr(), got, nh, nkv, hd, max_seq, hd ** -0.5)
        else:
            ck.attn_decode_fused_batch(q, k, v, kc, vc, cos, sin, d_pos, d_len, nh, nkv, hd, max_seq, hd ** -0.5, out=got)
        want = []
        for b, n in enumerate(lens):
            q1, k1 = q[b].clone().view(nh, hd), k[b].clone().view(nkv, hd)
            ck.rope_decode_dyn_inplace(q1, k1, cos, sin, nh, nkv, hd, d_pos[b:b + 1].data_ptr())
            s = torch.einsum("kgd,kld->kgl", q1.double().view(nkv, G, hd), kc[b, :, :n].double()) * hd ** -0.5
            want.append(torch.einsum("kgl,kld->kgd", s.softmax(-1), vc[b, :, :n].double()).reshape(-1))
        want = torch.stack(want)
    want = want.reshape(got.shape)
    assert ((got.double() - want).norm() / want.norm()).item() < 2.3e-4
