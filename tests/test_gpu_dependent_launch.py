"""GPU: results with programmatic dependent launch on (kernels may start while the one in front still runs) against the same
launches with it off, where a launch reads cache rows that the one in front writes.  The rows hold NaN before every call, so that
a read which comes too early shows whatever the tolerance."""
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


def _both(ck, torch, run):
    """run() with dependent launch off and on."""
    was, res = ck.set_pdl(False), []
    try:
        for on in (False, True):
            ck.set_pdl(on)
            res.append(run())
            torch.cuda.synchronize()
    finally:
        ck.set_pdl(was)
    return res


def _normal(torch, orc, shape, seed, sid):
    n = 1
    for s in shape:
        n *= s
    return dev(orc.to_act16(orc.fill_normal(n, seed, sid)), torch.float16).view(*shape)


@pytest.mark.parametrize("S,start,max_seq", [(2, 0, 64), (2, 700, 800), (6, 5, 200), (6, 1500, 1600), (16, 0, 64), (16, 250, 300)])
def test_short_prefill_blocks_see_their_own_rows(cuda, orc, S, start, max_seq):
    """The attention of a short block directly follows the launch that writes its rows, layer after layer."""
    from nve_b200 import cuda_kernels as ck
    from nve_b200 import gpu_layer as gl
    from test_gpu_glue import _make_state

    torch = cuda
    hidden, ffn, nh, nkv, hd, layers = 1024, 1792, 32, 8, 64, 6
    st = _make_state(torch, orc, hidden, ffn, nh, nkv, hd, layers, max_seq, 1105, True)
    x = _normal(torch, orc, (S, hidden), 1106, 1)
    old = [(_normal(torch, orc, (nkv, max_seq, hd), 1107, 2 * i), _normal(torch, orc, (nkv, max_seq, hd), 1107, 2 * i + 1)) for i in range(layers)]

    def run():
        for i in range(layers):
            for t, o in zip((st.kv_cache.k[i], st.kv_cache.v[i]), old[i]):
                t.copy_(o)
                t[:, start:] = float("nan")
        torch.cuda.synchronize()
        h = x
        for i in range(layers):
            h = gl.gpu_layer_forward_prefill(h, i, st, start)
        return [h] + [t[:, :start + S].clone() for t in st.kv_cache.k + st.kv_cache.v]

    off, on = _both(ck, torch, run)
    assert torch.isfinite(off[0].float()).all()
    assert all(torch.equal(a, b) for a, b in zip(off, on))


@pytest.mark.parametrize("nh,nkv,hd,max_seq,pos", [(32, 8, 128, 64, 40), (24, 8, 128, 1000, 777), (16, 16, 64, 3000, 200), (32, 8, 128, 3000, 2999)])
def test_plain_attention_behind_the_launch_that_writes_the_row(cuda, orc, nh, nkv, hd, max_seq, pos):
    """A fused launch lets its dependents start before it stores the new row; flash decode and a block of two rows come next."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    n, f16, scale = 8, torch.float16, hd ** -0.5
    q, k, v = (_normal(torch, orc, (h * hd,), 1110, i) for i, h in enumerate((nh, nkv, nkv)))
    q2 = _normal(torch, orc, (2, nh * hd), 1110, 4)
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    old = [(_normal(torch, orc, (nkv, max_seq, hd), 1111, 2 * i), _normal(torch, orc, (nkv, max_seq, hd), 1111, 2 * i + 1)) for i in range(n)]
    d_pos = torch.tensor([pos], dtype=torch.int32, device="cuda")
    d_len = d_pos + 1

    def run():
        caches = [(a.clone(), b.clone()) for a, b in old]
        for a, b in caches:
            a[:, pos:], b[:, pos:] = float("nan"), float("nan")
        first, single, block = (torch.zeros((n,) + s, dtype=f16, device="cuda") for s in ((nh, hd), (nh, hd), (2, nh * hd)))
        torch.cuda.synchronize()
        for i, (kc, vc) in enumerate(caches):
            ck.attn_decode_fused(q, k, v, kc, vc, cos, sin, d_pos.data_ptr(), d_len.data_ptr(), first[i], nh, nkv, hd, max_seq, scale)
            ck.flash_decode_dyn_into(q2[0], kc, vc, single[i], nh, nkv, d_len.data_ptr(), hd, scale, max_seq)
            ck.attn_decode_fused(q, k, v, kc, vc, cos, sin, d_pos.data_ptr(), d_len.data_ptr(), first[i], nh, nkv, hd, max_seq, scale)
            ck.attn_prefill_causal(q2, kc, vc, pos - 1, nh, nkv, hd, max_seq, scale, out=block[i])
        return [first, single, block] + [t[:, :pos + 1] for c in caches for t in c]

    off, on = _both(ck, torch, run)
    assert all(torch.isfinite(t.float()).all() for t in off[:3])
    assert all(torch.equal(a, b) for a, b in zip(off, on))


@pytest.mark.parametrize("cuda_core", [False, True])
@pytest.mark.parametrize("nh,nkv,hd,max_seq,pos", [(32, 8, 128, 64, 14), (24, 8, 128, 1000, 777), (16, 16, 64, 3000, 2000)])
def test_fused_attention_of_successive_positions(cuda, orc, nh, nkv, hd, max_seq, pos, cuda_core):
    """Three positions one after the other on the same cache, nothing in between: each reads the row that the launch in front writes.
    One sequence and several."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    B, steps, f16, scale = 4, 3, torch.float16, hd ** -0.5
    q, k, v = (_normal(torch, orc, (steps, B, h * hd), 1120, i) for i, h in enumerate((nh, nkv, nkv)))
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    old = [_normal(torch, orc, (B, nkv, max_seq, hd), 1121, i) for i in range(2)]
    d_pos = torch.arange(pos, pos + steps, dtype=torch.int32, device="cuda").view(steps, 1).repeat(1, B)
    d_len = d_pos + 1

    def run():
        out = torch.zeros((2, steps, B, nh * hd), dtype=f16, device="cuda")
        (kc, vc), (kb, vb) = ([t.clone() for t in old] for _ in range(2))
        for t in (kc, vc, kb, vb):
            t[:, :, pos:] = float("nan")
        torch.cuda.synchronize()
        for b in range(B):
            for s in range(steps):
                ck.attn_decode_fused(q[s, b], k[s, b], v[s, b], kc[b], vc[b], cos, sin, d_pos[s, b:].data_ptr(), d_len[s, b:].data_ptr(),
                                     out[0, s, b], nh, nkv, hd, max_seq, scale)
        for s in range(steps):
            ck.attn_decode_fused_batch(q[s], k[s], v[s], kb, vb, cos, sin, d_pos[s], d_len[s], nh, nkv, hd, max_seq, scale, out=out[1, s])
        return [out] + [t[:, :, :pos + steps].clone() for t in (kc, vc, kb, vb)]

    prev = ck.set_attn_decode_kernel(cuda_core)
    try:
        off, on = _both(ck, torch, run)
    finally:
        ck.set_attn_decode_kernel(prev)
    assert torch.isfinite(off[0].float()).all()
    assert all(torch.equal(a, b) for a, b in zip(off, on))


@pytest.mark.parametrize("M,N,K", [(9, 64, 64), (64, 2048, 256)])
def test_fused_attention_two_launches_behind(cuda, orc, M, N, K):
    """Attention of a position, a GEMM of another size, attention two positions on: rows that the first wrote are read early by the last, which
    may start when the GEMM's loads are done -- but not before the first is complete."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    nh, nkv, hd, max_seq, pos, f16 = 64, 8, 128, 1200, 1000, torch.float16
    q, k, v = (_normal(torch, orc, (2, h * hd), 1130, i) for i, h in enumerate((nh, nkv, nkv)))
    cos, sin = orc.rope_tables_f32(hd, max_seq, 10000.0)
    cos, sin = dev(orc.to_act16(cos), f16), dev(orc.to_act16(sin), f16)
    old = [_normal(torch, orc, (nkv, max_seq, hd), 1131, i) for i in range(2)]
    d_pos = torch.tensor([pos, pos + 40], dtype=torch.int32, device="cuda")
    d_len = d_pos + 1
    nib, sc = ck.q4_quantize(ck.fill_normal(N * K, 1132, 1, scale=0.02).view(N, K))
    x = _normal(torch, orc, (M, K), 1133, 1)

    def run():
        outs = []
        y = torch.empty((M, N), dtype=f16, device="cuda")
        for _ in range(8):
            kc, vc = (t.clone() for t in old)
            kc[:, pos], vc[:, pos], kc[:, pos + 40:], vc[:, pos + 40:] = (float("nan"),) * 4
            out = torch.zeros((2, nh, hd), dtype=f16, device="cuda")
            torch.cuda.synchronize()
            ck.attn_decode_fused(q[0], k[0], v[0], kc, vc, cos, sin, d_pos.data_ptr(), d_len.data_ptr(), out[0], nh, nkv, hd, max_seq, hd ** -0.5)
            ck.gemm_w4a16(x, nib, sc, N, K, out=y)
            ck.attn_decode_fused(q[1], k[1], v[1], kc, vc, cos, sin, d_pos[1:].data_ptr(), d_len[1:].data_ptr(), out[1], nh, nkv, hd, max_seq, hd ** -0.5)
            outs.append(out)
        return outs

    off, on = _both(ck, torch, run)
    assert all(torch.isfinite(t.float()).all() for t in off)
    assert all(torch.equal(a, b) for a, b in zip(off, on))
