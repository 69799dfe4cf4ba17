"""GPU: the batched GEMM beyond 64 rows of x and with what a layer does to its product (residual add + RMSNorm, SiLU*up)
finished inside: at the edges of its tiles (256 weight rows, 128 with SiLU*up; up to 256 rows of x; units of 256 along K),
with and without runs that cut tiles, against the separate launches and an f64 product of the dequantised weights."""
import pytest

from helpers import dev, rel_rms_err

pytestmark = pytest.mark.gpu


def _weights(torch, orc, N, K, seed):
    nib, sc = orc.extract_for_gpu(orc.quantize_q4(orc.fill_normal(N * K, seed, 1, scale=0.02).reshape(N, K)))
    dn, ds = dev(nib), dev(sc)
    q = torch.empty((N, K // 32, 32), dtype=torch.float64, device="cuda")
    b = dn.view(N, K // 32, 16)
    q[:, :, :16], q[:, :, 16:] = (b & 15).double() - 8, (b >> 4).double() - 8
    return (dn, ds, N), (q * ds.double()[:, :, None]).view(N, K)


def _x(torch, orc, M, K, seed):
    return dev(orc.to_act16(orc.fill_normal(M * K, seed, 2)), torch.float16).view(M, K)


@pytest.mark.parametrize("M,Ns,K", [(65, (256,), 64), (128, (257, 255), 320), (129, (512,), 4096), (256, (300,), 576), (257, (40, 600, 256), 1024),
                                    (513, (1024,), 14336), (700, (2304,), 512)])
def test_wide_gemm(cuda, orc, M, Ns, K):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x = _x(torch, orc, M, K, 990)
    ws = [_weights(torch, orc, n, K, 991 + i) for i, n in enumerate(Ns)]
    outs = [torch.full((M, n), float("nan"), dtype=torch.float16, device="cuda") for n in Ns]
    ck.gemm_w4a16_wide(x, [t for t, _ in ws], K, outs)
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    for o, (_, w) in zip(outs, ws):
        # f16 rounding of weights (2^-12 RMS each) and result: the bound of the narrow batches
        assert rel_rms_err(o.float().cpu().numpy(), (x.double() @ w.t()).cpu().numpy()) < 1e-2


@pytest.mark.parametrize("M,N,K", [(2, 64, 64), (33, 1024, 4096), (64, 4096, 512), (130, 3072, 1088), (300, 8192, 256)])
def test_gemm_add_rmsnorm_equals_separate_launches(cuda, orc, M, N, K):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x, (w, _) = _x(torch, orc, M, K, 995), _weights(torch, orc, N, K, 996)
    res = _x(torch, orc, M, N, 997)
    norm = dev(orc.to_act16(1.0 + 0.1 * orc.fill_normal(N, 998, 3)), torch.float16)
    h, normed = torch.empty_like(res), torch.empty_like(res)
    ck.gemm_w4a16_add_rmsnorm(x, w, K, res, norm, 1e-5, h, normed)
    want = torch.empty_like(res)
    ck.gemm_w4a16_wide(x, [w], K, [want])
    want_n = ck.add_rms_norm_rows(want, res, norm, 1e-5)
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    assert torch.equal(h, want) and torch.equal(normed, want_n)


@pytest.mark.parametrize("M,N,K,scratch", [(2, 64, 64, True), (16, 200, 4096, True), (61, 14336, 512, True), (64, 4096, 1024, False),
                                           (200, 129, 768, True), (300, 1536, 3072, True)])
def test_gemm_gateup_silu_matches_separate_launches(cuda, orc, M, N, K, scratch):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x, (g, gw), (u, uw) = _x(torch, orc, M, K, 1001), _weights(torch, orc, N, K, 1002), _weights(torch, orc, N, K, 1003)
    mid = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    # sixteen bytes hold no partial tile: every pair of SMs then takes whole tiles
    ck.gemm_w4a16_gateup_silu(x, g, u, K, mid, None if scratch else torch.empty(16, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    gd, ud = x.double() @ gw.t(), x.double() @ uw.t()
    # the two f16 products carry 3e-3 of their RMS at most, so does their combination (|silu'| <= 1.1)
    assert rel_rms_err(mid.float().cpu().numpy(), (torch.nn.functional.silu(gd) * ud).cpu().numpy()) < 2e-2


@pytest.mark.parametrize("S,start,nh,nkv,hd", [(2, 0, 16, 4, 64), (63, 5, 12, 4, 64), (130, 60, 6, 2, 128)])
def test_prefill_layer_equals_separate_launches(cuda, orc, S, start, nh, nkv, hd):
    from nve_b200 import gpu_layer as gl
    from test_gpu_glue import _make_state

    torch = cuda
    hidden, ffn, max_seq = 1024, 1792, 200
    st = _make_state(torch, orc, hidden, ffn, nh, nkv, hd, 1, max_seq, 1005, True)
    for t in (st.kv_cache.k[0], st.kv_cache.v[0]):
        t.copy_(_x(torch, orc, nkv * max_seq, hd, 1006).view(nkv, max_seq, hd))
    k0, v0 = st.kv_cache.k[0].clone(), st.kv_cache.v[0].clone()
    x = _x(torch, orc, S, hidden, 1007)
    got = gl.gpu_layer_forward_prefill(x, 0, st, start)
    k1, v1 = st.kv_cache.k[0].clone(), st.kv_cache.v[0].clone()
    st.kv_cache.k[0].copy_(k0), st.kv_cache.v[0].copy_(v0)
    # activation multipliers of one send every projection through its own launch
    w = st.layer_weights[0]
    for p in (w.q_proj, w.k_proj, w.v_proj, w.o_proj, w.gate_proj, w.up_proj, w.down_proj):
        p.awq_scales = torch.ones(p.k, dtype=torch.float32, device="cuda")
    want = gl.gpu_layer_forward_prefill(x, 0, st, start)
    torch.cuda.synchronize()
    # the same f16 values summed in another order where the split over K differs: a few f16 ulps after the layer
    for a, b in ((got, want), (k1, st.kv_cache.k[0]), (v1, st.kv_cache.v[0])):
        assert rel_rms_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < 5e-3
    assert torch.equal(k1[:, :start], k0[:, :start]) and torch.equal(k1[:, start + S:], k0[:, start + S:])


@pytest.mark.parametrize("M,N,K", [(5, 640, 2048), (16, 640, 4096), (200, 520, 1024)])
@pytest.mark.parametrize("off", [4, 8, 12])
def test_workspace_of_any_alignment(cuda, orc, M, N, K, off):
    """A workspace that starts between two 16-byte boundaries gives the bits of an aligned one, also where it is so much too small that
    runs get longer; the bytes around it stay as they are."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x, (g, _), (u, _) = _x(torch, orc, M, K, 1030), _weights(torch, orc, N, K, 1031), _weights(torch, orc, N, K, 1032)
    res, norm = _x(torch, orc, M, N, 1033), dev(orc.to_act16(1.0 + 0.1 * orc.fill_normal(N, 1034, 3)), torch.float16)
    need = max(ck.gemm_w4a16_multi_scratch_bytes(M, [N], K), ck.gemm_w4a16_silu_scratch_bytes(M, N, K))
    out = []
    for o, nbytes in ((0, need), (off, need), (0, 8), (off, 8)):
        buf = torch.full((nbytes + 32,), 255, dtype=torch.uint8, device="cuda")
        ws = buf[o:o + nbytes + 16]
        y, h, normed, mid = (torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(4))
        ck.gemm_w4a16_wide(x, [g], K, [y], ws)
        ck.gemm_w4a16_add_rmsnorm(x, g, K, res, norm, 1e-5, h, normed, ws)
        ck.gemm_w4a16_gateup_silu(x, g, u, K, mid, ws)
        torch.cuda.synchronize()
        assert ck.gemm_error() == 0 and (buf[:o] == 255).all() and (buf[o + nbytes + 16:] == 255).all()
        out.append((y, h, normed, mid))
    for a, b in ((0, 1), (2, 3)):
        assert all(torch.equal(s, t) for s, t in zip(out[a], out[b]))


def test_prefill_layer_refuses_what_does_not_fit(cuda, orc):
    """Rows on the host, rows of another width, projections of another size: errors as from the separate launches, not a read past the end."""
    from dataclasses import replace

    from nve_b200 import gpu_layer as gl
    from test_gpu_glue import _make_state

    torch = cuda
    hidden, ffn = 512, 1024
    st = _make_state(torch, orc, hidden, ffn, 8, 2, 64, 1, 64, 1045, True)
    x = _x(torch, orc, 4, hidden, 1046)
    assert tuple(gl.gpu_layer_forward_prefill(x, 0, st, 0).shape) == (4, hidden)
    with pytest.raises(ValueError):
        gl.gpu_layer_forward_prefill(x.cpu(), 0, st, 0)
    w = st.layer_weights[0]
    for bad in (dict(o_proj=gl.GpuW4(w.down_proj.nibbles, w.down_proj.scales, None, hidden, ffn)),
                dict(down_proj=gl.GpuW4(w.q_proj.nibbles, w.q_proj.scales, None, hidden, hidden))):
        st.layer_weights[0] = replace(w, **bad)
        with pytest.raises(ValueError):
            gl.gpu_layer_forward_prefill(x, 0, st, 0)
        st.layer_weights[0] = w
    with pytest.raises(ValueError):
        gl.gpu_layer_forward_prefill(_x(torch, orc, 4, hidden // 2, 1046), 0, st, 0)


@pytest.mark.parametrize("S,start,nh,nkv,hd,hidden", [(9, 0, 4, 2, 128, 512), (31, 1, 10, 2, 64, 512), (61, 0, 20, 5, 64, 1088), (257, 40, 6, 3, 128, 1024),
                                                       (300, 3, 8, 2, 64, 1024), (1500, 2, 18, 3, 128, 512)])
def test_prefill_layer_rope_and_cache_write(cuda, orc, S, start, nh, nkv, hd, hidden):
    """The launch that finishes q, k and v rotates them and writes the cache: both GEMM kernels before it, more than one tile of rows, k and
    v narrower than a tile, both head sizes, positions that start inside the cache.  On 148 SMs the tiles of q, k and v are whole (31 rows), cut
    in half (257 and 300 rows, two tiles of rows), cut by runs of two units that end one tile of five and begin the next (61 rows), and some
    whole, some cut by runs of three units over tiles of two (1500 rows).  Against the separate launches."""
    from nve_b200 import gpu_layer as gl
    from test_gpu_glue import _make_state

    torch = cuda
    ffn, max_seq = 768, start + S + 50
    st = _make_state(torch, orc, hidden, ffn, nh, nkv, hd, 1, max_seq, 1070, True)
    x = _x(torch, orc, S, hidden, 1071)
    caches = st.kv_cache.k[0], st.kv_cache.v[0]
    for t in caches:
        t.copy_(_x(torch, orc, nkv * max_seq, hd, 1072).view(nkv, max_seq, hd))
    before = [t.clone() for t in caches]
    got = gl.gpu_layer_forward_prefill(x, 0, st, start)
    mine = [t.clone() for t in caches]
    for t, b in zip(caches, before):
        t.copy_(b)
    w = st.layer_weights[0]
    for p in (w.q_proj, w.k_proj, w.v_proj, w.o_proj, w.gate_proj, w.up_proj, w.down_proj):
        p.awq_scales = torch.ones(p.k, dtype=torch.float32, device="cuda")
    want = gl.gpu_layer_forward_prefill(x, 0, st, start)
    # the bound of test_prefill_layer_equals_separate_launches
    for a, b in ((got, want), (mine[0], caches[0]), (mine[1], caches[1])):
        assert rel_rms_err(a.float().cpu().numpy(), b.float().cpu().numpy()) < 5e-3
    for a, b in zip(mine, before):
        assert torch.equal(a[:, :start], b[:, :start]) and torch.equal(a[:, start + S:], b[:, start + S:])
