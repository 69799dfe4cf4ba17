"""GPU: q, k and v projections of a batch and its attention in two launches (the attention sums the segments of the product) against the two
calls, bit for bit."""
import pytest

from helpers import dev, rel_rms_err
from test_gpu_gemm_finish import _weights, _x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cuda_core", [False, True])
@pytest.mark.parametrize("B,nh,nkv,hd,K,scratch", [
    (2, 24, 8, 128, 3072, True),    # three heads per KV head, runs of two units over tiles of twelve: six segments
    (7, 12, 4, 64, 512, True),
    (8, 8, 8, 128, 2048, True),     # one head per KV head
    (16, 16, 2, 64, 4096, True),    # eight heads
    (17, 32, 8, 128, 4096, True),   # the two-SM kernel, some tiles cut
    (64, 8, 2, 128, 256, True),     # whole tiles, nothing to sum
    (64, 10, 2, 64, 1088, False),   # a workspace without room for partial tiles
    (100, 20, 4, 128, 1024, True),  # more than 64 rows
    (300, 4, 2, 64, 1024, True),    # two tiles of rows: finished by the GEMM
    (3, 24, 2, 64, 768, True),      # twelve heads per KV head: the CUDA-core kernel
    (1, 8, 2, 64, 768, True),
])
def test_equals_the_two_calls(cuda, orc, B, nh, nkv, hd, K, scratch, cuda_core):
    equals_the_two_calls(cuda, orc, B, nh, nkv, hd, K, scratch, cuda_core, 150, [(37 * b + 3) % 150 for b in range(B)])


@pytest.mark.parametrize("B,nh,nkv,hd,K,max_seq", [
    (2, 24, 8, 128, 1024, 2000),   # clusters of seven or eight CTAs
    (5, 32, 8, 64, 1024, 2000),    # of several, two CTAs per SM
    (9, 24, 8, 64, 512, 900),
    (13, 40, 8, 128, 512, 700),    # five heads per KV head
    (5, 64, 8, 64, 512, 1500),     # eight
    (2, 32, 8, 64, 1024, 600),     # finished first: few units of small heads in a large cache
    (70, 32, 8, 64, 512, 300),     # four warps per unit
    (60, 64, 8, 128, 512, 200),
    (57, 8, 8, 64, 512, 100),      # the same with heads of 64: one and four heads per KV head are left to the attention, five are finished
    (57, 40, 8, 64, 512, 100),
])
def test_equals_the_two_calls_in_large_caches(cuda, orc, B, nh, nkv, hd, K, max_seq):
    equals_the_two_calls(cuda, orc, B, nh, nkv, hd, K, True, False, max_seq, [max_seq - 1 - 173 * b % max_seq for b in range(B)])  # the first to its end


def equals_the_two_calls(cuda, orc, B, nh, nkv, hd, K, scratch, cuda_core, max_seq, positions):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x = _x(torch, orc, B, K, 1201)
    Ns = [nh * hd, nkv * hd, nkv * hd]
    ws = [_weights(torch, orc, n, K, 1202 + i)[0] for i, n in enumerate(Ns)]
    kc, vc = (dev(orc.to_act16(orc.fill_normal(B * nkv * max_seq * hd, 1206, i)), torch.float16).view(B, nkv, max_seq, hd) for i in range(2))
    cos, sin = (dev(orc.to_act16(t), torch.float16) for t in orc.rope_tables_f32(hd, max_seq, 10000.0))
    d_pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
    d_len = d_pos + 1
    nbytes = ck.gemm_w4a16_multi_scratch_bytes(B, Ns, K) if scratch else 16
    buf = lambda: [torch.full((B, n), float("nan"), dtype=torch.float16, device="cuda") for n in Ns]
    space = torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda")
    with ck.attn_decode_kernel(cuda_core):
        q, k, v = ck.gemm_w4a16_wide(x, ws, K, buf(), space)
        k1, v1 = kc.clone(), vc.clone()
        want = ck.attn_decode_fused_batch(q, k, v, k1, v1, cos, sin, d_pos, d_len, nh, nkv, hd, max_seq, hd ** -0.5)
        k2, v2, got = kc.clone(), vc.clone(), torch.full_like(want, float("nan"))
        space.fill_(255)
        ck.qkv_attn_decode_batch(x, ws, K, buf(), space, k2, v2, cos, sin, d_pos, d_len, nh, nkv, hd, max_seq, hd ** -0.5, got)
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    assert torch.equal(got, want) and torch.equal(k1, k2) and torch.equal(v1, v2)
    assert not torch.equal(k1, kc)


def test_refuses_what_does_not_fit(cuda, orc):
    from nve_b200 import _ffi, cuda_kernels as ck

    torch = cuda
    x, ws = _x(torch, orc, 4, 512, 1210), [_weights(torch, orc, n, 512, 1211 + i)[0] for i, n in enumerate((512, 128, 128))]
    z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")
    outs, space, d = [z(4, n) for n in (512, 128, 128)], torch.empty(1 << 22, dtype=torch.uint8, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    run = lambda nh, nkv, hd, B=4: ck.qkv_attn_decode_batch(x, ws, 512, outs, space, z(B, nkv, 8, hd), z(B, nkv, 8, hd), z(8, hd // 2), z(8, hd // 2), d, d + 1, nh, nkv,
                                                            hd, 8, 0.1, z(4, nh * hd))
    run(8, 2, 64)
    for args in ((4, 2, 64), (8, 1, 64), (8, 2, 32)):
        with pytest.raises(_ffi.NveKernelError):
            run(*args)
    with pytest.raises(ValueError):
        run(8, 2, 64, B=3)


@pytest.mark.parametrize("what", ["nibbles", "scales"])
def test_many_rows_of_what_the_gemm_does_not_take(cuda, orc, what):
    """Above 128 sequences q, k and v weights off their boundaries go the dense way, as they do in matmul_x_multi."""
    from nve_b200.gpu_layer import BatchedDecodeScratch, BatchedKvCache, gpu_layer_forward_decode_batch
    from test_gpu_glue import _make_state

    torch = cuda
    B, hidden, ffn, nh, nkv, hd, max_seq = 130, 512, 768, 8, 2, 64, 40
    st = _make_state(torch, orc, hidden, ffn, nh, nkv, hd, 1, max_seq, 1220, True)
    x = _x(torch, orc, B, hidden, 1221)
    d_pos = torch.tensor([(7 * b + 1) % max_seq for b in range(B)], dtype=torch.int32, device="cuda")
    rows = dev(orc.to_act16(orc.fill_normal(2 * B * nkv * max_seq * hd, 1222, 1)), torch.float16).view(2, B, nkv, max_seq, hd)
    results = []
    for shifted in (False, True):
        if shifted:
            for p in (st.layer_weights[0].q_proj, st.layer_weights[0].v_proj):
                t = getattr(p, what)
                room = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
                off = 8 if what == "nibbles" else 1
                setattr(p, what, room[off:off + t.numel()].view(t.shape).copy_(t))
                assert getattr(p, what).data_ptr() % (16 if what == "nibbles" else 8) != 0
        kv = BatchedKvCache([rows[0].clone()], [rows[1].clone()], B, max_seq)
        scratch = BatchedDecodeScratch.make(st, B, hidden, ffn)
        out = gpu_layer_forward_decode_batch(x.clone(), 0, st, kv, d_pos, d_pos + 1, scratch)
        results.append((out.clone(), kv.k[0], kv.v[0]))
    for a, b in zip(*results):
        # the same f16 weights in another product: roundings (half an f16 ulp, 2.4e-4) of q, k, v and of the launches behind that may fall the other way
        assert rel_rms_err(b.float().cpu().numpy(), a.float().cpu().numpy()) < 2e-3
