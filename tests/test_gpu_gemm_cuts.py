"""GPU: the batched GEMM where runs are longer than a tile and end inside one: the finishing launch has a block per cut instead of one per
tile, and moves 16-bit values four at a time where rows and addresses allow it."""
import pytest

from helpers import dev, rel_rms_err
from test_gpu_gemm_finish import _weights, _x

pytestmark = pytest.mark.gpu


def _f16_weights(w):
    nib, sc, n = w
    b = nib.view(n, -1, 16)
    q = nib.new_empty((n, b.shape[1], 32)).double()
    q[:, :, :16], q[:, :, 16:] = (b & 15).double() - 8, (b >> 4).double() - 8
    return (q.half() * sc.half()[:, :, None]).view(n, -1).double()


# 33 tiles of weights by three of rows over 74 pairs of SMs: runs of five units over tiles of three, and the like
@pytest.mark.parametrize("M,Ns,K,dtype,shift", [(600, (8200,), 768, "float16", 0), (600, (8200,), 768, "float16", 1), (600, (8200,), 768, "bfloat16", 0),
                                                (513, (8197,), 640, "float16", 0), (130, (21001,), 512, "float16", 0), (700, (4096, 2055, 1300), 1024, "float16", 0),
                                                (64, (21004,), 512, "float32", 0), (17, (24000, 1500), 768, "float16", 0)])
def test_cut_tiles(cuda, orc, M, Ns, K, dtype, shift):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    dt = getattr(torch, dtype)
    x = _x(torch, orc, M, K, 1100).to(torch.bfloat16 if dtype == "bfloat16" else torch.float16)
    ws = [_weights(torch, orc, n, K, 1101 + i)[0] for i, n in enumerate(Ns)]
    outs = [torch.full((M * n + 2,), float("nan"), dtype=dt, device="cuda") for n in Ns]
    views = [o[shift:shift + M * n].view(M, n) for o, n in zip(outs, Ns)]  # shift 1: rows that are not aligned to four values
    scratch = torch.empty(ck.gemm_w4a16_multi_scratch_bytes(M, list(Ns), K), dtype=torch.uint8, device="cuda")
    before = ck.launch_count()
    if M <= 64:
        ck.gemm_w4a16_multi(x, ws, K, out_dtype=dt, outs=views, scratch=scratch)
    else:
        ck.gemm_w4a16_wide(x, ws, K, views, scratch)
    assert ck.launch_count() - before == (3 if dtype == "bfloat16" else 2)  # tiles are cut: a finishing launch (and the conversion of bf16)
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    for o, v, w in zip(outs, views, ws):
        want = x.double() @ _f16_weights(w).t()
        # f32 sums of K products (an MMA may cut off half an ulp on average: 2^-24 K / 16 of the partial sums) and one rounding of the result
        ulp = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8, "float32": 0.0}[dtype]
        assert ((v.double() - want).abs() <= ulp * want.abs() + 1e-4 * want.pow(2).mean().sqrt()).all()
        assert o[:shift].isnan().all() and o[shift + v.numel():].isnan().all()


@pytest.mark.parametrize("M,N,K", [(600, 4100, 768), (300, 6000, 576), (1300, 2050, 512)])
def test_cut_tiles_silu(cuda, orc, M, N, K):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x, g, u = _x(torch, orc, M, K, 1110), _weights(torch, orc, N, K, 1111)[0], _weights(torch, orc, N, K, 1112)[0]
    mid, gate, up = (torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(3))
    before = ck.launch_count()
    ck.gemm_w4a16_gateup_silu(x, g, u, K, mid)
    assert ck.launch_count() - before == 2
    gd, ud = ((x.double() @ _f16_weights(w).t()) for w in (g, u))
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    # half an f16 ulp of each product (|silu'| <= 1.1), of silu(g) * u, and the f32 sums as above
    silu = torch.nn.functional.silu(gd)
    want = silu * ud
    bound = 2.0 ** -11 * 1.01 * (1.1 * gd.abs() * ud.abs() + 2 * silu.abs() * ud.abs()) + 1e-3 * want.pow(2).mean().sqrt()
    assert ((mid.double() - want).abs() <= bound).all()


def test_cut_tiles_add(cuda, orc):
    """The down projection of a prefill layer adds the residual in its finish: eleven by eight tiles, runs of four units over tiles of three."""
    from nve_b200 import gpu_layer as gl
    from test_gpu_glue import _make_state

    torch = cuda
    S, hidden, ffn, nh, nkv, hd = 1901, 2816, 768, 4, 2, 64
    st = _make_state(torch, orc, hidden, ffn, nh, nkv, hd, 1, S + 1, 1120, True)
    x = _x(torch, orc, S, hidden, 1121)
    got = gl.gpu_layer_forward_prefill(x, 0, st, 0)
    w = st.layer_weights[0]
    for p in (w.q_proj, w.k_proj, w.v_proj, w.o_proj, w.gate_proj, w.up_proj, w.down_proj):
        p.awq_scales = torch.ones(p.k, dtype=torch.float32, device="cuda")  # every projection and the add through their own launches
    want = gl.gpu_layer_forward_prefill(x, 0, st, 0)
    # the same f16 values summed in another order where the split over K differs
    assert rel_rms_err(got.float().cpu().numpy(), want.float().cpu().numpy()) < 5e-3
