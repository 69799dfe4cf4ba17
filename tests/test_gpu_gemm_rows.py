"""GPU: the batched GEMM with up to eight rows of x and a workspace (weights straight into registers): ragged rows, columns and
matrices, runs that end inside a tile, K that is no multiple of its units (128), both activation types, every finish; nine
rows take the other kernel.  Against an f64 product of the dequantised weights and the separate launches."""
import pytest

from helpers import dev, rel_rms_err
from test_gpu_gemm_finish import _weights, _x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
@pytest.mark.parametrize("M,Ns,K", [(1, (33,), 64), (2, (257, 255), 192), (7, (40, 600, 256), 1088), (8, (4096,), 14336), (8, (20000,), 448),
                                    (9, (300,), 4096)])
def test_rows_gemm(cuda, orc, M, Ns, K, dt):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x = _x(torch, orc, M, K, 1010).to(getattr(torch, dt))
    ws = [_weights(torch, orc, n, K, 1011 + i) for i, n in enumerate(Ns)]
    scratch = torch.full((ck.gemm_w4a16_multi_scratch_bytes(M, list(Ns), K),), 255, dtype=torch.uint8, device="cuda")  # NaN as f32
    outs = [torch.full((M, n), float("nan"), dtype=x.dtype, device="cuda") for n in Ns]
    ck.gemm_w4a16_wide(x, [t for t, _ in ws], K, outs, scratch)
    for o, (_, w) in zip(outs, ws):
        # largest error over the RMS of the result: f16 rounding of the weights and f32 sums as in the tests of the other sizes
        # (3e-3), and half an ulp of a result of up to five times the RMS
        bound = 3e-3 + 5 * torch.finfo(x.dtype).eps / 2
        assert rel_rms_err(o.float().cpu().numpy(), (x.double() @ w.t()).cpu().numpy()) < bound


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (5, 3072, 1088), (8, 200, 4096)])
def test_rows_gemm_finishes(cuda, orc, M, N, K):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x, (g, wg), (u, wu) = _x(torch, orc, M, K, 1020), _weights(torch, orc, N, K, 1021), _weights(torch, orc, N, K, 1022)
    mid = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    ck.gemm_w4a16_gateup_silu(x, g, u, K, mid)
    a, b = x.double() @ wg.t(), x.double() @ wu.t()
    assert rel_rms_err(mid.float().cpu().numpy(), (a * torch.sigmoid(a) * b).cpu().numpy()) < 1e-2
    res, norm = _x(torch, orc, M, N, 1023), dev(orc.to_act16(1.0 + 0.1 * orc.fill_normal(N, 1024, 3)), torch.float16)
    h, normed = torch.empty_like(res), torch.empty_like(res)
    ck.gemm_w4a16_add_rmsnorm(x, g, K, res, norm, 1e-5, h, normed)
    want = torch.empty_like(res)
    scratch = torch.empty(ck.gemm_w4a16_multi_scratch_bytes(M, [N], K), dtype=torch.uint8, device="cuda")
    ck.gemm_w4a16_wide(x, [g], K, [want], scratch)
    want_n = ck.add_rms_norm_rows(want, res, norm, 1e-5)
    assert torch.equal(h, want) and torch.equal(normed, want_n)
