"""GPU parity: the batched W4A16 GEMM (mma.sync kernel up to 16 batch rows where it has a workspace, tcgen05 kernel otherwise) against the
reference's CPU semantics (q4_linear: one f32 GEMV per row of X, src/quantize.rs:1057-1075) on the same
16-bit-rounded activations."""
import numpy as np
import pytest

from helpers import TOL, dev, rel_rms_err
from oracle import np_oracle as npo

pytestmark = pytest.mark.gpu


def _case(orc, M, N, K, seed, bf):
    W = orc.fill_normal(N * K, seed, 1, scale=0.02).reshape(N, K)
    nib, sc = orc.extract_for_gpu(orc.quantize_q4(W))
    X16 = orc.to_act16(orc.fill_normal(M * K, seed, 2), bf).reshape(M, K)
    Wq = npo.unpack_gpu(nib).astype(np.float64) * np.repeat(sc.astype(np.float64), 32, axis=1)
    ref = orc.from_act16(X16, bf).astype(np.float64) @ Wq.T
    return nib, sc, X16, ref


@pytest.mark.parametrize("M,N,K", [(16, 128, 64), (16, 128, 512), (1, 256, 1024), (8, 384, 2048), (32, 1024, 4096),
                                    (64, 512, 4096), (33, 200, 1024), (64, 4096, 4096), (16, 2048, 14336),
                                    # more tiles than SMs: a CTA's run crosses tile boundaries (partial first and last segments)
                                    (16, 25600, 512), (32, 20480, 1024), (8, 19000, 768),
                                    # narrow batches (the mma.sync kernel): K not a multiple of 256, ragged N, split tiles
                                    (4, 300, 320), (8, 128, 64), (7, 1000, 4096), (2, 19000, 1280)])
@pytest.mark.parametrize("bf", [False, True])
def test_gemm_w4a16_tensor_core(cuda, orc, M, N, K, bf):
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    dt = torch.bfloat16 if bf else torch.float16
    nib, sc, X16, ref = _case(orc, M, N, K, 700 + M + N, bf)
    dx, dn, ds = dev(X16, dt), dev(nib), dev(sc)
    y32 = ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert ck.gemm_error() == 0
    # weights and scales are rounded to the activation type (as the reference dequantises to f16): ~2^-11 (f16)
    # or ~2^-8 (bf16) relative per weight; the f16 path stays far inside the stated tolerance, bf16 inside it
    assert rel_rms_err(y32.cpu().numpy(), ref) < 3e-3
    # the 16-bit output is the f32 accumulator rounded once (for bf16 that rounding alone is ~8e-3 of the RMS at
    # 4 sigma, so the tolerance is judged on the f32 output and the 16-bit output is checked as its rounding)
    y16 = ck.gemm_w4a16(dx, dn, ds, N, K)
    assert torch.equal(y16, y32.to(dt))
    if not bf:
        assert rel_rms_err(y16.float().cpu().numpy(), ref) < TOL
    # with a caller-provided workspace tiles are cut over K between CTAs: same result within f32 reassociation
    nbytes = ck.gemm_w4a16_scratch_bytes(M, N, K)
    if nbytes:
        scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        ys = ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32, scratch=scratch)
        assert rel_rms_err(ys.cpu().numpy(), ref) < 3e-3
        assert ck.gemm_error() == 0


def test_gemm_matches_gemv_rows(cuda, orc):
    """Row m of the batched result equals the batch-1 W4A16 GEMV of row m within tolerance (different arithmetic:
    f16 weights on tensor cores vs the integer path)."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    M, N, K = 16, 1024, 4096
    nib, sc, X16, ref = _case(orc, M, N, K, 801, False)
    dx, dn, ds = dev(X16, torch.float16), dev(nib), dev(sc)
    Y = ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32).cpu().numpy()
    for m in (0, 7, 15):
        y = ck.matvec_w4a16_multi(dx[m].contiguous(), None, [(dn, ds, N)], K, out_dtype=torch.float32)[0].cpu().numpy().reshape(-1)
        assert rel_rms_err(Y[m], y) < 3e-3


@pytest.mark.parametrize("M,Ns,K", [(16, (4096, 1024, 1024), 4096), (8, (256, 128), 512), (64, (1024, 1000, 40), 1024),
                                     (8, (12800, 12864), 512)])
def test_gemm_multi_matrix_equals_single_calls(cuda, orc, M, Ns, K):
    """q/k/v (or gate/up) in one launch: same numbers as one call per matrix without a workspace, and within f32
    reassociation of them when the workspace lets the runs of the CTAs cut tiles (also across the matrices)."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    X16 = orc.to_act16(orc.fill_normal(M * K, 950, 2)).reshape(M, K)
    dx = dev(X16, torch.float16)
    ws, singles = [], []
    for i, N in enumerate(Ns):
        nib, sc, _, _ = _case(orc, M, N, K, 960 + i, False)
        dn, ds = dev(nib), dev(sc)
        ws.append((dn, ds, N))
        singles.append(ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32))
    outs = ck.gemm_w4a16_multi(dx, ws, K, out_dtype=torch.float32)
    for y, want in zip(outs, singles):
        assert torch.equal(y, want)
    scratch = torch.empty(ck.gemm_w4a16_multi_scratch_bytes(M, Ns, K), dtype=torch.uint8, device="cuda")
    outs = ck.gemm_w4a16_multi(dx, ws, K, out_dtype=torch.float32, scratch=scratch)
    for y, want in zip(outs, singles):
        assert rel_rms_err(y.cpu().numpy(), want.cpu().numpy()) < 1e-5
    outs16 = ck.gemm_w4a16_multi(dx, ws, K, scratch=scratch)
    for y16, y in zip(outs16, outs):
        assert torch.equal(y16, y.to(torch.float16))
    assert ck.gemm_error() == 0


def test_gemm_rejects_bad_arguments(cuda):
    from nve_b200 import _ffi
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    x = torch.zeros((65, 64), dtype=torch.float16, device="cuda")
    nib = torch.zeros((128, 32), dtype=torch.uint8, device="cuda")
    sc = torch.zeros((128, 2), dtype=torch.float32, device="cuda")
    with pytest.raises(_ffi.NveKernelError):
        ck.gemm_w4a16(x, nib, sc, 128, 64)  # M > 64
    with pytest.raises(_ffi.NveKernelError):
        ck.gemm_w4a16(x[:8, :32].contiguous(), nib, sc, 128, 32)  # K % 64 != 0


@pytest.mark.parametrize("M", [1, 5, 64, 100, 130, 300])
@pytest.mark.parametrize("with_awq", [False, True])
def test_matmul_x_matches_q4_linear(cuda, orc, M, with_awq):
    """gpu_layer.matmul_x (the batch > 1 call site: GEMV at M == 1, the packed GEMM for any number of rows)
    against the reference's CPU semantics q4_linear on the same 16-bit activations."""
    from nve_b200.gpu_layer import GpuW4, matmul_x

    torch = cuda
    N, K = 768, 2048
    W = orc.fill_normal(N * K, 931, 1, scale=0.02).reshape(N, K)
    blocks = orc.quantize_q4(W)
    nib, sc = orc.extract_for_gpu(blocks)
    awq = (0.5 + np.abs(orc.fill_normal(K, 931, 3))).astype(np.float32) if with_awq else None
    X16 = orc.to_act16(orc.fill_normal(M * K, 931, 2)).reshape(M, K)
    w = GpuW4(dev(nib), dev(sc), None if awq is None else dev(awq), N, K)
    y = matmul_x(dev(X16, torch.float16), w)
    assert tuple(y.shape) == (M, N)
    ref = orc.q4_linear(blocks, orc.from_act16(X16), awq_inv=awq)
    assert rel_rms_err(y.float().cpu().numpy(), ref) < TOL


def test_matmul_x_dense_route_bf16(cuda, orc):
    """bf16 activations above 128 rows: converted to f16 for the GEMM, the result rounded to bf16 once (judged on the f32 reference within bf16's own rounding)."""
    from nve_b200.gpu_layer import DENSE_ROWS, GpuW4, matmul_x

    torch = cuda
    M, N, K = DENSE_ROWS + 72, 512, 1024
    nib, sc, X16, ref = _case(orc, M, N, K, 977, True)
    w = GpuW4(dev(nib), dev(sc), None, N, K)
    y = matmul_x(dev(X16, torch.bfloat16), w)
    assert y.dtype == torch.bfloat16 and tuple(y.shape) == (M, N)
    yf = y.float().cpu().numpy().astype(np.float64)
    rms = np.sqrt(np.mean(ref * ref))
    assert np.all(np.abs(yf - ref) <= np.abs(ref) * 2.0 ** -8 + 3e-3 * rms)  # half a bf16 ulp + the f16 GEMM's tolerance
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    assert matmul_x(dev(X16, torch.bfloat16), w, out=out) is out
    assert torch.equal(out, y)


@pytest.mark.parametrize("form", ["k32", "f32", "strided", "offset", "nibbles", "out_strided", "out_f32", "out_bf16", "small_scratch", "awq_k32"])
def test_matmul_x_forms_above_128_rows(cuda, orc, form):
    """What the packed GEMM does not take: K % 64 == 32, f32 or strided or unaligned x, unaligned nibbles, strided or other outputs,
    a workspace made for 64 rows."""
    from nve_b200 import cuda_kernels as ck
    from nve_b200.gpu_layer import GpuW4, matmul_x, matmul_x_multi

    torch = cuda
    M, N, K = 150, 264, 288 if form.endswith("k32") else 512
    nib, sc, X16, _ = _case(orc, M, N, K, 983, False)
    x, dn, awq, out, scratch = dev(X16, torch.float16), dev(nib), None, None, None
    if form == "f32":
        x = x.float()
    elif form == "strided":
        x = torch.cat([x, x], 1)[:, :K]
    elif form == "offset":
        x = torch.cat([x.flatten()[:1], x.flatten()])[1:].view(M, K)
    elif form == "nibbles":
        dn = torch.cat([dn.flatten()[:1], dn.flatten()])[1:].view(N, K // 2)
    elif form == "out_strided":
        out = torch.full((M, 2 * N), float("nan"), dtype=torch.float16, device="cuda")[:, ::2]
    elif form.startswith("out_"):
        out = torch.full((M, N), float("nan"), dtype=torch.float32 if form == "out_f32" else torch.bfloat16, device="cuda")
    elif form == "small_scratch":
        x = x.bfloat16()
        scratch = torch.empty(ck.gemm_w4a16_scratch_bytes(64, N, K), dtype=torch.uint8, device="cuda")
    elif form == "awq_k32":
        awq = dev((0.5 + np.abs(orc.fill_normal(K, 983, 3))).astype(np.float32))
    w = GpuW4(dn, dev(sc), awq, N, K)
    Wq = npo.unpack_gpu(nib).astype(np.float64) * np.repeat(sc.astype(np.float64), 32, axis=1)
    ref = (x.double() if awq is None else x.double() * awq.double()).cpu().numpy() @ Wq.T
    # weights and x * multiplier rounded to f16 (3e-3 of the RMS at most), and the rounding of results of up to ten times the RMS
    bound = 3e-3 + 5 * torch.finfo(torch.bfloat16 if form in ("out_bf16", "small_scratch") else torch.float16).eps
    for got in (matmul_x(x, w, scratch, out), matmul_x_multi(x, [w] * 2, scratch, None if out is None else [out] * 2)[1]):
        assert got is out or (out is None and got.dtype == x.dtype)
        assert tuple(got.shape) == (M, N) and rel_rms_err(got.float().cpu().numpy(), ref) < bound
    got = matmul_x_multi(x, [w] * 4, scratch)  # more than one launch takes
    assert len(got) == 4 and rel_rms_err(got[3].float().cpu().numpy(), ref) < bound


def test_matmul_x_of_a_workspace_for_64_rows_and_of_no_rows(cuda, orc):
    """Up to 128 rows a workspace made for 64 serves them in slices, with nothing allocated; zero rows give an empty result."""
    from nve_b200 import cuda_kernels as ck
    from nve_b200.gpu_layer import GpuW4, matmul_x, matmul_x_multi

    torch = cuda
    M, N, K = 100, 520, 1024
    for dt in (torch.float16, torch.bfloat16):
        nib, sc, X16, ref = _case(orc, M, N, K, 987, dt == torch.bfloat16)
        w, x = GpuW4(dev(nib), dev(sc), None, N, K), dev(X16, dt)
        scratch = torch.full((ck.gemm_w4a16_multi_scratch_bytes(64, [N, N], K) + 64,), 255, dtype=torch.uint8, device="cuda")
        out = [torch.full((M, N), float("nan"), dtype=dt, device="cuda") for _ in range(2)]
        before = torch.cuda.memory_allocated()
        assert matmul_x(x, w, scratch[:-64], out[0]) is out[0]
        assert all(a is b for a, b in zip(matmul_x_multi(x, [w, w], scratch[:-64], out), out))
        torch.cuda.synchronize()
        assert torch.cuda.memory_allocated() == before and (scratch[-64:] == 255).all()
        for o in out:
            assert rel_rms_err(o.float().cpu().numpy(), ref) < 3e-3 + 5 * torch.finfo(dt).eps
        assert tuple(matmul_x(x[:0], w).shape) == (0, N) and matmul_x(x[:0], w).dtype == dt
        assert [tuple(t.shape) for t in matmul_x_multi(x[:0], [w, w])] == [(0, N)] * 2


@pytest.mark.parametrize("M,N,K,one", [(1, 256, 64, False), (3, 300, 320, False), (8, 384, 2048, False), (7, 1000, 4096, False), (2, 19000, 1280, False),
                                        (5, 40000, 128, False), (9, 1000, 4096, False), (16, 384, 2048, False), (9, 2000, 512, True),
                                        (16, 300, 320, True), (13, 257, 7168, False), (17, 384, 2048, False)])
def test_few_rows_on_each_kernel(cuda, orc, M, N, K, one):
    """Up to sixteen rows: the kernel for few rows (two launches: it always leaves partial tiles) where the workspace holds its partial tiles,
    else the two-SM kernel, in whole tiles (one launch) where the workspace holds nothing.  `one`: nine rows or more of f16 on one tile per
    pair of SMs stay on the two-SM kernel.  bf16 rows tell the two apart: the two-SM kernel has them converted first."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    for bf in (False, True):
        nib, sc, X16, ref = _case(orc, M, N, K, 990, bf)
        dx, dn, ds = dev(X16, torch.bfloat16 if bf else torch.float16), dev(nib), dev(sc)
        full = torch.empty(ck.gemm_w4a16_scratch_bytes(M, N, K), dtype=torch.uint8, device="cuda")
        for scratch, launches in ((full, 2 if M <= 16 else 3),) if bf else ((None, 1), (full[:16], 1), (full, 1 if one else 2)):
            out = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")
            before = ck.launch_count()
            ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32, out=out, scratch=scratch)
            assert ck.launch_count() - before == launches
            torch.cuda.synchronize()
            assert ck.gemm_error() == 0
            assert rel_rms_err(out.cpu().numpy(), ref) < 3e-3  # f16 rounding of the weights, as above


@pytest.mark.parametrize("M", [8, 9])
def test_bf16_rows_without_room_for_their_copy(cuda, orc, M):
    """Up to eight bf16 rows are taken where the workspace holds the partial tiles, though it has no room for an f16 copy; more are refused."""
    from nve_b200 import _ffi
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    N, K = 64, 81920  # the copy is larger than the partial tiles of one tile of weights
    x = dev(orc.to_act16(orc.fill_normal(M * K, 991, 2), True), torch.bfloat16).view(M, K)
    nib, sc = dev(np.full((N, K // 2), 0x99, np.uint8)), dev(np.full((N, K // 32), 0.01, np.float32))  # every weight 0.01
    scratch = torch.empty(M * K * 2 - 16, dtype=torch.uint8, device="cuda")
    if M > 8:
        with pytest.raises(_ffi.NveKernelError):
            ck.gemm_w4a16(x, nib, sc, N, K, out_dtype=torch.float32, scratch=scratch)
        return
    y = ck.gemm_w4a16(x, nib, sc, N, K, out_dtype=torch.float32, scratch=scratch).double()
    want = x.double().sum(1, keepdim=True).expand(M, N) * float(np.float16(0.01))
    # f32 sums of 81920 terms against a sum that is their square root times as large: 2^-24 * sqrt(81920) / 16 of it at most
    assert float((y - want).abs().max()) < 1e-5 * float(x.double().norm(dim=1).max()) * 0.01


def _sums_error(N, K, sets, pairs):
    """Expected error of the f32 sums over K, relative to the result.  An MMA (16 elements of K) rounds its accumulator towards zero, by half
    an ulp on average: 2^-24 / (2 ln 2) of a sum with an even exponent distribution.  The sum after j of c MMAs is on average j / c of what
    the chain ends with, which is thus (c + 1) / 2 times that too small.  `sets` chains share the steps (eight MMAs) of a segment; segments are
    where the runs of two-SM pairs (units of two steps) cut a tile of 256 rows."""
    units, tiles = -(-K // 256), -(-N // 256)
    run = max(2, -(-tiles * units // pairs))
    total = 0.0
    for t in range(0, tiles * units, units):
        cuts = sorted({t, t + units} | set(range(-(-t // run) * run, t + units, run)))
        for a, b in zip(cuts, cuts[1:]):
            chains = [8 * len(range(w, 2 * (b - a), sets)) for w in range(sets)]
            total += sum(c * (c + 1) / 2 for c in chains) / (16 * units * tiles)
    return 2.0**-24 / (2 * np.log(2)) * total


@pytest.mark.parametrize("M,N,K", [(1, 512, 2048), (4, 40000, 1024), (8, 4096, 14336), (9, 2048, 4096), (16, 4096, 4096),
                                    (17, 4096, 4096), (32, 1024, 14336), (61, 2048, 2048), (64, 14336, 4096)])
def test_sums_over_k(cuda, orc, M, N, K):
    """f32 results against an f64 product of the weights as the kernel has them (f16), which leaves the error of the sums: three accumulator
    sets from 17 to 64 rows (two are 1.3 to 1.5 times further off); up to sixteen rows chains of eight MMAs, added up with K / 128 roundings to
    nearest (of one ulp / sqrt(12) each, of a sum that grows with the square root of their number).  A tenth for the spread."""
    from nve_b200 import cuda_kernels as ck

    torch = cuda
    nib, sc, X16, _ = _case(orc, M, N, K, 992, False)
    dx, dn, ds = dev(X16, torch.float16), dev(nib), dev(sc)
    y = ck.gemm_w4a16(dx, dn, ds, N, K, out_dtype=torch.float32,
                      scratch=torch.empty(ck.gemm_w4a16_scratch_bytes(M, N, K), dtype=torch.uint8, device="cuda"))
    b = dn.view(N, K // 32, 16)
    q = torch.cat([(b & 15).half() - 8, (b >> 4).half() - 8], dim=2)
    want = dx.double() @ (q * ds.half()[:, :, None]).view(N, K).double().t()
    if M <= 16:
        ulp = 2.0**-23 / (2 * np.log(2))
        bound = np.hypot(ulp / 2 * 4.5, ulp / np.sqrt(12) * np.sqrt(K / 256))
    else:
        bound = _sums_error(N, K, 3, torch.cuda.get_device_properties(0).multi_processor_count // 2)
    assert float((y.double() - want).norm() / want.norm()) < 1.1 * bound
