"""GPU: the on-device Q4 quantizer bit for bit against the oracle where its rounding and its rare path can go wrong: exact ties
of either sign, values one ulp beside a tie, NaN, infinities, subnormal maxima, block counts around a CTA's 128."""
import numpy as np
import pytest

from helpers import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,awq", [(1, 32, False), (127, 32, True), (128, 32, False), (3, 1376, True), (129, 64, False)])
def test_q4_quantize_edges(cuda, orc, n, k, awq):
    from nve_b200 import cuda_kernels as ck

    rng = np.random.default_rng(n * k)
    b = np.empty((n * k // 32, 32), np.float32)
    ties = np.array([s * (j + 0.5) for j in range(7) for s in (1, -1)], np.float32)
    for i in range(b.shape[0]):
        scale = np.float32(2.0) ** rng.integers(-20, 20)
        b[i] = rng.choice(ties, 32)
        b[i, 8:16] = np.nextafter(b[i, 8:16], np.float32(0))
        b[i, 16:24] = np.nextafter(b[i, 16:24], b[i, 16:24] * 2)
        b[i, rng.integers(32)] = rng.choice([7.0, -7.0])  # scale is then a power of two and ties stay ties
        b[i] *= scale
        kind = i % 9
        if kind == 1:
            b[i, rng.integers(32)] = np.nan
        elif kind == 2:
            b[i, rng.integers(32)] = rng.choice([np.inf, -np.inf])
        elif kind == 3:
            b[i] = rng.choice([0.0, -0.0, 1e-45, -3e-45, 2e-40], 32)
        elif kind == 4:
            b[i] = rng.standard_normal(32)
        elif kind == 5:
            b[i] = 0.0 if i % 2 else np.nan
        elif kind == 6:
            b[i] *= np.float32(1e-31) / scale
    W = b.reshape(n, k)
    f = (np.abs(rng.standard_normal(k)) + 0.1).astype(np.float32) if awq else None
    with np.errstate(all="ignore"):
        en, es = orc.extract_for_gpu(orc.quantize_q4(W if f is None else W * f[None, :]))
    dn, ds = ck.q4_quantize(dev(W), None if f is None else dev(f))
    assert np.array_equal(ds.cpu().numpy().view(np.uint32), es.view(np.uint32))
    assert np.array_equal(dn.cpu().numpy(), en)
