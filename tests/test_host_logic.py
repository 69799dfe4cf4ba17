"""CPU: host-side logic of the call sites (routing, normalisation) against the oracle restatement."""
import os
import re

import numpy as np
import pytest

from nve_b200.gpu_layer import RoutingConfig, normalize_importance


def test_routing_matches_oracle(orc, golden):
    scores = golden["r_scores"]
    norm = normalize_importance(list(scores))
    assert np.array_equal(np.array(norm), golden["r_norm"])
    for thr in (0.0, 0.3, 0.5, 0.7, 1.0):
        cfg = RoutingConfig(False, thr)
        for v in norm:
            assert cfg.use_w4a8(v) == orc.use_w4a8(v, thr, False)
    assert not any(RoutingConfig(True, 0.7).use_w4a8(v) for v in norm)


def test_routing_env_semantics():
    """src/gpu_layer.rs:1017-1025: NVE_NO_W4A8 set (any value) forces W4A16; threshold default 0.7; a value
    that does not parse falls back to the default."""
    assert RoutingConfig.from_env({}).threshold == 0.7 and not RoutingConfig.from_env({}).no_w4a8
    assert RoutingConfig.from_env({"NVE_NO_W4A8": ""}).no_w4a8
    assert RoutingConfig.from_env({"NVE_W4A8_THRESHOLD": "0.25"}).threshold == 0.25
    assert RoutingConfig.from_env({"NVE_W4A8_THRESHOLD": "abc"}).threshold == 0.7
    # importance 0.0 (no profile) selects W4A8, as the benchmark harness of the reference relies on
    assert RoutingConfig().use_w4a8(0.0)


def test_top_half_threshold_is_the_median(golden):
    """'Top 50% of the scores -> W4A16' is the predicate importance < threshold with the threshold at the
    16th largest normalised score."""
    norm = sorted(golden["r_norm"])
    thr = norm[len(norm) // 2]
    cfg = RoutingConfig(False, float(thr))
    routes = [cfg.use_w4a8(float(v)) for v in golden["r_norm"]]
    assert sum(routes) == len(routes) // 2


def test_degenerate_scores():
    assert normalize_importance([2.0, 2.0]) == [0.5, 0.5]
    assert normalize_importance([1.0, 3.0]) == [0.0, 1.0]


def test_pair_gemm_roles_wait_on_bounded_barriers_only():
    """A warp of the two-SM GEMM whose wait expires leaves for the end of the kernel.  Its siblings must get there too: between set-up and
    teardown no role may stand at a barrier of the whole group, which a warp that left never reaches."""
    path = os.path.join(os.path.dirname(__file__), "..", "nve_b200", "csrc", "gemm_w4a16_pair.cu")
    with open(path) as fh:
        kernel = fh.read().split("gemm_w4a16_pair_kernel(const PairParams p", 1)[1]
    loaders, rest = kernel.split("raw loaders (weights", 1)[1].split("tcgen05.alloc", 1)
    roles = rest.split("pg_cluster_wait();", 1)[1].split("// ---- teardown", 1)[0]
    for part in (loaders, roles):
        assert "pg_wait(" in part  # the split above still finds the roles
        assert not re.search(r"\bbar(rier)?\.(cta\.)?(sync|arrive|red)|__syncthreads|__barrier", part)


@pytest.mark.parametrize("wrong,words", [
    (dict(x=(4, 256)), "x must be"), (dict(x=(4, 1, 512)), "x must be"), (dict(k_dim=1024), "x must be"),
    (dict(drop=True), "three matrices"), (dict(outs=((4, 512), (4, 128))), "three matrices"), (dict(outs=((4, 512), (4, 128), (3, 128))), "three matrices"),
    (dict(k=(3, 2, 8, 64)), "one cache"), (dict(v=(4, 2, 7, 64)), "one cache"), (dict(pos=3), "one cache"), (dict(out=(4, 256)), "out must be"),
    (dict(), "CUDA tensor"),  # nothing wrong but that there is no GPU
])
def test_qkv_attn_decode_batch_refuses_shapes_that_do_not_fit(wrong, words):
    """Before any address is taken: a matrix too few or a row too short would be read past its end."""
    import torch

    from nve_b200 import cuda_kernels as ck

    z = lambda *s: torch.zeros(s, dtype=torch.float16)
    ws = [(torch.zeros((n, 256), dtype=torch.uint8), torch.zeros((n, 16)), n) for n in (512, 128, 128)]
    d = torch.zeros(wrong.get("pos", 4), dtype=torch.int32)
    with pytest.raises(ValueError, match=words):
        ck.qkv_attn_decode_batch(z(*wrong.get("x", (4, 512))), ws[:2] if wrong.get("drop") else ws, wrong.get("k_dim", 512),
                                 [z(*s) for s in wrong.get("outs", ((4, 512), (4, 128), (4, 128)))], torch.empty(64, dtype=torch.uint8),
                                 z(*wrong.get("k", (4, 2, 8, 64))), z(*wrong.get("v", (4, 2, 8, 64))), z(8, 32), z(8, 32), d, d, 8, 2, 64, 8, 0.125,
                                 z(*wrong.get("out", (4, 512))))
