"""The memory that prompt slices decode a matrix into: its size before anything is loaded, and the boot plan that counts it or does without."""
import dataclasses

import pytest

from rexl3_b200.models import dense, hybrid, moe
from rexl3_b200.server import main

GB = 1 << 30


def test_size_from_configs():
    front = 4096 * 4 + 74 * 256 * 256 * 4                      # counters and handed accumulators
    big = dense.CONFIGS["dense-27b"]
    assert dense.DenseGPU.prefill_workspace_bytes(big, 8192) == front + 2 * big.d_model * 2 * big.ffn_padded
    assert dense.DenseGPU.prefill_workspace_bytes(big, 64) == 0                                  # a window's rows take other kernels
    assert dense.DenseGPU.prefill_workspace_bytes(dataclasses.replace(big, bits=3.0), 8192) == 0  # other code widths, too
    gdn = hybrid.CONFIGS["gdn-hybrid-27b"]
    widest = max(2 * gdn.ffn_padded, gdn.gdn_proj_width)
    assert hybrid.HybridGPU.prefill_workspace_bytes(gdn, 8192) == front + 2 * max(gdn.d_model * widest, gdn.ffn_padded * gdn.d_model)
    experts = dataclasses.replace(dense.CONFIGS["moe-spec-30b"], bits=4.0)
    assert moe.MoEGPU.prefill_workspace_bytes(experts, 8192) <= front + 2 * experts.d_model * max(experts.qkv_width, experts.n_q * experts.head_dim)


def test_size_from_host_weights():
    cfg = dense.CONFIGS["test-hd128"]
    w = dense.random_weights(cfg)
    most = dense.DenseGPU.prefill_workspace_bytes(dataclasses.replace(cfg, bits=4.0), 1 << 20)
    have = dense.DenseGPU.prefill_workspace_bytes(w, 1 << 20)
    assert have == (most if w.layers[0].gate_up.trellis.shape[2] == 64 else 0)


def test_plan_counts_the_workspace_or_does_without():
    adm, kept = main.plan_memory(20 * GB, 10 * GB, 1 << 20, 4096, GB, 4, 1024, 4096)               # 20 - 1 - 10 - 2: 7 GB for 4 of KV and 1
    assert kept and adm.capacity == 6 * GB
    adm, kept = main.plan_memory(20 * GB, 10 * GB, 1 << 20, 6656, GB, 4, 1024, 6656)               # 6.5 of 7 GB are KV
    assert not kept and adm.capacity == 7 * GB
    with pytest.raises(RuntimeError, match="memory plan refused"):
        main.plan_memory(20 * GB, 10 * GB, 1 << 20, 7 * 1024 + 1, GB, 4, 1024, 7 * 1024 + 1)
    adm, kept = main.plan_memory(20 * GB, 10 * GB, 1 << 20, 7 * 1024, 0, 4, 1024, 7 * 1024)        # nothing to keep
    assert kept and adm.capacity == 7 * GB


@pytest.mark.parametrize("K,N,rows,form,tile_us,wide_us", [
    (8192, 8192, 900, "plain", 121, 151), (17408, 5120, 1650, "plain", 273, 322), (4096, 28672, 300, "plain", 119, 138), (17408, 5120, 1650, "swiglu", 299, 335),
    (12288, 4096, 2048, "store", 194, 222), (512, 6144, 3072, "store", 69, 47), (4096, 18432, 1280, "store", 232, 197), (5120, 34816, 2048, "swiglu", 850, 657),
    (17408, 5120, 2048, "plain", 391, 317), (1024, 4096, 4096, "store", 75, 57),
])
def test_slices_go_where_they_were_measured_faster(K, N, rows, form, tile_us, wide_us):
    """Times on a B200 of the kernel that decodes a matrix per tile of rows (and the finish kernel of the form) and of the one that decodes it once."""
    from rexl3_b200.ops import kernels as KK
    assert KK.wide_takes_shape(rows, K, N, form == "swiglu", form == "store") == (wide_us < tile_us)
