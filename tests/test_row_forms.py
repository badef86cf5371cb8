"""Where the row kernels of prompt slices (eight lanes a 128-block) take over from the forms of few rows: measured points, us on a B200 (few rows' form, slices' form)."""
import pytest

from rexl3_b200.ops import lib


@pytest.mark.parametrize("M,N,few,rows", [(149, 4224, 9.5, 6.9), (149, 1152, 5.5, 6.0), (296, 2048, 6.0, 6.4), (297, 2048, 8.1, 7.0), (511, 2048, 10.3, 7.2),
                                          (512, 1152, 5.7, 6.9), (592, 2048, 6.4, 7.6), (593, 2048, 8.5, 7.6), (296, 4096, 7.1, 8.2), (592, 4096, 10.3, 8.5),
                                          (8192, 5120, 152.5, 89.9)])
def test_residual_finish(M, N, few, rows):
    assert lib.load().rx_add_norm_rot_by_rows(M, N) == (rows < few)


@pytest.mark.parametrize("M,n_q,n_kv,few,lanes", [(593, 1, 1, 3.2, 3.9), (800, 4, 1, 3.7, 4.3), (900, 4, 1, 4.6, 4.4), (593, 8, 2, 4.8, 4.4), (593, 40, 8, 11.1, 8.3),
                                                  (300, 40, 8, 13.1, 16.3), (800, 4, 2, 4.0, 4.4), (8192, 1, 1, 13.1, 12.1)])
def test_qkv_finish(M, n_q, n_kv, few, lanes):
    assert lib.load().rx_qkv_rope_by_lanes(M, n_q, n_kv) == (lanes < few)


@pytest.mark.parametrize("rows,K,few,lanes", [(1024, 1024, 3.1, 3.3), (256, 4096, 2.5, 3.4), (296, 5120, 3.0, 3.6), (297, 5120, 4.7, 3.6), (128, 8192, 3.6, 3.4),
                                              (2048, 1024, 4.3, 4.1), (8192, 4096, 32.9, 27.3), (200, 16384, 5.8, 4.9)])
def test_plain_rotation(rows, K, few, lanes):
    assert lib.load().rx_rot_in_by_lanes(rows, K) == (lanes < few)


@pytest.mark.parametrize("rows,topk,d,few,lanes", [(256, 8, 2048, 6.6, 9.8), (450, 8, 2048, 9.5, 11.2), (800, 8, 2048, 15.1, 12.0), (160, 3, 4096, 4.6, 5.1),
                                                   (200, 3, 4096, 5.1, 4.2), (64, 2, 6144, 5.0, 3.6), (64, 1, 7168, 5.9, 2.9), (700, 1, 7168, 8.0, 8.3),
                                                   (3000, 1, 4096, 13.6, 16.1), (74, 4, 5120, 4.4, 5.0), (3000, 8, 2048, 56.2, 37.1)])
def test_routed_gather(rows, topk, d, few, lanes):
    assert lib.load().rx_moe_gather_by_rows(rows * topk, topk, d) == (lanes < few)


@pytest.mark.parametrize("pairs,F,few,lanes", [(2048, 768, 8.2, 7.6), (2400, 768, 8.6, 9.4), (1800, 1024, 8.5, 9.4), (4800, 768, 14.5, 14.3), (24000, 768, 63.8, 56.3),
                                               (1200, 1408, 11.6, 7.6)])
def test_routed_swiglu(pairs, F, few, lanes):
    assert lib.load().rx_moe_swiglu_by_rows(pairs, F) == (lanes < few)


@pytest.mark.parametrize("pairs,experts,N,low,tall", [(1600, 8, 1024, 14, 18), (1024, 8, 1024, 13, 17), (2400, 8, 1024, 23, 18), (800, 8, 28672, 421, 344), (1600, 16, 2048, 50, 44),
                                                      (16800, 128, 1536, 248, 190), (8800, 128, 1536, 158, 162), (10400, 128, 1536, 158, 156)])
def test_expert_tiles(pairs, experts, N, low, tall):
    from rexl3_b200.models.moe import tall_tiles
    assert tall_tiles(pairs, experts, N) == (tall < low)
