"""Decode windows go by the GEMM of equal shares where a dense model's layer was measured faster with it: us a layer on a B200 (by whole items, by equal shares)."""
import pytest

from rexl3_b200.ops import lib


@pytest.mark.parametrize("rows,K,N,items,shares", [
    (1, 4096, 28672, 88.1, 84.9), (32, 4096, 28672, 100.8, 100.3), (1, 4608, 24576, 93.6, 85.5), (17, 4608, 24576, 100.4, 98.1), (1, 4096, 22016, 89.4, 84.5),
    (16, 4096, 22016, 101.9, 105.2), (32, 4096, 22016, 113.0, 118.9), (1, 2560, 19456, 60.0, 66.0), (32, 2560, 19456, 74.3, 86.6), (1, 2048, 20480, 53.8, 57.5),
    (16, 2048, 20480, 58.6, 65.4), (1, 3072, 24576, 69.6, 66.1), (17, 3072, 24576, 80.6, 83.2), (1, 7168, 36864, 149.9, 151.9), (16, 7168, 36864, 159.0, 161.7),
    (1, 5120, 34816, 108.7, 109.6), (24, 5120, 34816, 120.8, 122.8), (1, 8192, 21504, 160.3, 139.7), (32, 3584, 28672, 93.6, 95.7), (65, 2560, 19456, 104.8, 92.0),
    (80, 5120, 34816, 181.7, 165.1),
])
def test_windows_go_where_they_were_measured_faster(rows, K, N, items, shares):
    assert lib.load().rx_exl3_step_takes(rows, K, N, 1) == (shares < items)
