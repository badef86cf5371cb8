"""The decode GEMM of equal shares for 33 to 96 rows, one accumulator and a group of warps for each 16 rows of it, against the one of whole items, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cb", ["3inst", "mul1"])
@pytest.mark.parametrize("K,N,splits", [
    (128, 148 * 128, 1),          # one chunk and one item a share: nothing is handed on
    (256, 149 * 128, 1),          # every share but the first takes an accumulator
    (1152, 17 * 128, 9),          # 153 items of one chunk: a group's next chunk is several pieces on
    (1664, 75 * 128, 2),          # items of six and seven chunks, odd shares
    (2048, 224 * 128, 1),         # shares of one item and a half
    (640, 1187 * 128, 1),         # eight items and more a share
    (4096, 40 * 128, 7),          # short items, pieces on both ends
])
def test_tall_step_gemm_has_the_bits_of_the_item_gemm(cb, K, N, splits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as KK, lib
    L = lib.load()
    g = torch.Generator(device="cuda").manual_seed(K + N)
    tr = torch.randint(-32768, 32768, (K // 16, N // 16, 64), dtype=torch.int16, device="cuda", generator=g)
    w = KK.Exl3Weight(tr, None, None, None, cb)
    st = KK.new_status()
    flags = torch.zeros(KK.step_flags(), dtype=torch.int32, device="cuda")
    for rows in (33, 48, 50, 65, 80, 96):
        x = torch.randn(rows, K, device="cuda", generator=g).half()
        a = torch.full((splits, rows, N), float("nan"), device="cuda")
        KK.exl3_gemm(x, w, a, splits, st)
        for _ in range(3):                                       # the flags are left as they were found
            b = torch.full((splits * rows * N + 128,), float("nan"), device="cuda")
            lib.check(L.rx_exl3_gemm_step(x.data_ptr(), rows, K, tr.data_ptr(), N, KK.CB_ID[cb], b.data_ptr(), splits, flags.data_ptr(), st.data_ptr(),
                                          lib.stream_ptr()), "rx_exl3_gemm_step")
            KK.check_status(st)
            assert torch.equal(a.view(-1), b[:-128]) and bool(b[-128:].isnan().all())
            assert int(flags.abs().sum()) == 0


def test_more_rows_are_refused():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as KK, lib
    x, tr = torch.zeros(97, 128, dtype=torch.float16, device="cuda"), torch.zeros(8, 148 * 8, 64, dtype=torch.int16, device="cuda")
    part, flags, st = torch.zeros(97, 148 * 128, device="cuda"), torch.zeros(KK.step_flags(), dtype=torch.int32, device="cuda"), KK.new_status()
    with pytest.raises(lib.KernelError):
        lib.check(lib.load().rx_exl3_gemm_step(x.data_ptr(), 97, 128, tr.data_ptr(), 148 * 128, KK.CB_ID["mcg"], part.data_ptr(), 1, flags.data_ptr(), st.data_ptr(),
                                               lib.stream_ptr()), "rx_exl3_gemm_step")
