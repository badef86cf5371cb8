"""The grouped GEMM over tiles of up to 256 rows, which decode the weights once for two accumulators, against tiles of 128 rows, bit for bit (those are held
to the decoded matrices elsewhere)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(xs, tr, counts, N, bits, cb, tile_rows, idle):
    from rexl3_b200.ops import kernels as KK
    from rexl3_b200.ops import lib
    off = np.concatenate([[0], np.cumsum(counts)])
    t = [(e, int(off[e]) + r, min(tile_rows, c - r)) for e, c in enumerate(counts) for r in range(0, c, tile_rows)]
    for i in idle:
        t.insert(min(i, len(t)), (0, 0, 0))
    tab = torch.tensor(t, dtype=torch.int32, device="cuda")
    rows, K = xs.shape
    part, st = torch.full((rows, N), float("nan"), device="cuda"), KK.new_status()
    lib.check(lib.load().rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 2 * bits, KK.CB_ID[cb], part.data_ptr(), 1, tab.data_ptr(),
                                              len(t), tile_rows, st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
    KK.check_status(st)
    return part


@pytest.mark.parametrize("bits,cb", [(3, "3inst"), (3, "mcg"), (4, "mul1"), (4, "3inst")])
@pytest.mark.parametrize("counts,K,N", [
    ([129], 128, 128),                                           # two units of one chunk, one item
    ([256, 1, 0, 255, 128, 192, 193], 384, 640),                 # full, ragged, one-box and two-box second units beside single ones
    ([300, 64, 65, 520, 127, 200] * 6, 640, 384),                # several items for a CTA, several tiles for an expert
    ([140] * 20, 128, 1536),                                     # every item two units of a single chunk
    ([1, 250, 16] * 30, 2048, 256),
])
@pytest.mark.parametrize("idle", [(), (0, 1, 3, 10 ** 6)])
def test_tall_tiles(bits, cb, counts, K, N, idle):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    g = torch.Generator(device="cuda").manual_seed(K + N)
    xs = torch.randn(sum(counts), K, device="cuda", generator=g).half()
    tr = torch.randint(-32768, 32768, (len(counts), K // 16, N // 16, 16 * bits), dtype=torch.int16, device="cuda", generator=g)
    want, got = (_run(xs, tr, counts, N, bits, cb, t, idle) for t in (128, 256))
    assert torch.isfinite(want).all() and want.abs().max() > 0 and torch.equal(got, want)


@pytest.mark.parametrize("rows,K,N", [(129, 128, 128), (300, 2048, 5120), (257, 256, 9600), (700, 384, 10112), (1300, 256, 4864)])
def test_rows_of_a_plain_product_do_not_depend_on_their_number(rows, K, N):
    """3.0 bpw, more than 128 rows: 128-row tiles, 256-row tiles and the kernel in between, against windows of 64 rows."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as KK
    from rexl3_b200.ops import lib
    g = torch.Generator(device="cuda").manual_seed(rows)
    xs = torch.randn(rows, K, device="cuda", generator=g).half()
    tr = torch.randint(-32768, 32768, (K // 16, N // 16, 48), dtype=torch.int16, device="cuda", generator=g)

    def run(x):
        part, st = torch.full((len(x), N), float("nan"), device="cuda"), KK.new_status()
        lib.check(lib.load().rx_exl3_gemm(x.data_ptr(), len(x), K, tr.data_ptr(), N, 6, KK.CB_ID["mcg"], part.data_ptr(), 1, st.data_ptr(), lib.stream_ptr()),
                  "rx_exl3_gemm")
        KK.check_status(st)
        return part
    got = run(xs)
    assert torch.isfinite(got).all() and got.abs().max() > 0 and torch.equal(got, torch.cat([run(xs[r:r + 64]) for r in range(0, rows, 64)]))
