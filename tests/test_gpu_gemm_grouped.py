"""The persistent grouped GEMM against the decoded matrices in float64 and, bit for bit, against itself over other tilings."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(E, K, N, bits, cb, counts, seed):
    from rexl3_b200.ops import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(seed)
    rows = sum(counts)
    xs = torch.randn(rows, K, device="cuda", generator=g).half()
    tr = torch.randint(-32768, 32768, (E, K // 16, N // 16, 16 * bits), dtype=torch.int16, device="cuda", generator=g)
    ones = lambda n: torch.ones(n, dtype=torch.float16, device="cuda")  # noqa: E731
    dense = [KK.exl3_unpack(KK.Exl3Weight(tr[e].contiguous(), ones(K), ones(N), None, cb)).double() for e in range(E)]
    return KK, xs, tr, dense


def _tiles(counts, tile_rows, extra):
    off = np.concatenate([[0], np.cumsum(counts)])
    t = [(e, int(off[e]) + r, min(tile_rows, c - r)) for e, c in enumerate(counts) for r in range(0, c, tile_rows)]
    return t + [(0, 0, 0)] * extra


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("cb", ["3inst", "mcg", "mul1"])
@pytest.mark.parametrize("counts,K,N,splits", [
    ([1], 128, 128, 1),                                   # one item of one chunk
    ([0, 3, 1, 0, 17, 32], 384, 256, 3),                  # items of one chunk, idle experts, full and ragged tiles
    ([5] * 40, 512, 640, 2),                              # more items than CTAs
    ([130, 1, 64, 127], 640, 384, 1),                     # several tiles of an expert
])
def test_grouped_gemm(bits, cb, counts, K, N, splits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    L, E, rows = lib.load(), len(counts), sum(counts)
    KK, xs, tr, dense = _problem(E, K, N, bits, cb, counts, bits + K)
    got = {}
    for tile_rows in (16, 32, 64, 128):
        tab = torch.tensor(_tiles(counts, tile_rows, 7), dtype=torch.int32, device="cuda")
        part = torch.full((splits, rows, N), float("nan"), device="cuda")
        st = KK.new_status()
        lib.check(L.rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 2 * bits, KK.CB_ID[cb], part.data_ptr(), splits, tab.data_ptr(),
                                         tab.shape[0], tile_rows, st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
        KK.check_status(st)
        got[tile_rows] = part
    off = np.concatenate([[0], np.cumsum(counts)])
    for s in range(splits):
        k0, k1 = (K // 128) * s // splits * 128, (K // 128) * (s + 1) // splits * 128
        for e in range(E):
            x, w = xs[off[e]:off[e + 1], k0:k1].double(), dense[e][k0:k1]
            # fp32 sums of exact products: one rounding (2^-24) per addition of up to K terms
            assert ((got[16][s, off[e]:off[e + 1]].double() - x @ w).abs() <= K * 2.0 ** -24 * (x.abs() @ w.abs()) + 1e-30).all()
    for t in (32, 64, 128):
        assert torch.equal(got[t], got[16])


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("K,splits", [(384, 2), (640, 2), (640, 3), (1408, 5), (512, 4)])       # all but the last: splits that end in half a chunk
def test_splits_are_cut_at_64(bits, K, splits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    counts, N = [3, 40, 1, 100], 256
    L, rows = lib.load(), sum(counts)
    KK, xs, tr, dense = _problem(len(counts), K, N, bits, "3inst", counts, bits + K)
    off = np.concatenate([[0], np.cumsum(counts)])
    for tile_rows in (16, 128):
        tab = torch.tensor(_tiles(counts, tile_rows, 3), dtype=torch.int32, device="cuda")
        part, st = torch.full((splits, rows, N), float("nan"), device="cuda"), KK.new_status()
        lib.check(L.rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 2 * bits, KK.CB_ID["3inst"], part.data_ptr(), splits,
                                         tab.data_ptr(), tab.shape[0], tile_rows, st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
        KK.check_status(st)
        for s in range(splits):
            k0, k1 = K // 64 * s // splits * 64, K // 64 * (s + 1) // splits * 64
            for e in range(len(counts)):
                x, w = xs[off[e]:off[e + 1], k0:k1].double(), dense[e][k0:k1]
                assert ((part[s, off[e]:off[e + 1]].double() - x @ w).abs() <= K * 2.0 ** -24 * (x.abs() @ w.abs()) + 1e-30).all()


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("tile_rows", [16, 128])
@pytest.mark.parametrize("counts,K,N,splits", [([3, 1, 17, 32], 384, 256, 3), ([5] * 40, 512, 640, 2)])
def test_idle_tiles_may_stand_anywhere(bits, tile_rows, counts, K, N, splits):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    L, rows = lib.load(), sum(counts)
    KK, xs, tr, _ = _problem(len(counts), K, N, bits, "3inst", counts, bits + K)
    tiles = _tiles(counts, tile_rows, 0)
    got = []
    for tab in (tiles, [(0, 0, 0)] * 3 + [t for u in tiles for t in (u, (0, 0, 0))] + [(0, 0, 0)] * 40, tiles[::-1]):
        tab = torch.tensor(tab, dtype=torch.int32, device="cuda")
        part, st = torch.full((splits, rows, N), float("nan"), device="cuda"), KK.new_status()
        lib.check(L.rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 2 * bits, KK.CB_ID["3inst"], part.data_ptr(), splits,
                                         tab.data_ptr(), tab.shape[0], tile_rows, st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
        KK.check_status(st)
        got.append(part)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("rows", [65, 100, 128])
@pytest.mark.parametrize("bits,splits", [(3, 4), (4, 4), (4, 3)])
def test_plain_gemm_of_65_to_128_rows(rows, bits, splits):
    """These windows take the persistent kernel; smaller ones the general one: the same bits for a row either way."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    K, N = 1024, 384
    KK, xs, tr, dense = _problem(1, K, N, bits, "3inst", [rows], 1)
    w = KK.Exl3Weight(tr[0].contiguous(), torch.ones(K, dtype=torch.float16, device="cuda"), torch.ones(N, dtype=torch.float16, device="cuda"), None, "3inst")
    st, part, few = KK.new_status(), torch.zeros(splits, rows, N, device="cuda"), torch.zeros(splits, 33, N, device="cuda")
    KK.exl3_gemm(xs, w, part, splits, st)
    KK.exl3_gemm(xs[:33].contiguous(), w, few, splits, st)
    KK.check_status(st)
    assert torch.equal(part[:, :33], few)
    x = xs.double()
    assert ((part.double().sum(0) - x @ dense[0]).abs() <= K * 2.0 ** -23 * (x.abs() @ dense[0].abs())).all()


@pytest.mark.parametrize("rows", [65, 128])
@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("N", [4736, 4864])                # 148 and 152 items: one for a CTA, and more
def test_plain_gemm_of_many_items(rows, bits, N):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    K, splits = 1024, 4
    KK, xs, tr, dense = _problem(1, K, N, bits, "3inst", [rows], 1)
    w = KK.Exl3Weight(tr[0].contiguous(), None, None, None, "3inst")
    st, part, few = KK.new_status(), torch.zeros(splits, rows, N, device="cuda"), torch.zeros(splits, 33, N, device="cuda")
    KK.exl3_gemm(xs, w, part, splits, st)
    KK.exl3_gemm(xs[:33].contiguous(), w, few, splits, st)
    KK.check_status(st)
    assert torch.equal(part[:, :33], few)
    x = xs.double()
    assert ((part.double().sum(0) - x @ dense[0]).abs() <= K * 2.0 ** -23 * (x.abs() @ dense[0].abs())).all()


@pytest.mark.parametrize("how", ["abort", "limit"])
def test_waits_that_give_up_leave_the_device_usable(how):
    """The abort word, or a wait limit of a microsecond: the call returns, says so if a wait gave up, and the next call is right."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    counts, K, N = [70] * 24, 2048, 1536
    L, rows = lib.load(), sum(counts)
    KK, xs, tr, _ = _problem(len(counts), K, N, 3, "3inst", counts, 9)
    tab = torch.tensor(_tiles(counts, 128, 9), dtype=torch.int32, device="cuda")

    def run(st):
        part = torch.zeros(2, rows, N, device="cuda")
        lib.check(L.rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 6, 0, part.data_ptr(), 2, tab.data_ptr(), tab.shape[0], 128,
                                         st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
        return part, st.tolist()[0]
    want, code = run(KK.new_status())
    assert code == 0
    for _ in range(3):
        st = KK.new_status()
        KK.set_abort(st) if how == "abort" else KK.set_wait_limit(st, 1)
        part, code = run(st)
        assert code in (0, KK.ST_ABORTED if how == "abort" else KK.ST_TIMEOUT)
        assert code != 0 or torch.equal(part, want)
        part, code = run(KK.new_status())
        assert code == 0 and torch.equal(part, want)
