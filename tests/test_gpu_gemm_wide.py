"""The GEMM that decodes a matrix once per call against the one that decodes it per tile, bit for bit, and against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(rows, K, N, cb, seed=0):
    from rexl3_b200.ops import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(seed + rows + K + N)
    tr = torch.randint(-32768, 32768, (K // 16, N // 16, 64), dtype=torch.int16, device="cuda", generator=g)
    w = KK.Exl3Weight(tr, torch.randn(K, device="cuda", generator=g).half(), (0.05 * torch.randn(N, device="cuda", generator=g)).half(), None, cb)
    work = torch.zeros(KK.wide_bytes(K, N), dtype=torch.uint8, device="cuda")
    return KK, w, torch.randn(rows, K, device="cuda", generator=g).half(), work, KK.new_status(), g


def _wide(KK, x, w, part, work, st):
    from rexl3_b200.ops import lib
    lib.check(lib.load().rx_exl3_gemm_wide(x.data_ptr(), x.shape[0], w.K, w.trellis.data_ptr(), w.N, KK.CB_ID[w.codebook], part.data_ptr(), work.data_ptr(),
                                           work.numel(), st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_wide")


@pytest.mark.parametrize("cb", ["3inst", "mcg", "mul1"])
@pytest.mark.parametrize("rows,K,N", [
    (1, 256, 128),            # the smallest: one piece, a column tile of one strip
    (257, 384, 640),          # an odd number of 128 k, a last strip without a partner, a row tile of one row
    (511, 1280, 2304),        # a segment of one piece; fewer tiles than pairs of CTAs
    (2304, 512, 2176),        # 81 tiles for 74 pairs: accumulators handed on
    (2100, 1152, 5120),       # two bands of row tiles, shares of more than two tiles
    (4736, 2176, 1024),       # 76 tiles, all whole or split near an end
    (1184, 256, 3840),        # 75 tiles of four k blocks: too few to be split
    (1184, 1024, 3840),       # 75 tiles of sixteen: split in the middle or not at all
])
def test_wide_gemm_has_the_bits_of_the_tile_gemm(cb, rows, K, N):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    KK, w, x, work, st, g = _problem(rows, K, N, cb)
    a = torch.full((rows, N), float("nan"), device="cuda")
    KK.exl3_gemm(x, w, a, 1, st)
    for _ in range(2):                                       # the counters are left as they were found
        b = torch.full((rows + 1, N), float("nan"), device="cuda")
        _wide(KK, x, w, b, work, st)
        KK.check_status(st)
        assert torch.equal(a, b[:rows]) and bool(b[rows].isnan().all())
        assert int(work[:4096 * 4].view(torch.int32).abs().sum()) == 0
    ones = lambda n: torch.ones(n, dtype=torch.float16, device="cuda")  # noqa: E731
    dense = KK.exl3_unpack(KK.Exl3Weight(w.trellis, ones(K), ones(N), None, cb)).double()
    # fp32 sums of exact products: one rounding (2^-24) per addition of up to K terms
    assert ((a.double() - x.double() @ dense).abs() <= K * 2.0 ** -24 * (x.double().abs() @ dense.abs()) + 1e-30).all()


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("rows,K,F", [(1, 256, 128), (300, 640, 256), (2200, 512, 1152), (1030, 1024, 2176)])
def test_wide_swiglu_has_the_bits_of_gemm_and_finish(rows, K, F, bias):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    KK, w, x, work, st, g = _problem(rows, K, 2 * F, "3inst")
    w.bias = torch.randn(2 * F, device="cuda", generator=g) if bias else None
    suh = torch.randn(F, device="cuda", generator=g).half()
    part = torch.empty(rows, 2 * F, device="cuda")
    a = torch.full((rows, F), float("nan"), device="cuda", dtype=torch.float16)
    b = torch.full((rows + 1, F), float("nan"), device="cuda", dtype=torch.float16)
    KK.exl3_gemm(x, w, part, 1, st)
    KK.finish_swiglu_rot(part, 1, rows, w, suh, a)
    KK.exl3_gemm_swiglu_rot(x, w, suh, b, work, st)
    KK.check_status(st)
    assert torch.equal(a, b[:rows]) and bool(b[rows].isnan().all())


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("rows,K,N", [(1, 256, 128), (257, 384, 640), (2304, 512, 2176), (2100, 1152, 5120), (1184, 1024, 3840)])
def test_wide_store_has_the_bits_of_gemm_and_finish(rows, K, N, bias):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    KK, w, x, work, st, g = _problem(rows, K, N, "mcg")
    w.bias = torch.randn(N, device="cuda", generator=g) if bias else None
    part, a = torch.empty(rows, N, device="cuda"), torch.full((rows, N), float("nan"), device="cuda")
    b = torch.full((rows + 1, N), float("nan"), device="cuda")
    KK.exl3_gemm(x, w, part, 1, st)
    KK.finish_store(part, 1, rows, w, a)
    for _ in range(2):
        KK.exl3_gemm_store(x, w, b, work, st)
        KK.check_status(st)
        assert torch.equal(a, b[:rows]) and bool(b[rows].isnan().all())


def test_prompt_slice_through_either_gemm_gives_the_same_logits():
    """A model whose slice of 1100 rows takes the wide kernel, against the same model without its workspace."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models import dense
    cfg = dense.DenseConfig(n_layers=2, d_model=4096, n_q=8, n_kv=2, head_dim=128, ffn=14336, vocab=512, bits=4.0)
    T = 1100
    m = dense.DenseGPU(cfg, num_pages=20, max_rows=64, max_seqs=1, max_blocks_per_seq=20, max_prefill_rows=T)
    assert m.wide is not None and m.K.wide_takes(m.layers[0]["gate_up"], T, True)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    pos = list(range(T))
    pf = dict(seq_ids=i32([0]), q_start=i32([0]), q_len=i32([T]), pos0=i32([0]), nseq=1, max_qlen=T)
    args = (i32([7 * p % 512 for p in pos]), i32(pos), i32(pos), i32([0] * T), i32([p + 1 for p in pos]), i32([list(range(20))]))
    out = []
    for work in (m.wide, None):
        m.wide = work
        out.append(m.forward_rows(*args, prefill=pf, logit_rows=torch.arange(T - 200, T, device="cuda")).clone())
        m.check()
    assert torch.equal(*out)
