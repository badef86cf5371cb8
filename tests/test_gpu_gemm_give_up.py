"""GEMMs whose waits give up (the abort word, or a limit that is too short): the call returns, says so where a wait gave up, and the next call is right."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LIMITS = (1, 2, 5, 10, 20, 40, 100)          # microseconds: from the first copy to the last accumulator


def _check(call, want_like):
    """`call(out, status)` under every limit and the abort word, with plain calls after each.  Returns how many gave up."""
    from rexl3_b200.ops import kernels as KK
    want = torch.full_like(want_like, float("nan"))
    st = KK.new_status()
    call(want, st)
    KK.check_status(st)
    gave_up = 0
    for us in ("abort",) + LIMITS + ("abort",):
        st = KK.new_status()
        KK.set_abort(st) if us == "abort" else KK.set_wait_limit(st, us)
        got = torch.full_like(want, float("nan"))
        call(got, st)
        code = st.tolist()[0]
        assert code in (0, KK.ST_ABORTED if us == "abort" else KK.ST_TIMEOUT)
        gave_up += code != 0
        assert code != 0 or torch.equal(got.view(torch.int32), want.view(torch.int32))
        for _ in range(2):
            st, got = KK.new_status(), torch.full_like(want, float("nan"))
            call(got, st)
            KK.check_status(st)
            assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    return gave_up


def _weights(K, N, words=64, cb="3inst"):
    from rexl3_b200.ops import kernels as KK
    g = torch.Generator(device="cuda").manual_seed(K + N)
    tr = torch.randint(-32768, 32768, (K // 16, N // 16, words), dtype=torch.int16, device="cuda", generator=g)
    return KK, KK.Exl3Weight(tr, None, None, None, cb), g


@pytest.fixture(scope="module")
def long_kernel():
    """A GEMM of 74 CTAs and some 300 us; what comes next in the stream may begin on the other SMs meanwhile."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    K, N = 131072, 74 * 128
    KK, w, g = _weights(K, N)
    x, part, st = torch.randn(1, K, device="cuda", generator=g).half(), torch.empty(1, N, device="cuda"), KK.new_status()
    yield lambda: KK.exl3_gemm(x, w, part, 1, st)
    KK.check_status(st)


@pytest.mark.parametrize("rows,words", [(1, 64), (100, 64), (20, 32), (20, 40), (20, 96)])
def test_item_gemm_behind_a_long_kernel(long_kernel, rows, words):
    """4.0 bpw decoded into tensor memory, and code widths of 2, 2.5 and 6 bits, the three forms of the general kernel's decode loop."""
    K, N = 4096, 1152
    KK, w, g = _weights(K, N, words, "mul1" if words == 40 else "3inst")
    x = torch.randn(rows, K, device="cuda", generator=g).half()

    def call(out, st):
        long_kernel()
        KK.exl3_gemm(x, w, out, 1, st)
    _check(call, torch.empty(rows, N, device="cuda"))


@pytest.mark.parametrize("rows,words,step", [(1, 64, False), (100, 64, False), (20, 32, False), (20, 40, False), (20, 64, None), (20, 96, False), (1, 64, True),
                                             (80, 64, True)])
def test_the_time_of_the_kernel_before_does_not_count(long_kernel, rows, words, step):
    """A GEMM that begins under a kernel of some 300 us, with a limit that is below that and above each of its own waits.  step None: the general kernel."""
    from rexl3_b200.ops import lib
    K, N = 4096, 224 * 128 if step else 1152
    KK, w, g = _weights(K, N, words, "mul1" if words == 40 else "3inst")
    x, part = torch.randn(rows, K, device="cuda", generator=g).half(), torch.empty(rows, N, device="cuda")
    flags, st = torch.zeros(KK.step_flags(), dtype=torch.int32, device="cuda"), KK.new_status()
    KK.set_wait_limit(st, 100)
    for _ in range(5):
        long_kernel()
        if step:
            lib.check(lib.load().rx_exl3_gemm_step(x.data_ptr(), rows, K, w.trellis.data_ptr(), N, KK.CB_ID[w.codebook], part.data_ptr(), 1, flags.data_ptr(),
                                                   st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_step")
        else:
            KK.exl3_gemm(x, w, part, 1, st, force_generic=step is None)
        KK.check_status(st)


@pytest.mark.parametrize("rows,K,N,splits", [
    (1, 2048, 224 * 128, 1),      # shares of one item and a half
    (17, 1664, 75 * 128, 2),      # odd shares
    (80, 2048, 224 * 128, 1),     # one accumulator, blocks of 16 rows
    (96, 4096, 40 * 128, 7),      # short items, pieces on both ends
])
@pytest.mark.parametrize("kept", [False, True])
def test_step_gemm(rows, K, N, splits, kept):
    """kept: all calls use one flags buffer, as an executor's do; one that gave up leaves it as it found it, too."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    KK, w, g = _weights(K, N)
    x = torch.randn(rows, K, device="cuda", generator=g).half()

    one = torch.zeros(KK.step_flags(), dtype=torch.int32, device="cuda")

    def call(out, st):
        flags = one if kept else torch.zeros_like(one)
        lib.check(lib.load().rx_exl3_gemm_step(x.data_ptr(), rows, K, w.trellis.data_ptr(), N, KK.CB_ID[w.codebook], out.data_ptr(), splits, flags.data_ptr(),
                                               st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_step")
        assert int(flags.abs().sum()) == 0
    assert _check(call, torch.empty(splits, rows, N, device="cuda")) > 0


@pytest.mark.parametrize("form", ["plain", "swiglu", "store"])
@pytest.mark.parametrize("rows,K,N", [
    (300, 1280, 2304),            # fewer tiles than pairs of CTAs
    (2304, 1024, 4352),           # accumulators handed on, a last strip without a partner in the plain form
])
def test_wide_gemm(form, rows, K, N):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    N = N + (128 if form == "plain" else 0)
    KK, w, g = _weights(K, N)
    w.svh, suh = (0.05 * torch.randn(N, device="cuda", generator=g)).half(), torch.randn(N // 2, device="cuda", generator=g).half()
    x = torch.randn(rows, K, device="cuda", generator=g).half()
    work = torch.zeros(KK.wide_bytes(K, N), dtype=torch.uint8, device="cuda")

    def call(out, st):
        if form == "plain":
            lib.check(lib.load().rx_exl3_gemm_wide(x.data_ptr(), rows, K, w.trellis.data_ptr(), N, KK.CB_ID[w.codebook], out.data_ptr(), work.data_ptr(),
                                                   work.numel(), st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_wide")
        elif form == "swiglu":
            KK.exl3_gemm_swiglu_rot(x, w, suh, out, work, st)
        else:
            KK.exl3_gemm_store(x, w, out, work, st)
    assert _check(call, torch.empty(rows, N // 2, dtype=torch.float16, device="cuda") if form == "swiglu" else torch.empty(rows, N, device="cuda")) > 0


def test_expert_tiles_of_256_rows():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    E, K, N, counts = 12, 2048, 1536, [300, 0, 256, 17, 129, 400, 64, 200, 255, 1, 90, 257]
    g = torch.Generator(device="cuda").manual_seed(5)
    from rexl3_b200.ops import kernels as KK
    tr = torch.randint(-32768, 32768, (E, K // 16, N // 16, 48), dtype=torch.int16, device="cuda", generator=g)
    rows, tab, at = sum(counts), [], 0
    for e, n in enumerate(counts):
        tab += [(e, at + i, min(256, n - i)) for i in range(0, n, 256)]
        at += n
    tab = torch.tensor(tab, dtype=torch.int32, device="cuda")
    xs = torch.randn(rows, K, device="cuda", generator=g).half()

    def call(out, st):
        lib.check(lib.load().rx_exl3_gemm_grouped(xs.data_ptr(), rows, K, tr.data_ptr(), tr[0].numel(), N, 6, 0, out.data_ptr(), 1, tab.data_ptr(), tab.shape[0],
                                                  256, st.data_ptr(), lib.stream_ptr()), "rx_exl3_gemm_grouped")
    assert _check(call, torch.empty(rows, N, device="cuda")) > 0
