"""The tensor-core prefill attention at the edges of its tiles and pages, against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,pos", [
    ([1], [0]),                              # one row, one page
    ([64, 65], [0, 63]),                     # one page; two pages by one row
    ([128, 129, 1], [0, 64, 511]),           # an empty and a one-row second tile
    ([256, 257, 300], [1, 127, 0]),          # full tiles, a second CTA
    ([513], [700]),
])
@pytest.mark.parametrize("n_q,n_kv", [(4, 2), (5, 1)])
def test_prefill_attention(lens, pos, n_q, n_kv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    hd, rows = 128, sum(lens)
    g = torch.Generator(device="cuda").manual_seed(rows + n_q)
    total = [p + n for p, n in zip(pos, lens)]
    blocks = max((t + 63) // 64 for t in total)
    pages = len(lens) * blocks + 3
    kc, vc = (torch.randn(pages, n_kv, 64, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.randperm(pages, device="cuda", generator=g)[:len(lens) * blocks].view(len(lens), blocks).int()
    q = torch.randn(rows, n_q * hd, device="cuda", generator=g).bfloat16()
    out = torch.full((rows, n_q * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    starts = [sum(lens[:i]) for i in range(len(lens))]
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    st = K.new_status()
    K.attn_prefill(K.KvTensorMap(kc), K.KvTensorMap(vc), q, bt, dev(list(range(len(lens)))), dev(starts), dev(lens), dev(pos), out, len(lens), max(lens), n_q, n_kv, hd,
                   1 / math.sqrt(hd), st)
    K.check_status(st)
    for i, (n, p) in enumerate(zip(lens, pos)):
        k, v = (c[bt[i].long()].transpose(1, 2).reshape(-1, n_kv, hd)[:total[i]].double().repeat_interleave(n_q // n_kv, 1) for c in (kc, vc))
        x = q[starts[i]:starts[i] + n].view(n, n_q, hd).double()
        s = torch.einsum("rhd,khd->hrk", x, k) / math.sqrt(hd)
        s = s.masked_fill(torch.arange(total[i], device="cuda")[None, None] > (p + torch.arange(n, device="cuda"))[None, :, None], float("-inf"))
        w = s.softmax(-1)
        want, mass = torch.einsum("hrk,khd->rhd", w, v), torch.einsum("hrk,khd->rhd", w, v.abs())
        got = out[starts[i]:starts[i] + n].view(n, n_q, hd).double()
        # bf16 probabilities and a bf16 result: 8 significant bits, so a rounding moves a value by 2^-8 of it at most; 2^-11 for the fp32 scores, their exponentials and sums
        assert ((got - want).abs() <= (2 * 2.0 ** -8 + 2.0 ** -11) * mass).all()


@pytest.mark.parametrize("how", ["abort", "limit"])
def test_waits_that_give_up_leave_the_device_usable(how):
    """The abort word, or a wait limit of a microsecond: the call returns, says so if a wait gave up, and the next call is right."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    n_q, n_kv, hd, rows = 8, 2, 128, 1500
    g = torch.Generator(device="cuda").manual_seed(2)
    kc, vc = (torch.randn(24, n_kv, 64, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.randperm(24, device="cuda", generator=g).view(1, 24).int()
    q = torch.randn(rows, n_q * hd, device="cuda", generator=g).bfloat16()
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    maps, a = (K.KvTensorMap(kc), K.KvTensorMap(vc)), (dev([0]), dev([0]), dev([rows]), dev([0]))

    def run(st):
        out = torch.zeros_like(q)
        K.attn_prefill(*maps, q, bt, *a, out, 1, rows, n_q, n_kv, hd, 1 / math.sqrt(hd), st)
        return out, st.tolist()[0]
    want, code = run(K.new_status())
    assert code == 0
    for _ in range(3):
        st = K.new_status()
        K.set_abort(st) if how == "abort" else K.set_wait_limit(st, 1)
        out, code = run(st)
        assert code in (0, K.ST_ABORTED if how == "abort" else K.ST_TIMEOUT)
        assert code != 0 or torch.equal(out, want)
        out, code = run(K.new_status())
        assert code == 0 and torch.equal(out, want)
