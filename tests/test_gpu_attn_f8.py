"""Decode attention over an E4M3 cache against float64, at the edges of pages, chunks and tiles, and a row's independence of its window."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(ctxs, rows_per_seq, n_q, n_kv, seed):
    """Sequences of the given contexts (keys before the window's rows), `rows_per_seq` adjacent rows each; pages shuffled."""
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(seed)
    hd, need = 128, [(c + rows_per_seq + 63) // 64 for c in ctxs]
    pages = sum(need)
    perm = torch.randperm(pages, device="cuda", generator=g).int()
    bt = torch.zeros(len(ctxs), max(need), dtype=torch.int32, device="cuda")
    for i, n in enumerate(need):
        bt[i, :n] = perm[sum(need[:i]):sum(need[:i]) + n]
    kc, vc = (torch.randn(pages, n_kv, 64, hd, device="cuda", generator=g).to(torch.float8_e4m3fn) for _ in range(2))
    q = (2 * torch.randn(len(ctxs) * rows_per_seq, n_q * hd, device="cuda", generator=g)).bfloat16()
    scale = 0.5 + torch.rand(2, n_kv, device="cuda", generator=g)
    seq = torch.tensor([i for i in range(len(ctxs)) for _ in range(rows_per_seq)], dtype=torch.int32, device="cuda")
    ctx = torch.tensor([c + r + 1 for c in ctxs for r in range(rows_per_seq)], dtype=torch.int32, device="cuda")
    maps = K.KvTensorMap(kc.view(torch.uint8)), K.KvTensorMap(vc.view(torch.uint8))
    return K, kc, vc, q, scale, seq, ctx, bt, maps


def _run(K, maps, q, scale, seq, ctx, bt, n_q, n_kv, msr):
    st, mx = K.new_status(), int(ctx.max())
    out = torch.zeros_like(q)
    K.attn_decode(*maps, q, bt, seq, ctx, K.attn_decode_scratch(q.shape[0], n_q, 128, mx), n_q, n_kv, 128, mx, 1 / math.sqrt(128), None, None, out, st,
                  kv_scale=scale, max_seq_rows=msr)
    K.check_status(st)
    return out


@pytest.mark.parametrize("n_q,n_kv", [(40, 8), (3, 3), (16, 1)])
@pytest.mark.parametrize("rows", [1, 3, 7])
def test_decode_over_e4m3_pages(n_q, n_kv, rows):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctxs = [0, 1, 62, 63, 64, 254, 255, 256, 511, 700, 1023, 1024, 1279, 1280, 3000]
    K, kc, vc, q, scale, seq, ctx, bt, maps = _case(ctxs, rows, n_q, n_kv, n_q + rows)
    out = _run(K, maps, q, scale, seq, ctx, bt, n_q, n_kv, rows)
    for r in range(len(seq)):
        s, c = int(seq[r]), int(ctx[r])
        pg = bt[s, :(c + 63) // 64].long()
        k, v = ((t[pg].double() * scale[i].double()[None, :, None, None]).transpose(1, 2).reshape(-1, n_kv, 128)[:c] for i, t in enumerate((kc, vc)))
        qq = q[r].double().view(n_kv, n_q // n_kv, 128)
        p = torch.softmax(torch.einsum("kgd,skd->kgs", qq, k) / math.sqrt(128), -1)
        want = torch.einsum("kgs,skd->kgd", p, v).reshape(-1)
        # probabilities rounded to fp16 (2^-11 each, of terms no larger than 448 / 15 times the output's size here) and one rounding to bf16
        assert (out[r].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 2.0 ** -11 * v.abs().max(), (r, c)
    # the same rows one by one: the same bits, whatever tile and block they had
    one = torch.cat([_run(K, maps, q[r:r + 1].contiguous(), scale, seq[r:r + 1], ctx[r:r + 1], bt, n_q, n_kv, 1) for r in range(len(seq))])
    assert torch.equal(out, one)


@pytest.mark.parametrize("n_q,n_kv", [(40, 8), (3, 3), (16, 1)])
@pytest.mark.parametrize("rows", [1, 3, 7])
@pytest.mark.parametrize("spread", [1.0, 40.0])           # 40: the running maxima move
def test_sums_do_not_depend_on_the_kernel(n_q, n_kv, rows, spread):
    """Queries that are not 8-byte aligned go through the kernel that expands the pages: the same bits, in short contexts and long ones."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctxs = [0, 1, 15, 16, 63, 64, 81, 255, 256, 300, 700, 1023, 1024, 1025, 1279, 1280, 1999, 3000]
    K, kc, vc, q, scale, seq, ctx, bt, maps = _case(ctxs, rows, n_q, n_kv, n_q + rows)
    q = (q.float() * spread).bfloat16()
    off = torch.empty(q.numel() + 2, dtype=q.dtype, device="cuda")[2:].view(q.shape)
    off.copy_(q)
    assert q.data_ptr() % 8 == 0 and off.data_ptr() % 8 == 4
    a, b = (_run(K, maps, x, scale, seq, ctx, bt, n_q, n_kv, rows) for x in (q, off))
    assert torch.isfinite(a.float()).all() and a.abs().max() > 0 and torch.equal(a, b)


@pytest.mark.parametrize("how", ["abort", "limit"])
def test_waits_that_give_up_leave_the_device_usable(how):
    """The abort word, or a wait limit of a microsecond: the call returns, says so if a wait gave up, and the next call is right."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    n_q, n_kv = 40, 8
    K, kc, vc, q, scale, seq, ctx, bt, maps = _case([5000, 9, 700, 3000], 7, n_q, n_kv, 5)
    want = _run(K, maps, q, scale, seq, ctx, bt, n_q, n_kv, 7)
    for _ in range(3):
        st, mx, out = K.new_status(), int(ctx.max()), torch.zeros_like(q)
        K.set_abort(st) if how == "abort" else K.set_wait_limit(st, 1)
        K.attn_decode(*maps, q, bt, seq, ctx, K.attn_decode_scratch(q.shape[0], n_q, 128, mx), n_q, n_kv, 128, mx, 1 / math.sqrt(128), None, None, out, st,
                      kv_scale=scale, max_seq_rows=7)
        code = st.tolist()[0]
        assert code in (0, K.ST_ABORTED if how == "abort" else K.ST_TIMEOUT)
        assert code != 0 or torch.equal(out, want)
        assert torch.equal(_run(K, maps, q, scale, seq, ctx, bt, n_q, n_kv, 7), want)
