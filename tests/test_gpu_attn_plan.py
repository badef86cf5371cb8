"""The window plan of decode attention against a walk over the rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HEAD, CAP, CHUNK = 8, 1024, 256


def _walk(seq, ctx, rb, n_kv, tree):
    blocks, r, rows = [], 0, len(seq)
    while r < rows:
        n = 1
        while n < rb and r + n < rows and seq[r + n] == seq[r]:
            n += 1
        nch = (tree[r] + 1) // CHUNK if tree else -(-max(ctx[r:r + n]) // CHUNK)
        if nch:
            blocks.append((r, n, nch, seq[r], 0))
        r += n
    for r in range(rows if tree else 0):
        c0 = (tree[r] + 1) // CHUNK
        nch = -(-ctx[r] // CHUNK) - c0
        if nch > 0:
            blocks.append((r, 1, nch, -1 - r, c0))
    prefix = [0]
    for b in blocks:
        prefix.append(prefix[-1] + b[2] * n_kv)
    return blocks, prefix


@pytest.mark.parametrize("rows", [1, 31, 80, 256, 257, 512, 1024])
@pytest.mark.parametrize("n_q,n_kv,run", [(40, 8, 5), (32, 2, 1), (8, 8, 37), (12, 4, 3)])
@pytest.mark.parametrize("tree", [False, True])
def test_plan_equals_a_walk_over_the_rows(rows, n_q, n_kv, run, tree):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    if tree and 2 * rows > CAP:
        pytest.skip("a tree's plan holds two blocks per row")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator().manual_seed(rows + run)
    seq = [(r // run) * 3 % 50 for r in range(rows)]
    base = {s: int(torch.randint(0, 2000, (1,), generator=g)) for s in set(seq)}
    ctx = [base[s] + 1 + int(torch.randint(0, 60, (1,), generator=g)) for s in seq]
    if not tree:
        ctx[rows // 2] = 0                                       # an idle row
    tb = [base[s] for s in seq] if tree else None
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    plan = K.attn_plan_buffer("cuda")
    K.attn_plan(dev(seq), dev(ctx), n_q, n_kv, run, plan, dev(tb) if tree else None)
    got = plan.tolist()
    items, nb, rb, kv = got[:4]
    blocks, prefix = _walk(seq, ctx, rb, n_kv, tb)
    assert (items, nb, kv) == (prefix[-1], len(blocks), n_kv)
    at = lambda i, n: got[HEAD + i:HEAD + i + n]  # noqa: E731
    assert list(zip(at(0, nb), at(CAP, nb), at(2 * CAP, nb), at(4 * CAP + 1, nb), at(5 * CAP + 1, nb))) == blocks
    assert at(3 * CAP, nb + 1) == prefix


@pytest.mark.parametrize("cache", ["bf16", "fp8", "int8"])
@pytest.mark.parametrize("rows,ctx", [(1, 5000), (1, 200), (15, 3000)])
def test_own_plan_is_read_after_it_is_written(cache, rows, ctx):
    """Calls that bring no plan make one in their scratch; its readers begin before it is there.  Zeroed scratch holds an empty plan: a reader that does not
    wait leaves chunks out."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import math
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(rows + ctx)
    n_q, n_kv, hd, need = 40, 8, 128, (ctx + 63) // 64
    bt = torch.randperm(rows * need, device="cuda", generator=g).int().view(rows, need)
    x = [torch.randn(rows * need, n_kv, 64, hd, device="cuda", generator=g) for _ in range(2)]
    kw = {}
    if cache == "bf16":
        kv = [t.bfloat16() for t in x]
    elif cache == "fp8":
        kv, kw["kv_scale"] = [t.to(torch.float8_e4m3fn).view(torch.uint8) for t in x], torch.ones(2, n_kv, device="cuda")
    else:
        kv, kw["kv_tscale"] = [(t * 30).round().clamp(-127, 127).to(torch.int8) for t in x], [torch.full((rows * need, n_kv, 64), 2.0 ** -5, device="cuda") for _ in range(2)]
    q = torch.randn(rows, n_q * hd, device="cuda", generator=g).bfloat16()
    seq = torch.arange(rows, dtype=torch.int32, device="cuda")
    lens = torch.full((rows,), ctx, dtype=torch.int32, device="cuda")
    maps, st, plan = [K.KvTensorMap(t) for t in kv], K.new_status(), K.attn_plan_buffer("cuda")
    K.attn_plan(seq, lens, n_q, n_kv, 1, plan)
    scratch = K.attn_decode_scratch(rows, n_q, hd, ctx)

    def run(plan):
        out = torch.zeros_like(q)
        scratch.zero_()
        torch.cuda.synchronize()
        K.attn_decode(*maps, q, bt, seq, lens, scratch, n_q, n_kv, hd, ctx, 1 / math.sqrt(hd), None, None, out, st, plan=plan, **kw)
        return out
    want = run(plan)
    for _ in range(30):
        assert torch.equal(run(None), want)
    K.check_status(st)
