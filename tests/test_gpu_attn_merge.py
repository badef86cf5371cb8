"""The merge of attention chunks: the form for a few rows against the one for many, bit for bit."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,n_q,n_kv", [(128, 8, 2), (64, 8, 2)])
@pytest.mark.parametrize("lens", [(1, 255, 256, 257), (8000, 8192, 8448, 8449), (33000, 5, 16384, 32769)])
def test_few_rows_merge_as_many_do(hd, n_q, n_kv, lens):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(sum(lens))
    blocks = [(n + 63) // 64 for n in lens]
    pages, top = sum(blocks), max(lens)
    k, v = (torch.randn(pages, n_kv, 64, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.zeros(len(lens), max(blocks), dtype=torch.int32, device="cuda")
    at = 0
    for i, b in enumerate(blocks):
        bt[i, :b] = torch.arange(at, at + b)
        at += b
    copies = 1 + 296 // (n_q * hd // 128) // len(lens)                     # as many rows as the other form is chosen for, the same ones again
    suh = (torch.randn(n_q * hd, device="cuda", generator=g)).half()
    q0 = torch.randn(len(lens), n_q * hd, device="cuda", generator=g).bfloat16()
    out = []
    for reps in (1, copies):
        R = reps * len(lens)
        row_seq = torch.arange(len(lens), dtype=torch.int32, device="cuda").repeat(reps)
        ctx = torch.tensor(lens, dtype=torch.int32, device="cuda").repeat(reps)
        scratch = K.attn_decode_scratch(R, n_q, hd, (top + 255) // 256 * 256, "cuda")
        xr, plain, st = torch.empty(R, n_q * hd, dtype=torch.float16, device="cuda"), torch.empty(R, n_q * hd, dtype=torch.bfloat16, device="cuda"), K.new_status()
        K.attn_decode(K.KvTensorMap(k), K.KvTensorMap(v), q0.repeat(reps, 1), bt, row_seq, ctx, scratch, n_q, n_kv, hd, (top + 255) // 256 * 256,
                      1.0 / math.sqrt(hd), suh, xr, plain, st)
        K.check_status(st)
        out.append((xr, plain))
    for a, b in zip(*out):
        assert not bool(a.isnan().any())
        for r in range(copies):
            assert torch.equal(a, b[r * len(lens):(r + 1) * len(lens)])
