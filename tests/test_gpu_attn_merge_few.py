"""The merge for a few rows, chosen by the longest context that a window may have, on contexts of few chunks and around its groups of 32 and 128 chunks."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("lens", [(1, 255, 256, 257), (31 * 256, 32 * 256, 32 * 256 + 1, 33 * 256 - 1), (127 * 256 + 1, 128 * 256, 128 * 256 + 1, 129 * 256)])
def test_few_rows_merge_as_many_do(hd, lens):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    n_q, n_kv, max_ctx, g = 8, 2, max(33 * 256, max(lens)), torch.Generator(device="cuda").manual_seed(sum(lens))
    blocks = [(n + 63) // 64 for n in lens]
    k, v = (torch.randn(sum(blocks), n_kv, 64, hd, device="cuda", generator=g).bfloat16() for _ in range(2))
    bt = torch.zeros(len(lens), max(blocks), dtype=torch.int32, device="cuda")
    for i, b in enumerate(blocks):
        bt[i, :b] = torch.arange(sum(blocks[:i]), sum(blocks[:i + 1]))
    suh = torch.randn(n_q * hd, device="cuda", generator=g).half()
    q0 = torch.randn(len(lens), n_q * hd, device="cuda", generator=g).bfloat16()
    out = []
    for reps in (1, 1 + 296 // (n_q * hd // 128) // len(lens)):           # the second: more rows than this form takes, the same ones again
        R = reps * len(lens)
        row_seq, ctx = torch.arange(len(lens), device="cuda").int().repeat(reps), torch.tensor(lens, device="cuda").int().repeat(reps)
        xr, plain = torch.empty(R, n_q * hd, dtype=torch.float16, device="cuda"), torch.empty(R, n_q * hd, dtype=torch.bfloat16, device="cuda")
        st, scratch = K.new_status(), K.attn_decode_scratch(R, n_q, hd, max_ctx, "cuda")
        K.attn_decode(K.KvTensorMap(k), K.KvTensorMap(v), q0.repeat(reps, 1), bt, row_seq, ctx, scratch, n_q, n_kv, hd, max_ctx, 1.0 / math.sqrt(hd), suh, xr, plain, st)
        K.check_status(st)
        out.append((xr, plain))
    for a, b in zip(*out):
        assert not bool(a.isnan().any()) and torch.equal(a.repeat(len(b) // len(a), 1), b)
