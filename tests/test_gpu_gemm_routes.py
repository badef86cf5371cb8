"""Executors whose products go by the kernels of equal shares, of matrices decoded once and of expert tiles of 256 rows: the logits of the same rows by the other kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _slice(ids, first, pages):
    """Rows first .. of sequence 0 as a prompt slice."""
    T = len(ids)
    pos = list(range(first, first + T))
    rows = (_i32(ids), _i32(pos), _i32(pos), _i32([0] * T), _i32([p + 1 for p in pos]), _i32([list(range(pages))]))
    return rows, dict(seq_ids=_i32([0]), q_start=_i32([0]), q_len=_i32([T]), pos0=_i32([first]), nseq=1, max_qlen=T)


@pytest.mark.parametrize("seqs,each", [(1, 1), (16, 1), (16, 5)])
def test_window_by_equal_shares(seqs, each):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models import dense
    from rexl3_b200.ops import lib
    cfg = dense.DenseConfig(n_layers=3, d_model=4096, n_q=8, n_kv=2, head_dim=128, ffn=14336, vocab=512, bits=4.0)
    m = dense.DenseGPU(cfg, num_pages=16, max_rows=80, max_seqs=16, max_blocks_per_seq=1, max_prefill_rows=80)
    w = m.layers[0]["gate_up"]
    assert lib.load().rx_exl3_step_takes(seqs * each, w.K, w.N, m.splits[("decode", "gate_up")])
    pos = list(range(each)) * seqs
    seq = [s for s in range(seqs) for _ in range(each)]
    args = (_i32([7 * i % 512 for i in range(len(pos))]), _i32(pos), _i32([s * 64 + p for s, p in zip(seq, pos)]), _i32(seq), _i32([p + 1 for p in pos]),
            _i32([[i] for i in range(16)]))
    run = lambda: m.forward_rows(*args, max_ctx=256)  # noqa: E731
    out = [run().clone(), run().clone()]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        lg = run()
    for _ in range(3):
        lg.zero_()
        g.replay()
        out.append(lg.clone())
    m.check()
    flags, m.step_flags = m.step_flags, None
    want = run().clone()
    m.check()
    assert int(flags.abs().sum()) == 0 and bool(want.isfinite().all()) and bool(want.any())
    assert all(torch.equal(o, want) for o in out)


def test_recurrent_slice_with_and_without_the_workspace():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models import hybrid
    cfg = hybrid.HybridConfig(n_layers=3, d_model=2048, n_q=8, n_kv=2, head_dim=128, ffn=2048, vocab=512, bits=4.0, pattern="MGA", ssm_heads=64, ssm_groups=8,
                              gdn_k_heads=8, gdn_v_heads=16)
    T, pages = 2100, 33
    m = hybrid.HybridGPU(cfg, num_pages=pages, max_rows=64, max_seqs=1, max_blocks_per_seq=pages, max_prefill_rows=T)
    assert m.wide is not None and all(m.K.wide_takes(m.layers[i]["in_proj"], T, store=True) for i in (0, 1))
    rows, pf = _slice([7 * p % 512 for p in range(T)], 0, pages)
    out = []
    for work in (m.wide, None):
        m.wide = work
        lg = m.forward_rows(*rows, prefill=pf, logit_rows=torch.arange(T - 200, T, device="cuda")).clone()
        m.check()
        out.append((lg, *(p.clone() for pool in (m.conv_pool, m.ssm_pool) for p in pool.values())))
    assert bool(out[0][0].isfinite().all()) and bool(out[0][0].any())
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_routed_slice_by_tall_tiles():
    """One slice of 80 rows for an expert on average against the same prompt in two slices, whose tiles have 128 rows."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models import moe
    cfg = moe.MoEConfig(n_layers=2, d_model=512, n_q=4, n_kv=2, head_dim=128, ffn=128, vocab=512, bits=3.0, n_experts=8, top_k=4, expert_ffn=1280)
    T, pages = 400, 7
    m = moe.MoEGPU(cfg, num_pages=pages, max_rows=64, max_seqs=1, max_blocks_per_seq=pages, max_prefill_rows=T)
    tiles, grouped = [], m._grouped_shifted
    m._grouped_shifted = lambda xs, st, splits, max_tiles, tile_rows, cap: (tiles.append(tile_rows), grouped(xs, st, splits, max_tiles, tile_rows, cap))
    ids, got = [7 * p % 512 for p in range(T)], []
    for cuts in ((0, T), (0, 150, 300, T)):
        for a, b in zip(cuts, cuts[1:]):
            rows, pf = _slice(ids[a:b], a, pages)
            got.append(m.forward_rows(*rows, prefill=pf, logit_rows=torch.arange(b - a - 100, b - a, device="cuda")).clone())
            m.check()
    assert set(tiles[:4]) == {256} and set(tiles[4:]) == {128}
    assert bool(got[0].isfinite().all()) and bool(got[0].any()) and torch.equal(got[0], got[-1])
