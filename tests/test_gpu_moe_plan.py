"""The planning sort of the routed experts against a stable sort on the host, and the forms of the finish kernels for one plane against the general ones."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [1, 31, 33, 128, 1024, 1025, 16801])
@pytest.mark.parametrize("E,lo,hi", [(1, 0, 1), (128, 0, 128), (128, 32, 64), (512, 3, 511)])
def test_plan_is_a_stable_sort(pairs, E, lo, hi):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    L = lib.load()
    rng = np.random.default_rng(pairs + E)
    ids = rng.integers(-1 if pairs % 2 else 0, E, size=pairs).astype(np.int32)       # -1: a pair nobody owns
    ids[rng.random(pairs) < 0.3] = lo                                                # one busy expert
    tile_rows = 32
    order = [p for e in range(lo, hi) for p in np.flatnonzero(ids == e)]
    cnt = [int((ids == e).sum()) if lo <= e < hi else 0 for e in range(E)]
    offs = np.concatenate([[0], np.cumsum(cnt)])
    tiles = [(e, int(offs[e]) + r, min(tile_rows, cnt[e] - r)) for e in range(E) for r in range(0, cnt[e], tile_rows)]
    for max_tiles in (len(tiles) + 5, max(1, len(tiles) - 1)):                       # idle tiles are zeroed; too small a table is cut
        z = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")  # noqa: E731
        d_ids, d_offs, d_pos, d_pair, d_exp, d_tab, d_tot = torch.from_numpy(ids).cuda(), z(E + 1), z(pairs), z(pairs), z(pairs), z(3 * max_tiles), z(1)
        lib.check(L.rx_moe_plan(d_ids.data_ptr(), pairs, E, lo, hi, tile_rows, max_tiles, d_offs.data_ptr(), d_pos.data_ptr(), d_pair.data_ptr(),
                                d_exp.data_ptr(), d_tab.data_ptr(), d_tot.data_ptr(), lib.stream_ptr()), "rx_moe_plan")
        n = len(order)
        assert d_tot.item() == n and d_offs.tolist() == offs.tolist()
        assert d_pair[:n].tolist() == [int(p) for p in order] and d_exp[:n].tolist() == [int(ids[p]) for p in order]
        want = np.full(pairs, -1)
        want[order] = np.arange(n)
        assert d_pos.tolist() == want.tolist()
        assert d_tab.view(-1, 3).tolist() == [list(t) for t in (tiles + [(0, 0, 0)] * 5)[:max_tiles]]


@pytest.mark.parametrize("M,topk", [(3, 1), (70, 8), (70, 10), (5, 17)])
def test_forms_of_few_planes_equal_the_general_ones(M, topk):
    """Further planes of zeros select the other forms (one plane, up to four, any number) and change no bit of a sum."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models.moe import CombineDst
    from rexl3_b200.ops import lib
    L, E, d, F, pairs = lib.load(), 24, 384, 256, M * topk
    g = torch.Generator(device="cuda").manual_seed(M * topk)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    ids = torch.randint(0, E, (pairs,), device="cuda", generator=g).int()
    pos = torch.randperm(pairs, device="cuda", generator=g).int()
    pos[::7] = -1                                                                    # another rank's pairs
    w, svh, gu, dn = r(pairs).abs(), r(E, d).half(), r(pairs, 2 * F), r(pairs, d)
    svh_gu, suh, exp, tot = r(E, 2 * F).half(), r(E, F).half(), ids.clone(), torch.tensor([pairs], dtype=torch.int32, device="cuda")
    got = []
    for S in (1, 2, 4, 5):
        planes = lambda t: torch.stack([t] + [torch.zeros_like(t)] * (S - 1))  # noqa: E731,B023
        slot, act = torch.zeros(M, d, device="cuda"), torch.zeros(pairs, F, dtype=torch.float16, device="cuda")
        dst = CombineDst()
        dst.ranks, dst.rank, dst.rows_cap, dst.dst[0] = 1, 0, M, slot.data_ptr()
        a, b = planes(dn), planes(gu)
        lib.check(L.rx_moe_combine(a.data_ptr(), S, pairs, M, d, topk, ids.data_ptr(), w.data_ptr(), pos.data_ptr(), svh.data_ptr(), None,
                                   ctypes.byref(dst), lib.stream_ptr()), "rx_moe_combine")
        lib.check(L.rx_moe_swiglu_rot(b.data_ptr(), S, pairs, F, exp.data_ptr(), tot.data_ptr(), svh_gu.data_ptr(), suh.data_ptr(), act.data_ptr(),
                                      lib.stream_ptr()), "rx_moe_swiglu_rot")
        got.append((slot, act))
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert torch.isfinite(x.float()).all() and x.abs().max() > 0 and torch.equal(x, y)



@pytest.mark.parametrize("S", [2, 3, 4, 5, 9])
@pytest.mark.parametrize("M,topk", [(3, 1), (70, 8), (5, 17)])
def test_planes_are_added_in_order(S, M, topk):
    """Random planes against one plane that holds their sums, added in plane order in fp32: every plane counts once, in its place, in every form."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models.moe import CombineDst
    from rexl3_b200.ops import lib
    L, E, d, F, pairs = lib.load(), 24, 384, 256, M * topk
    g = torch.Generator(device="cuda").manual_seed(M * topk + S)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    ids = torch.randint(0, E, (pairs,), device="cuda", generator=g).int()
    pos = torch.randperm(pairs, device="cuda", generator=g).int()
    pos[::7] = -1
    w, svh, gu, dn = r(pairs).abs(), r(E, d).half(), r(S, pairs, 2 * F), r(S, pairs, d)
    svh_gu, suh, tot = r(E, 2 * F).half(), r(E, F).half(), torch.tensor([pairs], dtype=torch.int32, device="cuda")

    def added(t):
        acc = t[0]
        for p in t[1:]:
            acc = acc + p
        return acc[None].contiguous()
    got = []
    for a, b in ((dn, gu), (added(dn), added(gu))):
        slot, act = torch.zeros(M, d, device="cuda"), torch.zeros(pairs, F, dtype=torch.float16, device="cuda")
        dst = CombineDst()
        dst.ranks, dst.rank, dst.rows_cap, dst.dst[0] = 1, 0, M, slot.data_ptr()
        lib.check(L.rx_moe_combine(a.data_ptr(), a.shape[0], pairs, M, d, topk, ids.data_ptr(), w.data_ptr(), pos.data_ptr(), svh.data_ptr(), None,
                                   ctypes.byref(dst), lib.stream_ptr()), "rx_moe_combine")
        lib.check(L.rx_moe_swiglu_rot(b.data_ptr(), b.shape[0], pairs, F, ids.data_ptr(), tot.data_ptr(), svh_gu.data_ptr(), suh.data_ptr(), act.data_ptr(),
                                      lib.stream_ptr()), "rx_moe_swiglu_rot")
        got.append((slot, act))
    for x, y in zip(*got):
        assert torch.isfinite(x.float()).all() and x.abs().max() > 0 and torch.equal(x, y)
