"""The prompt-slice forms of the routed experts' kernels against the window forms, to the bit: their sums run in the same order."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [2047, 2048, 2049, 8193])
@pytest.mark.parametrize("E,lo,hi", [(1, 0, 1), (128, 32, 96), (512, 0, 512)])
def test_plan_of_a_cluster_is_a_stable_sort(pairs, E, lo, hi):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    rng = np.random.default_rng(pairs + E)
    ids = rng.integers(-1, E, size=pairs).astype(np.int32)
    ids[rng.random(pairs) < 0.3] = lo
    own = (ids >= lo) & (ids < hi)
    order = [int(p) for p in np.argsort(np.where(own, ids, E), kind="stable")[:own.sum()]]
    cnt = np.bincount(ids[own], minlength=E)
    tiles = [[e, int(cnt[:e].sum()) + r, int(min(32, cnt[e] - r))] for e in range(E) for r in range(0, int(cnt[e]), 32)]
    d_ids = torch.from_numpy(ids).cuda()
    z = lambda n: torch.full((n,), -7, dtype=torch.int32, device="cuda")  # noqa: E731
    offs, pos, pair, exp, tab, tot = z(E + 1), z(pairs), z(pairs), z(pairs), z(3 * len(tiles) + 3), z(1)
    lib.check(lib.load().rx_moe_plan(d_ids.data_ptr(), pairs, E, lo, hi, 32, len(tiles) + 1, offs.data_ptr(), pos.data_ptr(), pair.data_ptr(), exp.data_ptr(),
                                     tab.data_ptr(), tot.data_ptr(), lib.stream_ptr()), "rx_moe_plan")
    want = np.full(pairs, -1)
    want[order] = np.arange(len(order))
    assert tot.item() == len(order) and offs.tolist() == [0] + np.cumsum(cnt).tolist() and pos.tolist() == want.tolist()
    assert pair[:len(order)].tolist() == order and exp[:len(order)].tolist() == ids[order].tolist()
    assert tab.view(-1, 3).tolist() == tiles + [[0, 0, 0]]


@pytest.mark.parametrize("M,topk,d", [(1281, 1, 256), (430, 10, 768), (165, 7, 2048)])
@pytest.mark.parametrize("rotated", [True, False])
def test_gather_of_a_slice_equals_its_windows(M, topk, d, rotated):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    L, E, pairs = lib.load(), 9, M * topk
    g = torch.Generator(device="cuda").manual_seed(M)
    x, suh = torch.randn(M, d, device="cuda", generator=g).bfloat16(), torch.randn(E, d, device="cuda", generator=g).half()
    ids = torch.randint(0, E, (pairs,), device="cuda", generator=g).int()
    pos = torch.randperm(pairs, device="cuda", generator=g).int()
    pos[::7] = -1
    pos[3 * topk:40 * topk] = -1                                                     # whole warps without a pair of this rank
    s = suh.data_ptr() if rotated else None
    a, b = torch.zeros(pairs, d, dtype=torch.float16, device="cuda"), torch.zeros(pairs, d, dtype=torch.float16, device="cuda")
    n = pairs - (topk > 1)                                                           # a last row with a slot less
    lib.check(L.rx_moe_gather_rot(x.data_ptr(), ids.data_ptr(), pos.data_ptr(), n, topk, d, s, a.data_ptr(), lib.stream_ptr()), "rx_moe_gather_rot")
    for r in range(0, M, 16):
        o = r * topk
        lib.check(L.rx_moe_gather_rot(x[r:].data_ptr(), ids[o:].data_ptr(), pos[o:].data_ptr(), min(n - o, 16 * topk), topk, d, s, b.data_ptr(), lib.stream_ptr()),
                  "rx_moe_gather_rot")
    assert a.abs().max() > 0 and torch.isfinite(a.float()).all() and torch.equal(a, b)


@pytest.mark.parametrize("M,topk,d,F", [(641, 1, 128, 128), (833, 5, 384, 384), (300, 17, 2048, 1408)])
@pytest.mark.parametrize("rotated", [True, False])
def test_finish_of_a_slice_equals_the_general_form(M, topk, d, F, rotated):
    """A second plane of zeros selects the general form and changes no bit."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.models.moe import CombineDst
    from rexl3_b200.ops import lib
    L, E, pairs = lib.load(), 24, M * topk
    g = torch.Generator(device="cuda").manual_seed(M)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    ids = torch.randint(0, E, (pairs,), device="cuda", generator=g).int()
    pos = torch.randperm(pairs, device="cuda", generator=g).int()
    pos[::7] = -1
    w, svh, gu, dn, shared = r(pairs).abs(), r(E, d).half(), r(2, pairs, 2 * F), r(2, pairs, d), r(M, d)
    gu[1], dn[1] = 0, 0
    svh_gu, suh, tot = r(E, 2 * F).half(), r(E, F).half(), torch.tensor([pairs - 3], dtype=torch.int32, device="cuda")
    p = lambda t: t.data_ptr() if rotated else None  # noqa: E731
    got = []
    for S in (1, 2):
        slot, act = torch.zeros(2, M + 1, d, device="cuda"), torch.zeros(pairs, F, dtype=torch.float16, device="cuda")
        dst = CombineDst()
        dst.ranks, dst.rank, dst.rows_cap, dst.dst[0] = 1, 0, M + 1, slot.data_ptr()
        lib.check(L.rx_moe_combine(dn.data_ptr(), S, pairs, M, d, topk, ids.data_ptr(), w.data_ptr(), pos.data_ptr(), p(svh), shared.data_ptr(),
                                   ctypes.byref(dst), lib.stream_ptr()), "rx_moe_combine")
        lib.check(L.rx_moe_swiglu_rot(gu.data_ptr(), S, pairs, F, ids.data_ptr(), tot.data_ptr(), p(svh_gu), p(suh), act.data_ptr(), lib.stream_ptr()),
                  "rx_moe_swiglu_rot")
        got.append((slot, act))
    for x, y in zip(*got):
        assert torch.isfinite(x.float()).all() and x.abs().max() > 0 and torch.equal(x, y)
    assert got[0][1][pairs - 3:].abs().max() == 0
