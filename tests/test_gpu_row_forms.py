"""The row kernels of prompt slices at the ends of the sizes that go by them, against the forms of few rows, to the bit."""
import pytest
import torch

import test_gpu_aux_rows as aux
import test_gpu_moe_rows as moe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(297, 1152), (511, 2048), (593, 2048), (297, 4096)])
def test_residual_finish(M, N):
    aux.test_finish_of_a_slice_equals_the_general_form(M, N, True, True, True)


@pytest.mark.parametrize("nq,nkv", [(1, 1), (6, 1), (4, 2)])
def test_qkv_finish_of_narrow_rows(nq, nkv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    M, N, pages = 901, (nq + 2 * nkv) * 128, 15
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    part, svh, w, inv, pos = r(M, N), r(N).half(), (1 + 0.1 * r(128)).bfloat16(), torch.rand(64, device="cuda", generator=g), torch.arange(7, 7 + M, device="cuda").int()
    slot = torch.randperm(pages * 64, device="cuda", generator=g)[:M].int()
    slot[::5] = -1
    got = []
    for step in (M, 100):
        q, kc, vc = (torch.zeros(*s, dtype=torch.bfloat16, device="cuda") for s in ((M + 1, nq * 128), (pages, nkv, 64, 128), (pages, nkv, 64, 128)))
        for r0 in range(0, M, step):
            lib.check(lib.load().rx_finish_qkv_rope(part[r0:].data_ptr(), 1, min(step, M - r0), nq, nkv, 128, svh.data_ptr(), None, w.data_ptr(), w.data_ptr(), 1e-6,
                                                    pos[r0:].data_ptr(), inv.data_ptr(), slot[r0:].data_ptr(), q[r0:].data_ptr(), kc.data_ptr(), vc.data_ptr(),
                                                    lib.stream_ptr(), None, None, None, 0, 0, None, None, 0), "rx_finish_qkv_rope")
        got.append((q, kc, vc))
    for x, y in zip(*got):
        assert x.abs().max() > 0 and torch.isfinite(x.float()).all() and torch.equal(x, y)


@pytest.mark.parametrize("M,N", [(16385, 128), (5462, 384), (297, 4096)])
def test_plain_rotation(M, N):
    aux.test_rotation_of_a_slice_equals_its_windows(M, N)


@pytest.mark.parametrize("M,topk,d", [(433, 1, 768), (3201, 2, 256), (1601, 3, 512), (801, 10, 1536), (601, 7, 2048)])
@pytest.mark.parametrize("rotated", [True, False])
def test_routed_gather(M, topk, d, rotated):
    moe.test_gather_of_a_slice_equals_its_windows(M, topk, d, rotated)
