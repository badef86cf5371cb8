"""The prompt-slice forms of the residual finish and of the plain rotation against the forms of few rows, to the bit: their sums run in the same order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(149, 1152), (150, 2048), (301, 2688), (149, 4992), (600, 5120)])
@pytest.mark.parametrize("norm,rotate,bias", [(True, True, False), (True, True, True), (False, True, False), (True, False, True), (False, False, False)])
def test_finish_of_a_slice_equals_the_general_form(M, N, norm, rotate, bias):
    """A second plane of zeros selects the general form and changes no bit."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    part, svh, b, h0, w, suh = r(2, M, N), r(N).half(), r(N), r(M, N).bfloat16(), (1 + 0.1 * r(N)).bfloat16(), r(N).half()
    part[1] = 0
    got = []
    for S in (1, 2):
        h, xr, xn = h0.clone(), torch.zeros(M + 1, N, dtype=torch.float16, device="cuda"), torch.zeros(M + 1, N, dtype=torch.bfloat16, device="cuda")
        lib.check(lib.load().rx_finish_add_norm_rot(part.data_ptr(), S, M, N, svh.data_ptr(), b.data_ptr() if bias else None, h.data_ptr(),
                                                    w.data_ptr() if norm else None, 1e-6, suh.data_ptr() if rotate else None, xr.data_ptr(), lib.stream_ptr(),
                                                    xn.data_ptr() if norm else None), "rx_finish_add_norm_rot")
        got.append((h, xr, xn))
    for x, y in zip(*got):
        assert torch.isfinite(x.float()).all() and torch.equal(x, y)
    assert not torch.equal(got[0][0], h0) and bool(got[0][1].any()) == rotate and bool(got[0][2].any()) == norm


@pytest.mark.parametrize("M,N", [(8192, 128), (2731, 384), (129, 8192)])
def test_rotation_of_a_slice_equals_its_windows(M, N):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, suh = torch.randn(M, N, device="cuda", generator=g).bfloat16(), torch.randn(N, device="cuda", generator=g).half()
    a, b = (torch.zeros(M + 1, N, dtype=torch.float16, device="cuda") for _ in range(2))
    K.norm_rot_in(x, None, 1e-6, suh, a)
    for r in range(0, M, 64):
        K.norm_rot_in(x[r:r + 64], None, 1e-6, suh, b[r:])
    assert a.abs().max() > 0 and torch.isfinite(a.float()).all() and torch.equal(a, b)


@pytest.mark.parametrize("nq,nkv", [(1, 1), (6, 2), (32, 4), (40, 8), (80, 16)])           # 3 to 112 blocks a row: one to three passes
@pytest.mark.parametrize("qn,kn,bias,axes", [(True, True, False, False), (False, False, True, False), (True, False, True, True), (False, True, False, False)])
def test_rope_of_a_slice_equals_its_windows(nq, nkv, qn, kn, bias, axes):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import lib
    M, N, pages = 601, (nq + 2 * nkv) * 128, 11
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    part, svh, b, wq, wk, inv = r(M, N), r(N).half(), r(N), (1 + 0.1 * r(128)).bfloat16(), (1 + 0.1 * r(128)).bfloat16(), torch.rand(64, device="cuda", generator=g)
    pos, pos3 = torch.arange(7, 7 + M, device="cuda").int(), torch.randint(0, 900, (M, 3), device="cuda", generator=g).int()
    slot = torch.randperm(pages * 64, device="cuda", generator=g)[:M].int()
    slot[::5] = -1                                                                          # rows that are not cached
    p = lambda t, on=True: t.data_ptr() if on else None  # noqa: E731
    got = []
    for step in (M, 100):
        q, kc, vc = (torch.zeros(*s, dtype=torch.bfloat16, device="cuda") for s in ((M + 1, nq * 128), (pages, nkv, 64, 128), (pages, nkv, 64, 128)))
        for r0 in range(0, M, step):
            sec = 16 if axes else 0
            lib.check(lib.load().rx_finish_qkv_rope(p(part[r0:]), 1, min(step, M - r0), nq, nkv, 128, p(svh), p(b, bias), p(wq, qn), p(wk, kn), 1e-6, p(pos[r0:]),
                                                    p(inv), p(slot[r0:]), p(q[r0:]), p(kc), p(vc), lib.stream_ptr(), None, None, p(pos3[r0:], axes), sec, sec, None,
                                                    None, 0), "rx_finish_qkv_rope")
        got.append((q, kc, vc))
    for x, y in zip(*got):
        assert x.abs().max() > 0 and torch.isfinite(x.float()).all() and torch.equal(x, y)
