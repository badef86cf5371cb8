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
