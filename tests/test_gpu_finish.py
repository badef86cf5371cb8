"""The finish kernels' forms for many rows against their forms for few: a row's bits do not depend on the rows beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weight(N, g):
    from rexl3_b200.ops import kernels as K
    tr = torch.zeros(8, N // 16, 64, dtype=torch.int16, device="cuda")
    return K.Exl3Weight(tr, torch.ones(128, dtype=torch.float16, device="cuda"), (0.1 * torch.randn(N, device="cuda", generator=g)).half(),
                        torch.randn(N, device="cuda", generator=g))


@pytest.mark.parametrize("N", [128, 1024, 1152, 5120, 5248])       # up to five blocks a warp take the row form, one more does not
@pytest.mark.parametrize("norm", [False, True])
def test_add_norm_rot_rows_do_not_depend_on_their_number(N, norm):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    M, w = 523, _weight(N, g)
    part, h0, nw, suh = r(M, N), r(M, N).bfloat16(), (1 + 0.1 * r(N)).bfloat16() if norm else None, r(N).half()
    whole = [h0.clone(), torch.zeros(M, N, dtype=torch.float16, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")]
    K.finish_add_norm_rot(part, 1, M, w, whole[0], nw, 1e-6, suh, whole[1], whole[2])
    cut = [h0.clone(), torch.zeros_like(whole[1]), torch.zeros_like(whole[2])]
    for a, b in ((0, 511), (511, M)):
        K.finish_add_norm_rot(part[a:b], 1, b - a, w, cut[0][a:b], nw, 1e-6, suh, cut[1][a:b], cut[2][a:b])
    for x, y in zip(whole, cut):
        assert torch.isfinite(x.float()).all() and torch.equal(x, y)
    H = torch.tensor([[1.0 - 2 * (bin(i & j).count("1") & 1) for j in range(128)] for i in range(128)], device="cuda").double() / 128 ** 0.5
    y = (part.double().view(M, -1, 128) @ H).view(M, N) * w.svh.double() + w.bias.double() + h0.double()
    assert (whole[0].double() - y).abs().max() <= 2.0 ** -8 * y.abs().max() + 1e-5      # one rounding to bf16


@pytest.mark.parametrize("M,N", [(592, 5120), (593, 3072), (593, 5120), (601, 4224), (593, 5248), (2048, 2048), (2049, 1152), (2049, 2048), (2049, 1024)])
def test_add_norm_rot_at_the_edges_of_the_row_form(M, N):
    """Both sides of every bound of the row form: the same bits as in calls of few rows."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    w, part, h0, nw, suh = _weight(N, g), r(M, N), r(M, N).bfloat16(), (1 + 0.1 * r(N)).bfloat16(), r(N).half()
    got = []
    for step in (M, 300):
        out = [h0.clone(), torch.zeros(M, N, dtype=torch.float16, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")]
        for a in range(0, M, step):
            b = min(M, a + step)
            K.finish_add_norm_rot(part[a:b], 1, b - a, w, out[0][a:b], nw, 1e-6, suh, out[1][a:b], out[2][a:b])
        got.append(out)
    for x, y in zip(*got):
        assert torch.isfinite(x.float()).all() and torch.equal(x, y)


@pytest.mark.parametrize("N", [128, 640, 3968, 4096, 5120, 8192, 8320])     # clusters: up to 16 rows below 4096, up to 64 from there to 8192
@pytest.mark.parametrize("S", [1, 7, 18])
@pytest.mark.parametrize("norm,rot,xn", [(True, True, True), (False, True, False), (True, False, True), (True, False, False)])
def test_add_norm_rot_of_few_rows(N, S, norm, rot, xn):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(N + S)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    M, w = 146, _weight(N, g)
    part, h0, nw, suh = r(S, M, N), r(M, N).bfloat16(), (1 + 0.1 * r(N)).bfloat16() if norm else None, r(N).half() if rot else None

    def run(*cuts):
        out = [h0.clone(), torch.zeros(M, N, dtype=torch.float16, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")]
        for a, b in zip(cuts, cuts[1:]):
            o = [t[a:b] for t in out]
            K.finish_add_norm_rot(part[:, a:b].contiguous(), S, b - a, w, o[0], nw, 1e-6, suh, o[1], o[2] if xn else None)
        return out
    for x, y in zip(run(0, M), run(0, 1, 17, 81, M)):
        assert torch.isfinite(x.float()).all() and torch.equal(x, y)


@pytest.mark.parametrize("M", [1, 16, 37, 64, 65, 523])               # clusters, one CTA a row, the row form
@pytest.mark.parametrize("N", [640, 2048, 5120])
def test_add_norm_rot_rounds_as_norm_rot_in(M, N):
    """Residual rows of powers of two have the same sum of squares in any order; the rotated rows are then those of norm_rot_in, bit for bit, also
    for input scales that are not +-1."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = _weight(N, g)
    w.bias = None
    h = torch.exp2(torch.randint(-2, 3, (M, N), device="cuda", generator=g).float()).bfloat16()
    nw, suh = (1 + 0.1 * torch.randn(N, device="cuda", generator=g)).bfloat16(), torch.randn(N, device="cuda", generator=g).half()
    xr, want = (torch.zeros(M, N, dtype=torch.float16, device="cuda") for _ in range(2))
    K.norm_rot_in(h, nw, 1e-6, suh, want)
    K.finish_add_norm_rot(torch.zeros(2, M, N, device="cuda"), 2 if M < 512 else 1, M, w, h.clone(), nw, 1e-6, suh, xr)
    assert torch.isfinite(xr).all() and xr.abs().max() > 0 and torch.equal(xr, want)


@pytest.mark.parametrize("hd,n_q,n_kv", [(128, 40, 8), (128, 3, 1), (64, 4, 2)])
def test_qkv_rope_rows_do_not_depend_on_their_number(hd, n_q, n_kv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(hd + n_q)
    N, M = (n_q + 2 * n_kv) * hd, 1030
    w = _weight(N, g)
    part = torch.randn(M, N, device="cuda", generator=g)
    pos = torch.arange(5, 5 + M, dtype=torch.int32, device="cuda")
    inv = (1e6 ** (-torch.arange(0, hd, 2, device="cuda") / hd)).float()
    slot = torch.randperm(1088, device="cuda", generator=g)[:M].int()

    def run(a, b, q, k, v):
        K.finish_qkv_rope(part[a:b], 1, b - a, n_q, n_kv, hd, w, None, None, 1e-6, pos[a:b], inv, slot[a:b], q[a:b], k, v)
    got = []
    for cuts in ((0, M), (0, 7, 600, M)):
        out = [torch.zeros(M, n_q * hd, dtype=torch.bfloat16, device="cuda")] + [torch.zeros(17, n_kv, 64, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        for a, b in zip(cuts, cuts[1:]):
            run(a, b, *out)
        got.append(out)
    for x, y in zip(*got):
        assert torch.isfinite(x.float()).all() and x.float().abs().max() > 0 and torch.equal(x, y)
