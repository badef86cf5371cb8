"""The prefill forms of the recurrent mixers against the per-row forms: the same bits of states and outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(width, conv, M, ldp, lens, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    proj = torch.zeros(M, ldp, device="cuda")
    proj[:, :width] = r(M, width)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    starts = [sum(lens[:i]) for i in range(len(lens))]
    # sequence 0 starts afresh, the others continue from what the pools hold
    pos = [p + (0 if i == 0 else 7) for i, n in enumerate(lens) for p in range(n)]
    seq = [len(lens) - 1 - i for i, n in enumerate(lens) for _ in range(n)]
    return r, proj, i32(seq), i32(pos), i32(starts), i32(lens), r(len(lens), 3, conv)


@pytest.mark.parametrize("lens", [[1], [3, 1], [16, 4, 5], [33, 2, 17, 1], [64, 7]])
@pytest.mark.parametrize("pad", [0, 1])          # an odd row stride: nothing may be read in vectors then
@pytest.mark.parametrize("kda", [False, True])
def test_delta_prefill_equals_row_form(lens, pad, kda):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    Hk, Hv, D, M = 2, 6, 128, sum(lens)
    C, width = (2 * Hk + Hv) * D, (2 * Hk + 2 * Hv) * D + Hv + (Hv * D if kda else Hv)
    r, proj, seq, pos, st, ln, conv0 = _inputs(width, C, M, width + pad, lens, 3)
    args = (r(C, 4).bfloat16(), r(C).bfloat16(), r(Hv * D if kda else Hv), -r(Hv).abs(), (1 + 0.1 * r(D)).bfloat16())
    s0 = 0.3 * r(len(lens), Hv, D, D)
    got = []
    for y32 in (torch.empty(M * Hv * D, device="cuda"), None):       # with scratch: the split scan; without: the fused one
        conv, pool, out = conv0.clone(), s0.clone(), torch.zeros(M, Hv * D, dtype=torch.bfloat16, device="cuda")
        K.gdn_mixer(proj, M, Hk, Hv, D, seq, pos, st, ln, len(lens), *args, 1e-6, conv, pool, torch.empty(M * C, device="cuda"), out, kda=kda, y32=y32)
        got.append((out, conv, pool))
    for a, b in zip(*got):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)


@pytest.mark.parametrize("lens", [[1], [3, 1], [16, 4, 5], [33, 2, 17, 1], [64, 7]])
@pytest.mark.parametrize("H,G,pad", [(8, 2, 0), (8, 2, 1), (6, 2, 2), (48, 1, 0)])      # groups of 256, 192 and 3072 channels
def test_mamba_prefill_equals_row_form(lens, H, G, pad):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    P, N, M = 64, 128, sum(lens)
    DI = H * P
    C, width = DI + 2 * G * N, 2 * DI + 2 * G * N + H
    r, proj, seq, pos, st, ln, conv0 = _inputs(width, C, M, width + pad, lens, 5)
    args = (0.5 * r(C, 4).bfloat16(), 0.1 * r(C).bfloat16(), r(H) - 2, -r(H).abs(), r(H), (1 + 0.1 * r(DI)).bfloat16())
    s0 = 0.3 * r(len(lens), H, P, N)
    got = []
    for seg in ((st, ln, len(lens)), (None, None, 0)):
        conv, pool, out = conv0.clone(), s0.clone(), torch.zeros(M, DI, dtype=torch.bfloat16, device="cuda")
        K.ssm_mixer(proj, M, H, P, G, N, seq, pos, *seg, *args, 1e-6, conv, pool, torch.empty(M * C, device="cuda"), torch.empty(M * DI, device="cuda"), out)
        got.append((out.float(), conv, pool))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and torch.equal(a, b)


def test_conv_walking_rows_equals_one_row_per_thread():
    """The walking form of the convolution (rows in eighths, taken from 148 blocks on) against the one-row form, which an odd row stride selects:
    bit for bit, over segments that begin inside an eighth, and with the last eighth not full."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    Hk, Hv, D = 16, 48, 128
    lens = [1, 2, 3, 11, 8, 60, 1, 1]
    M, C = sum(lens), (2 * Hk + Hv) * D
    width = (2 * Hk + 2 * Hv) * D + 2 * Hv
    got = []
    for pad in (0, 1):
        r, proj, seq, pos, st, ln, conv0 = _inputs(width, C, M, width + pad, lens, 11)
        args = (r(C, 4).bfloat16(), r(C).bfloat16(), r(Hv), -r(Hv).abs(), (1 + 0.1 * r(D)).bfloat16())
        xbc, out = torch.empty(M * C, device="cuda"), torch.zeros(M, Hv * D, dtype=torch.bfloat16, device="cuda")
        K.gdn_mixer(proj, M, Hk, Hv, D, seq, pos, st, ln, len(lens), *args, 1e-6, conv0, r(len(lens), Hv, D, D), xbc, out,
                    y32=torch.empty(M * Hv * D, device="cuda"))
        got.append((xbc, out, conv0))
    for a, b in zip(*got):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
