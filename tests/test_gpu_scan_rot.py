"""The recurrent mixers with the next projection's input rotation against the mixer and the rotation kernel one after the other, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(width, C, lens, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    starts = [sum(lens[:i]) for i in range(len(lens))]
    seq = i32([i for i, n in enumerate(lens) for _ in range(n)])
    pos = i32([5 + t for n in lens for t in range(n)])
    return r, r(sum(lens), width), seq, pos, (i32(starts), i32(lens), len(lens)), r(len(lens), C, 3)


@pytest.mark.parametrize("segments", [True, False])
@pytest.mark.parametrize("lens", [[1], [1, 1, 1], [7, 1, 40]])
@pytest.mark.parametrize("H,G", [(2, 1), (16, 2), (32, 1)])           # groups of 128, 512 and 2048 channels: the last beyond what a thread keeps
def test_mamba_rows_leave_rotated(H, G, lens, segments):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    P, N, M = 64, 128, sum(lens)
    DI = H * P
    C, width = DI + 2 * G * N, 2 * DI + 2 * G * N + H
    r, proj, seq, pos, seg, conv0 = _inputs(width, C, lens, H)
    args = (0.5 * r(C, 4).bfloat16(), 0.1 * r(C).bfloat16(), r(H) - 2, -r(H).abs(), r(H), (1 + 0.1 * r(DI)).bfloat16())
    s0, suh, got = 0.3 * r(len(lens), H, P, N), r(DI).half(), []
    for fused in (False, True):
        out, xr = torch.zeros(M, DI, dtype=torch.bfloat16, device="cuda"), torch.zeros(M, DI, dtype=torch.float16, device="cuda")
        conv, pool = conv0.clone(), s0.clone()
        K.ssm_mixer(proj, M, H, P, G, N, seq, pos, *(seg if segments else (None, None, 0)), *args, 1e-6, conv, pool, torch.empty(M * C, device="cuda"),
                    torch.empty(M * DI, device="cuda"), out, rot=(suh, xr) if fused else None)
        if not fused:
            K.norm_rot_in(out, None, 1e-6, suh, xr)
        got.append((xr, conv, pool))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and a.abs().max() > 0 and torch.equal(a, b)


@pytest.mark.parametrize("segments", [True, False])
@pytest.mark.parametrize("lens", [[1], [1, 1, 1], [7, 1, 40]])
@pytest.mark.parametrize("Hk,Hv", [(1, 1), (2, 6), (3, 9)])
@pytest.mark.parametrize("kda", [False, True])
def test_delta_rows_leave_rotated(kda, Hk, Hv, lens, segments):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    D, M = 128, sum(lens)
    C, width = (2 * Hk + Hv) * D, (2 * Hk + 2 * Hv) * D + Hv + (Hv * D if kda else Hv)
    r, proj, seq, pos, seg, conv0 = _inputs(width, C, lens, Hv)
    args = (r(C, 4).bfloat16(), r(C).bfloat16(), r(Hv * D if kda else Hv), -r(Hv).abs(), (1 + 0.1 * r(D)).bfloat16())
    s0, suh, got = 0.3 * r(len(lens), Hv, D, D), r(Hv * D).half(), []
    for fused in (False, True):
        out, xr = torch.zeros(M, Hv * D, dtype=torch.bfloat16, device="cuda"), torch.zeros(M, Hv * D, dtype=torch.float16, device="cuda")
        conv, pool = conv0.clone(), s0.clone()
        K.gdn_mixer(proj, M, Hk, Hv, D, seq, pos, *(seg if segments else (None, None, 0)), *args, 1e-6, conv, pool, torch.empty(M * C, device="cuda"), out, kda=kda,
                    y32=torch.empty(M * Hv * D, device="cuda") if segments else None, rot=(suh, xr) if fused else None)
        if not fused:
            K.norm_rot_in(out, None, 1e-6, suh, xr)
        got.append((xr, conv, pool))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and a.abs().max() > 0 and torch.equal(a, b)
