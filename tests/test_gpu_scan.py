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


def _fma(a, b, c):
    return (a.double() * b.double() + c.double()).float()        # (one rounding but for cases of 2^-29: products of fp32 are exact in fp64)


def _norm_inv(x):
    s = (x * x).view(4, 32)
    for o in (16, 8, 4, 2, 1):
        s = s[:, :o] + s[:, o:]
    return torch.rsqrt(s[0, 0] + s[1, 0] + s[2, 0] + s[3, 0] + 1e-6)


def _dot(st, x):
    """S.x of every column (st [columns, 128]): per half of the keys four sums over every fourth key, then (0 + 1) + (2 + 3), then the halves."""
    acc = torch.zeros(st.shape[0], 2, 4, device="cuda")
    for i in range(16):
        acc = _fma(st.view(-1, 2, 16, 4)[:, :, i], x.view(2, 16, 4)[:, i], acc)
    s = (acc[..., 0] + acc[..., 1]) + (acc[..., 2] + acc[..., 3])
    return s[:, 0] + s[:, 1]


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("T", [1, 6, 21])
def test_delta_rule_adds_in_its_order(split, T):
    """States and outputs bit for bit as the delta rule in fp32 gives them in the documented order of its sums (no decay, write strength 1)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    D, C = 128, 3 * 128
    r, proj, seq, pos, st, ln, conv = _inputs(D + C + 2, C, T, D + C + 2, [T], T)
    proj[:, D + C] = 60.0                                             # sigmoid -> 1
    pool, xbc, y32 = r(1, D * D), torch.empty(T * C, device="cuda"), torch.zeros(T, D, device="cuda")
    pos += 3                                                          # goes on from the pool
    S = pool.view(8, 16, 16, 2, 4).permute(0, 2, 3, 1, 4).reshape(D, D)   # [column / 16][step][column % 16][half][e] -> [column][key]
    one, zero = torch.ones(1, device="cuda"), torch.zeros(1, device="cuda")
    K.gdn_mixer(proj, T, 1, 1, D, seq, pos, *((st, ln, 1) if split else (None, None, 0)), 0.5 * r(C, 4).bfloat16(), r(C).bfloat16(), one, zero,
                torch.ones(D, dtype=torch.bfloat16, device="cuda"), 1e-6, conv, pool, xbc, torch.zeros(T, D, dtype=torch.bfloat16, device="cuda"),
                y32=y32 if split else None)
    want = []
    for q, k, v in xbc.view(T, 3, D):
        kinv = _norm_inv(k)
        delta = _fma(-_dot(S, k), kinv, v) * kinv
        S = _fma(delta[:, None], k, S)
        want.append(_dot(S, q) * (_norm_inv(q) * 0.08838834764831845))
    assert torch.isfinite(S).all() and torch.equal(pool.view(8, 16, 16, 2, 4).permute(0, 2, 3, 1, 4).reshape(D, D), S)
    if split:
        assert torch.equal(y32, torch.stack(want))


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


@pytest.mark.parametrize("kept", [[1], [4], [1, 4, 2, 0, 3], [9, 1, 1, 0], [5, 3, 5], [17, 16]])       # up to four rows a segment: short chunks
@pytest.mark.parametrize("kind", ["mamba", "delta", "kda"])
def test_commit_equals_row_form(kind, kept):
    """The pools after a commit over the first `kept` rows of a window's segments against those after a direct run of these rows alone."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    lens = [max(1, k) if len(kept) == 4 else k + (i % 2) for i, k in enumerate(kept)]     # some segments lose rows, some lose all
    M, kda = sum(lens), kind == "kda"
    if kind == "mamba":
        H, G = 8, 2
        C, width = H * 64 + 2 * G * 128, 2 * H * 64 + 2 * G * 128 + H
    else:
        H, D = 6, 128
        C, width = (4 + H) * D, (4 + 2 * H) * D + H + (H * D if kda else H)
    r, proj, seq, pos, st, ln, conv0 = _inputs(width, C, M, width, lens, 7)
    if kind == "mamba":
        args = (0.5 * r(C, 4).bfloat16(), 0.1 * r(C).bfloat16(), r(H) - 2, -r(H).abs(), r(H), (1 + 0.1 * r(H * 64)).bfloat16())
        s0 = 0.3 * r(len(lens), H, 64, 128)
    else:
        args = (r(C, 4).bfloat16(), r(C).bfloat16(), r(H * D if kda else H), -r(H).abs(), (1 + 0.1 * r(D)).bfloat16())
        s0 = 0.3 * r(len(lens), H, D, D)

    def run(proj, seq, pos, seg, conv, pool, xbc, mode):
        n, y = proj.shape[0], torch.empty(proj.shape[0] * H * 128, device="cuda")
        out = torch.zeros(n, H * (64 if kind == "mamba" else 128), dtype=torch.bfloat16, device="cuda")
        if kind == "mamba":
            K.ssm_mixer(proj, n, H, 64, G, 128, seq, pos, *seg, *args, 1e-6, conv, pool, xbc, y, out, mode=mode)
        else:
            K.gdn_mixer(proj, n, 2, H, D, seq, pos, *seg, *args, 1e-6, conv, pool, xbc, out, kda=kda, mode=mode, y32=y if seg[0] is not None else None)
    conv, pool, xbc = conv0.clone(), s0.clone(), torch.empty(M * C, device="cuda")
    run(proj, seq, pos, (None, None, 0), conv, pool, xbc, K.SCAN_RECORD)
    assert torch.equal(conv, conv0) and torch.equal(pool, s0)
    run(proj, seq, pos, (st, torch.tensor(kept, dtype=torch.int32, device="cuda"), len(kept)), conv, pool, xbc, K.SCAN_COMMIT)
    rows = torch.tensor([sum(lens[:i]) + t for i, k in enumerate(kept) for t in range(k)], device="cuda")
    conv1, pool1 = conv0.clone(), s0.clone()
    run(proj[rows].contiguous(), seq[rows].contiguous(), pos[rows].contiguous(), (None, None, 0), conv1, pool1, torch.empty(len(rows) * C, device="cuda"), K.SCAN_FINAL)
    assert not torch.equal(pool, s0) and torch.equal(pool, pool1) and torch.equal(conv, conv1)


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


@pytest.mark.parametrize("lens", [[1] * 70, [5] * 16, [2, 1, 4, 3] * 8, [64], [63, 1]])
@pytest.mark.parametrize("record", [False, True])
def test_conv_walking_rows_over_short_segments(lens, record):
    """The same over segments shorter than the convolution, in prompt slices and recorded windows, with sequences that go on from position 1."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from rexl3_b200.ops import kernels as K
    Hk, Hv, D = 16, 48, 128
    M, C = sum(lens), (2 * Hk + Hv) * D
    width = (2 * Hk + 2 * Hv) * D + 2 * Hv
    got = []
    for pad in (0, 1):
        r, proj, seq, pos, st, ln, conv0 = _inputs(width, C, M, width + pad, lens, 11)
        if len(lens) > 1:
            pos = pos - 6 * (seq == 0).int()                          # one sequence goes on from position 1: two of the three before it are zero
        args = (r(C, 4).bfloat16(), r(C).bfloat16(), r(Hv), -r(Hv).abs(), (1 + 0.1 * r(D)).bfloat16())
        xbc, out = torch.empty(M * C, device="cuda"), torch.zeros(M, Hv * D, dtype=torch.bfloat16, device="cuda")
        seg = (None, None, 0) if record else (st, ln, len(lens))
        K.gdn_mixer(proj, M, Hk, Hv, D, seq, pos, *seg, *args, 1e-6, conv0, r(len(lens), Hv, D, D), xbc, out,
                    y32=torch.empty(M * Hv * D, device="cuda"), mode=K.SCAN_RECORD if record else K.SCAN_FINAL)
        got.append((xbc, out, conv0))
    for a, b in zip(*got):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b)
