"""What is timed: one model call of an engine that serves EXL3 checkpoints, as the serving backend makes it.

A case is either one decode / verify window (`mode` "step": every sequence feeds `rows` tokens over `ctx` cached ones, replayed from a CUDA graph
as the backend does) or one prompt slice (`mode` "prefill": prompts of the lengths `len_lo` .. `len_hi` over `ctx` cached tokens, launched directly).
The models are the repository's own configurations cut in depth (and, with the depth, in vocabulary, so that the head keeps the few per cent of a
step that it has in the whole model); layer widths, head counts, code widths and cache formats are the configurations' own.  Weights and
caches are random: any bit ring is a valid trellis, and keys and queries of unit variance give attention rows that are neither flat nor one-hot.
"""
import dataclasses
import math

import torch

from rexl3_b200.models import dense, hybrid, moe

PAGE = 64
VOCAB = 32768

# name of the model -> (configuration, executor class)
MODELS = {
    "dense": (dense.CONFIGS["dense-27b"], dense.DenseGPU),
    "gdn": (hybrid.CONFIGS["gdn-hybrid-27b"], hybrid.HybridGPU),
    "mamba": (hybrid.CONFIGS["hybrid-h-56l"], hybrid.HybridGPU),
    "moe": (dense.CONFIGS["moe-spec-30b"], moe.MoEGPU),
}


def _case(name, model, mode, layers, seqs, rows, ctx, len_lo=0, len_hi=0, kv="bf16"):
    c = {"model": model, "mode": mode, "layers": layers, "seqs": seqs, "rows": rows, "ctx": ctx, "len_lo": len_lo, "len_hi": len_hi, "kv": kv}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # one user, short conversation: nothing but latency, launches and the weight stream
        _case("dense_step_1", "dense", "step", 8, 1, 1, 937),
        # the throughput point of a loaded server: 64 sequences at 8K, bound by the cache
        _case("dense_step_64_8k", "dense", "step", 4, 64, 1, 8192),
        # speculative verify windows: 16 sequences with 4 drafts each
        _case("dense_window_16x5", "dense", "step", 8, 16, 5, 3001),
        # long conversations on the byte-wide cache
        _case("dense_step_fp8_32k", "dense", "step", 4, 6, 1, 32100, kv="fp8"),
        # time to first token of a long prompt
        _case("dense_prefill_8k", "dense", "prefill", 4, 1, 0, 0, 8192, 8192),
        # a burst of short chat prompts of odd lengths over a cached system prompt, one slice
        _case("dense_prefill_ragged", "dense", "prefill", 4, 7, 0, 333, 61, 411),
        # routed experts, decode and prompt
        _case("moe_step_16", "moe", "step", 4, 16, 1, 2050),
        _case("moe_prefill_2k", "moe", "prefill", 2, 3, 0, 0, 500, 900),
        # delta-net hybrid: decode of a small batch, prompt slice
        _case("gdn_step_16", "gdn", "step", 8, 16, 1, 1501),
        _case("gdn_prefill_2k", "gdn", "prefill", 4, 2, 0, 0, 900, 1148),
        # Mamba2 hybrid: one user, prompt slice
        _case("mamba_step_1", "mamba", "step", 7, 1, 1, 700),
        _case("mamba_prefill_2k", "mamba", "prefill", 7, 1, 0, 0, 2047, 2047),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["dense", "dense", "dense", "dense", "moe", "gdn", "mamba"])
    if rng.random() < 0.55:                                  # a window: plain decode, or verify with up to 7 drafts
        layers = {"dense": 4, "moe": 4, "gdn": 4, "mamba": 7}[model]
        rows = rng.choice([1, 1, 1, log(2, 8)]) if model in ("dense", "moe") else 1
        seqs = log(1, min(64, 256 // rows))
        top = min(32768, 524288 // seqs) if model == "dense" else min(8192, 131072 // seqs)
        return _case(None, model, "step", layers, seqs, rows, log(20, top), kv=rng.choice(["bf16", "bf16", "fp8"]) if model == "dense" else "bf16")
    seqs = log(1, 8)
    total = log(64, 8192 if model == "dense" else 2048)
    mean = max(2, total // seqs)
    spread = rng.uniform(0.0, 0.6)
    lo, hi = max(1, int(mean * (1 - spread))), max(1, int(mean * (1 + spread)))
    ctx = 0 if model in ("gdn", "mamba") else rng.choice([0, 0, log(1, 2000)])
    # every recurrent prompt starts at 0, as a new request does
    hi = min(hi, (6000 if ctx else 8192) // seqs)
    return _case(None, model, "prefill", 7 if model == "mamba" else 2 if model == "moe" else 4, seqs, 0, ctx, min(lo, hi), hi)


def _config(case):
    cfg = MODELS[case["model"]][0]
    cut = {"n_layers": case["layers"], "vocab": VOCAB}
    if hasattr(cfg, "pattern"):
        cut["pattern"] = cfg.pattern[:case["layers"]]
    return dataclasses.replace(cfg, **cut)


def _lengths(case):
    """New tokens of every sequence of the call."""
    n, lo, hi = case["seqs"], case["len_lo"], case["len_hi"]
    if case["mode"] == "step":
        return [case["rows"]] * n
    return [lo + (hi - lo) * i // max(1, n - 1) for i in range(n)]


def _contexts(case):
    """Cached tokens of every sequence before the call: around `ctx`, no two alike where there are several."""
    n, c = case["seqs"], case["ctx"]
    return [c - (c // 8) * i // n if n > 1 else c for i in range(n)]


def prepare(case, seed):
    dev = "cuda"
    cfg, cls = _config(case), MODELS[case["model"]][1]
    lens, ctx = _lengths(case), _contexts(case)
    n, M = case["seqs"], sum(_lengths(case))
    blocks = [(c + l + PAGE - 1) // PAGE for c, l in zip(ctx, lens)]
    kw = {} if case["kv"] == "bf16" else {"kv_dtype": case["kv"]}
    step = case["mode"] == "step"
    m = cls(cfg, num_pages=sum(blocks), max_rows=256, max_seqs=n, max_blocks_per_seq=max(blocks), max_prefill_rows=256 if step else M, seed=seed, **kw)
    for L in m.layers:
        if "router" in L:
            # a trained router is decisive; of a random one every few rows have two experts tied for the last place, at an eighth of the row's weight
            L["router"].mul_(4.0)
    g = torch.Generator(device=dev).manual_seed(seed * 3 + 1)
    h = torch.Generator().manual_seed(seed * 3 + 2)
    order = torch.randperm(sum(blocks), generator=h).tolist()            # pages of a served cache lie anywhere
    bt = torch.zeros(n, max(blocks), dtype=torch.int32)
    ids, pos, slot, row_seq = [], [], [], []
    first = 0
    for i in range(n):
        pages = order[first:first + blocks[i]]
        first += blocks[i]
        bt[i, :len(pages)] = torch.tensor(pages, dtype=torch.int32)
        p = list(range(ctx[i], ctx[i] + lens[i]))
        pos += p
        slot += [pages[x // PAGE] * PAGE + x % PAGE for x in p]
        row_seq += [i] * lens[i]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    ids = torch.randint(0, cfg.vocab, (M,), dtype=torch.int32, device=dev, generator=g)
    rows = (ids, i32(pos), i32(slot), i32(row_seq), i32([p + 1 for p in pos]), bt.to(dev))
    s = {"model": m, "cfg": cfg, "rows": rows, "lens": lens, "ctx": ctx, "bt": bt, "step": step}
    if step:
        m.window_seq_rows = max(lens)
        top = max(c + l for c, l in zip(ctx, lens))
        s["max_ctx"] = min(m.max_ctx_alloc, (top + 2047) // 2048 * 2048)
        _window(s)                                                        # warm-up before the capture, as the backend does it
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            s["out"] = _window(s)
        s["graph"] = graph
    else:
        starts = [sum(lens[:i]) for i in range(n)]
        s["prefill"] = dict(seq_ids=i32(list(range(n))), q_start=i32(starts), q_len=i32(lens), pos0=i32(ctx), nseq=n, max_qlen=max(lens))
        s["last"] = torch.tensor([a + l - 1 for a, l in zip(starts, lens)], dtype=torch.long, device=dev)
    # what earlier calls left behind: cached keys and values, recurrent states
    for c in m.k_cache + m.v_cache:
        if c is not None:
            for p in range(0, c.shape[0], 1024):
                x = torch.randn(c[p:p + 1024].shape, device=dev, generator=g)
                c[p:p + 1024] = x.to(torch.float8_e4m3fn).view(torch.uint8) if c.dtype == torch.uint8 else x.to(c.dtype)
    for li in getattr(m, "ssm_pool", {}):
        m.conv_pool[li].normal_(generator=g)
        m.ssm_pool[li].normal_(std=0.1, generator=g)
    return s


def _window(s):
    m = s["model"]
    logits = m.forward_rows(*s["rows"], max_ctx=s["max_ctx"])
    return logits, m.candidates(logits, 16)


def _outputs(s, logits, values):
    """Logits, the candidates' values (their ids are left out: two of nearly the same logit change places with the order of any sum) and the
    state that the call has moved on: the caches, the recurrent pools."""
    m = s["model"]
    out = {"logits": logits, "values": values, "k": [c for c in m.k_cache if c is not None], "v": [c for c in m.v_cache if c is not None]}
    if getattr(m, "ssm_pool", None):
        out["conv"] = [m.conv_pool[li] for li in sorted(m.conv_pool)]
        out["state"] = [m.ssm_pool[li] for li in sorted(m.ssm_pool)]
    return out


def run(s):
    m = s["model"]
    if s["step"]:
        s["graph"].replay()
        logits, (_, values) = s["out"]
    else:
        logits = m.forward_rows(*s["rows"], prefill=s["prefill"], logit_rows=s["last"])
        _, values = m.candidates(logits, 16)
    return _outputs(s, logits, values)


def work(case):
    """Bytes: every weight a row of the call can need read once (of the experts, those that uniform picks hit on average), every cached row of the
    sequences read once, new rows and states and logits written once.  Operations: two per weight and row, four per head element and key."""
    cfg = _config(case)
    lens, ctx = _lengths(case), _contexts(case)
    M, n = sum(lens), case["seqs"]
    R = M if case["mode"] == "step" else n                               # rows with logits
    d, hd, F = cfg.d_model, cfg.head_dim, cfg.ffn_padded
    pattern = getattr(cfg, "pattern", "") or "A" * cfg.n_layers
    wbytes = wflops = kv = att = state = 0.0
    esz = 1 if case["kv"] == "fp8" else 2
    for kind in pattern:
        if kind == "A":
            p = d * cfg.qkv_width + cfg.n_q * hd * d
            kv += 2 * cfg.n_kv * hd * esz * sum(c + 2 * l if l < 64 else c + l for c, l in zip(ctx, lens))
            att += sum(4.0 * cfg.n_q * hd * (l * c + l * (l + 1) / 2) for c, l in zip(ctx, lens))
        elif kind == "G":
            p = d * cfg.gdn_proj_width + cfg.gdn_inner * d
            state += 8.0 * n * (cfg.gdn_v_heads * 128 * 128 + 3 * cfg.gdn_conv_channels)
            att += 6.0 * M * cfg.gdn_v_heads * 128 * 128
        else:
            p = d * cfg.in_proj_width + cfg.d_inner * d
            state += 8.0 * n * (cfg.ssm_heads * cfg.ssm_head_dim * cfg.ssm_state + 3 * cfg.conv_channels)
            att += 5.0 * M * cfg.ssm_heads * cfg.ssm_head_dim * cfg.ssm_state
        wflops += 2.0 * M * p
        if case["model"] == "moe":
            one = 3 * d * cfg.expert_ffn
            hit = cfg.n_experts * (1 - (1 - cfg.top_k / cfg.n_experts) ** M)
            wbytes += (p + hit * one) * cfg.bits / 8 + cfg.n_experts * d * 2
            wflops += 2.0 * M * cfg.top_k * one
        else:
            wbytes += (p + 3 * d * F) * cfg.bits / 8
            wflops += 2.0 * M * 3 * d * F
    head = d * cfg.vocab_padded
    return {"bytes": wbytes + head * cfg.bits / 8 + kv + state + M * d * 2 + R * cfg.vocab_padded * 4.0, "flops": wflops + 2.0 * R * head + att}


def tolerance(case):
    # bf16 residual rows and cache rows: logits of 4 to 8 layers stand 0.7 % to 1.2 % off exact(), each way of rounding on its own side of it;
    # bytes of an E4M3 cache: only the call's own rows may round the other way
    return {"rel": 0.02, "max": 0.5, "differ": 0.002}


# ------------------------------------------------------------------------------------------------ the same call in 64 bits
def _codebook(name):
    s = torch.arange(65536, dtype=torch.int64, device="cuda")
    assert name == "3inst"
    x = (s * 89226354 + 64248484) & 0xFFFFFFFF
    x = (x & 0x8FFF8FFF) ^ 0x3B603B60
    half = lambda v: v.to(torch.int32).to(torch.int16).view(torch.float16).double()  # noqa: E731
    sgn = lambda v: torch.where(v >= 32768, v - 65536, v)  # noqa: E731
    return (half(sgn(x & 0xFFFF)) + half(sgn(x >> 16))).to(torch.float16).double()


def _unpack(trellis, table):
    """int16 [K/16, N/16, 16 bits] -> the coded matrix, float64 [K, N]: value p of a tile is the 16-bit window that ends at bit (p + 1) * bits of its ring."""
    kt, nt, words = trellis.shape
    bits = words // 16
    assert words == 16 * bits
    p = torch.arange(256, device="cuda")
    ring = 256 * bits
    start = (p + 1) * bits + ring - 16
    lane, j = p // 8, p % 8
    r, c = 2 * (lane % 4) + (j & 1) + 8 * ((j >> 1) & 1), lane // 4 + 8 * (j >> 2)
    back = torch.empty(256, dtype=torch.long, device="cuda")
    back[r * 16 + c] = p
    start = start[back]                                                  # row-major order of the tile
    i0, off = (start // 32) % (ring // 32), start % 32
    i1 = (i0 + 1) % (ring // 32)
    out = torch.empty(kt * 16, nt * 16, dtype=torch.float64, device="cuda")
    for k in range(0, kt, 32):
        u = trellis[k:k + 32].to(torch.int64) & 0xFFFF
        w = u[..., 0::2] | (u[..., 1::2] << 16)
        # the window out of two neighbouring 32-bit words, without the sign of a full 64-bit pair
        hi, lo = w[..., i0], w[..., i1]
        st = torch.where(off <= 16, (hi >> (16 - off).clamp(min=0)) & 0xFFFF, ((hi << (off - 16).clamp(min=0)) | (lo >> (48 - off).clamp(max=32))) & 0xFFFF)
        a = st.shape[0]
        out[k * 16:(k + a) * 16] = table[st].view(a, nt, 16, 16).transpose(1, 2).reshape(a * 16, nt * 16)
    return out


class _Exact:
    def __init__(self, s):
        self.s, self.m, self.cfg = s, s["model"], s["cfg"]
        self.table = _codebook(self.cfg.codebook)
        i = torch.arange(128, device="cuda")
        pc = sum(((i[:, None] & i[None, :]) >> b) & 1 for b in range(7)) & 1
        self.H = (1.0 - 2.0 * pc.double()) / math.sqrt(128.0)

    def rot(self, x):
        return (x.reshape(-1, 128) @ self.H).reshape(x.shape)

    def linear(self, x, trellis, suh, svh):
        K, N = trellis.shape[0] * 16, trellis.shape[1] * 16
        xr = self.rot(x * suh.double())
        y = torch.empty(x.shape[0], N, dtype=torch.float64, device="cuda")
        for n in range(0, N, 4096):
            y[:, n:n + 4096] = xr @ _unpack(trellis[:, n // 16:(n + 4096) // 16], self.table)
        return self.rot(y) * svh.double()

    def lin(self, x, w):
        return self.linear(x, w.trellis, w.suh, w.svh)

    def norm(self, x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + self.cfg.eps) * w.double()

    def rope(self, x, pos):
        ang = pos.double()[:, None] * self.m.inv_freq.double()[None]
        cos, sin = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
        a, b = x.chunk(2, -1)
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def attention(self, li, L, x):
        cfg, s = self.cfg, self.s
        hd, T = cfg.head_dim, x.shape[0]
        y = self.lin(x, L["qkv"])
        q, k, v = (t.reshape(T, -1, hd) for t in y.split([cfg.n_q * hd, cfg.n_kv * hd, cfg.n_kv * hd], 1))
        pos, slot = s["rows"][1].long(), s["rows"][2].long()
        q, k = self.rope(q, pos), self.rope(k, pos)
        whole = []
        for new, cache in ((k, self.m.k_cache[li]), (v, self.m.v_cache[li])):
            c = (cache.view(torch.float8_e4m3fn) if cache.dtype == torch.uint8 else cache).float()
            c[slot // PAGE, :, slot % PAGE] = new.float()
            whole.append(c)
        kc, vc = whole
        out, a = torch.empty(T, cfg.n_q, hd, dtype=torch.float64, device="cuda"), 0
        for i, (n, c) in enumerate(zip(s["lens"], s["ctx"])):
            pages = s["bt"][i, :(c + n + PAGE - 1) // PAGE].long().cuda()
            kk, vv = (t[pages].transpose(1, 2).reshape(-1, cfg.n_kv, hd)[:c + n].double() for t in (kc, vc))
            kk[c:], vv[c:] = k[a:a + n], v[a:a + n]                      # this call's own rows, before they are rounded to the cache's type
            kp = torch.arange(c + n, device="cuda")
            for b in range(0, n, 512):
                e = min(n, b + 512)
                qq = q[a + b:a + e].reshape(e - b, cfg.n_kv, -1, hd)
                sc = torch.einsum("tkgd,skd->kgts", qq, kk[:c + e]) / math.sqrt(hd)
                sc.masked_fill_(kp[None, :c + e] > (c + torch.arange(b, e, device="cuda"))[:, None], float("-inf"))
                out[a + b:a + e] = torch.einsum("kgts,skd->tkgd", torch.softmax(sc, -1), vv[:c + e]).reshape(e - b, cfg.n_q, hd)
            a += n
        return self.lin(out.reshape(T, -1), L["o"]), kc, vc

    def conv(self, L, x, hist, DI):
        """Causal depthwise convolution of width 4 with SiLU per sequence; returns the rows and each sequence's last three inputs."""
        w, b, out, left, a = L["conv_w"].double(), L["conv_b"].double(), torch.empty_like(x), torch.zeros_like(hist), 0
        for i, n in enumerate(self.s["lens"]):
            h = hist[i].double() if self.s["ctx"][i] else torch.zeros_like(hist[i]).double()
            full = torch.cat([h, x[a:a + n]])
            y = b[None] + sum(w[:, j][None] * full[j:j + n] for j in range(4))
            out[a:a + n] = y * torch.sigmoid(y)
            left[i] = full[-3:]
            a += n
        return out, left

    def delta(self, li, L, x):
        cfg, lens, ctx, D = self.cfg, self.s["lens"], self.s["ctx"], 128
        Hk, Hv, DI, C, T = cfg.gdn_k_heads, cfg.gdn_v_heads, cfg.gdn_inner, cfg.gdn_conv_channels, x.shape[0]
        y = self.lin(x, L["qkv"])
        z, b, al = y[:, :DI], y[:, DI + C:DI + C + Hv], y[:, DI + C + Hv:DI + C + 2 * Hv]
        act, left = self.conv(L, y[:, DI:DI + C], self.m.conv_pool[li], DI)
        l2 = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q = (l2(act[:, :Hk * D].reshape(T, Hk, D)) / math.sqrt(D)).repeat_interleave(Hv // Hk, 1)
        k = l2(act[:, Hk * D:2 * Hk * D].reshape(T, Hk, D)).repeat_interleave(Hv // Hk, 1)
        v = act[:, 2 * Hk * D:].reshape(T, Hv, D)
        decay = torch.exp(L["a_neg"].double() * torch.nn.functional.softplus(al + L["dt_bias"].double()))
        beta = torch.sigmoid(b)
        # the pool as stored: [slot, head, value / 16, step, value % 16, half, 4] of S[value][key = 64 half + 4 step + e]
        pool = self.m.ssm_pool[li]
        S = pool.double().reshape(-1, Hv, 8, 16, 16, 2, 4).permute(0, 1, 2, 4, 5, 3, 6).reshape(-1, Hv, D, D).clone()
        o, start = torch.empty(T, Hv, D, dtype=torch.float64, device="cuda"), torch.tensor([sum(lens[:i]) for i in range(len(lens))], device="cuda")
        S[[i for i, c in enumerate(ctx) if not c]] = 0
        for t in range(max(lens)):                                       # all sequences that still have a token, together
            on = [i for i, n in enumerate(lens) if n > t]
            r = start[on] + t
            Z = S[on] * decay[r][:, :, None, None]
            kt = k[r][:, :, None]
            Z += ((v[r] - (Z * kt).sum(-1)) * beta[r][:, :, None])[..., None] * kt
            o[r] = (Z * q[r][:, :, None]).sum(-1)
            S[on] = Z
        o = self.norm(o, L["norm_w"]).reshape(T, DI)
        S = S.reshape(-1, Hv, 8, 16, 2, 16, 4).permute(0, 1, 2, 5, 3, 4, 6).reshape(pool.shape)
        return self.lin(o * z * torch.sigmoid(z), L["o"]), left, S

    def mamba(self, li, L, x):
        cfg, lens, ctx = self.cfg, self.s["lens"], self.s["ctx"]
        H, P, G, N, DI, C, T = cfg.ssm_heads, cfg.ssm_head_dim, cfg.ssm_groups, cfg.ssm_state, cfg.d_inner, cfg.conv_channels, x.shape[0]
        y = self.lin(x, L["qkv"])
        z, dt = y[:, :DI], torch.nn.functional.softplus(y[:, DI + C:DI + C + H] + L["dt_bias"].double())
        act, left = self.conv(L, y[:, DI:DI + C], self.m.conv_pool[li], DI)
        xs = act[:, :DI].reshape(T, H, P)
        Bm, Cm = (act[:, DI + i * G * N:DI + (i + 1) * G * N].reshape(T, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
        dA = torch.exp(dt * L["a_neg"].double())
        S, out, a = self.m.ssm_pool[li].double().clone(), torch.empty(T, H, P, dtype=torch.float64, device="cuda"), 0
        for i, n in enumerate(lens):
            Z = S[i] * (1.0 if ctx[i] else 0.0)
            for t in range(a, a + n):
                Z = Z * dA[t][:, None, None] + (xs[t] * dt[t][:, None])[:, :, None] * Bm[t][:, None]
                out[t] = (Z * Cm[t][:, None]).sum(-1) + L["d_skip"].double()[:, None] * xs[t]
            S[i] = Z
            a += n
        g = (out.reshape(T, DI) * z * torch.sigmoid(z)).reshape(T, G, DI // G)
        g = (g * torch.rsqrt(g.square().mean(-1, keepdim=True) + cfg.eps)).reshape(T, DI) * L["norm_w"].double()
        return self.lin(g, L["o"]), left, S

    def ffn(self, L, h):
        cfg = self.cfg
        x = self.norm(h, L["ffn_norm"])
        act = lambda y: torch.nn.functional.silu(y.chunk(2, -1)[0]) * y.chunk(2, -1)[1]  # noqa: E731
        if "router" not in L:
            return h + self.lin(act(self.lin(x, L["gate_up"])), L["down"])
        p = torch.softmax(x @ L["router"].double().T, -1)
        w, e = p.topk(cfg.top_k, -1)
        w = w / w.sum(-1, keepdim=True)
        out, gu, dn = h.clone(), L["gu"], L["down"]
        for i in range(cfg.n_experts):
            r, j = (e == i).nonzero(as_tuple=True)
            if len(r):
                y = self.linear(act(self.linear(x[r], gu.trellis[i], gu.suh[i], gu.svh[i])), dn.trellis[i], dn.suh[i], dn.svh[i])
                out.index_add_(0, r, w[r, j][:, None] * y)
        return out

    def run(self):
        s, m = self.s, self.m
        out = {"k": [], "v": [], "conv": [], "state": []}
        h = m.embed[s["rows"][0].long()].double()
        for li, L in enumerate(m.layers):
            x, kind = self.norm(h, L["attn_norm"]), L.get("kind", "A")
            y, a, b = (self.attention if kind == "A" else self.mamba if kind == "M" else self.delta)(li, L, x)
            for key, t in zip(("k", "v") if kind == "A" else ("conv", "state"), (a, b)):
                out[key].append(t.float())
            h = self.ffn(L, h + y)
        x = self.norm(h, m.final_norm)
        logits = self.lin(x if s["step"] else x[s["last"]], m.lm_head)
        out.update(logits=logits, values=logits.topk(16, -1).values)
        if any(c is not None and c.dtype == torch.uint8 for c in m.k_cache):
            out["k"], out["v"] = [None] * len(out["k"]), [None] * len(out["v"])      # bytes: compared as they are
        if not out["state"]:
            del out["conv"], out["state"]
        return out


@torch.no_grad()
def exact(case, seed):
    """The call of run() on the same weights, caches and tokens in 64 bits: rows are not rounded between the layers, the trellis is decoded by
    its definition, experts and sequences run one after the other.  (prepare() is used for what it draws, not for any arithmetic.)"""
    s = prepare(case, seed)
    s.pop("graph", None)
    return _Exact(s).run()
