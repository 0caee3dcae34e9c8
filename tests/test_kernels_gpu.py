"""Numerics of every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DT = [torch.float16, torch.bfloat16]


def _tol(dt):
    return (2e-2, 2e-2) if dt == torch.bfloat16 else (4e-3, 4e-3)


def _close(a, b, dt, scale=1.0):
    rtol, atol = _tol(dt)
    torch.testing.assert_close(a.float(), b.float(), rtol=rtol, atol=atol * scale)


@pytest.fixture(autouse=True)
def _seed():
    torch.manual_seed(0)


@pytest.fixture()
def status():
    s = torch.zeros(8, dtype=torch.int32, device="cuda")
    yield s
    torch.cuda.synchronize()
    assert s[0].item() == 0, f"kernel status {s.tolist()}"


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(1, 256, 512), (5, 384, 1024), (16, 4096, 4096), (64, 1000, 4304), (200, 640, 320),
                                   (128, 256, 64), (300, 512, 1024), (1024, 768, 2048), (257, 1152, 1152)])
def test_gemm_plain(dt, M, N, K, status):
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    y = K_.gemm(x, w, status=status)
    ref = x.float() @ w.float().t()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))


@pytest.mark.parametrize("swap", [0, 1])
@pytest.mark.parametrize("splits", [1, 3])
def test_gemm_epilogue_bias_residual_scale(swap, splits, status):
    from rhinoforge_b200.ops import kernels as K_
    dt = torch.float16
    M, N, K = 48, 640, 1536
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    b = torch.randn(N, device="cuda").to(dt)
    sc = (torch.rand(N, device="cuda") + 0.5).to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    rs = torch.rand(M, device="cuda") + 0.5
    y = K_.gemm(x, w, bias=b, scale=sc, residual=r, row_scale=rs, status=status, force_swap=swap,
                force_splits=splits)
    ref = (x.float() @ w.float().t()) * rs[:, None] * sc.float() + b.float() + r.float()
    _close(y, ref, dt, scale=4.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,swap,splits", [(3, 1, 1), (40, 1, 2), (40, 0, 1), (300, 0, 1)])
@pytest.mark.parametrize("act", ["silu_mul", "gelu_tanh_mul"])
def test_gemm_dual_glu(dt, M, swap, splits, act, status):
    from rhinoforge_b200.ops import kernels as K_
    N, K = 384, 1024
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(2 * N, K, device="cuda") * 0.05).to(dt)
    y = K_.gemm(x, w, act=act, dual=True, status=status, force_swap=swap, force_splits=splits)
    g = x.float() @ w[:N].float().t()
    u = x.float() @ w[N:].float().t()
    a = torch.nn.functional.silu(g) if act == "silu_mul" else torch.nn.functional.gelu(g, approximate="tanh")
    _close(y, a * u, dt, scale=2.0)


@pytest.mark.parametrize("act", ["gelu_tanh", "gelu_erf", "silu"])
def test_gemm_unary_act(act, status):
    from rhinoforge_b200.ops import kernels as K_
    dt = torch.float16
    x = (torch.randn(70, 512, device="cuda") * 0.5).to(dt)
    w = (torch.randn(256, 512, device="cuda") * 0.05).to(dt)
    y = K_.gemm(x, w, act=act, status=status)
    z = x.float() @ w.float().t()
    ref = {"gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh"),
           "gelu_erf": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[act](z)
    _close(y, ref, dt)


def test_gemm_is_deterministic(status):
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(32, 4096, device="cuda") * 0.5).half()
    w = (torch.randn(1024, 4096, device="cuda") * 0.05).half()
    a = K_.gemm(x, w, status=status, force_splits=4).clone()
    b = K_.gemm(x, w, status=status, force_splits=4)
    assert torch.equal(a, b)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M", [1, 2, 3, 8])
@pytest.mark.parametrize("int8", [False, True])
def test_gemv(dt, M, int8):
    from rhinoforge_b200.ops import kernels as K_
    N, K = 515, 1024
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    if int8:
        w = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8)
        sc = (torch.rand(N, device="cuda") * 0.01).to(dt)
        y = K_.gemm(x, w, scale=sc, residual=r, use_gemv=True)
        ref = (x.float() @ w.float().t()) * sc.float() + r.float()
    else:
        w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
        y = K_.gemm(x, w, residual=r, use_gemv=True)
        ref = x.float() @ w.float().t() + r.float()
    _close(y, ref, dt, scale=4.0)


def test_gemv_dual():
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(2, 512, device="cuda") * 0.5).half()
    w = (torch.randn(2 * 300, 512, device="cuda") * 0.05).half()
    y = K_.gemm(x, w, act="silu_mul", dual=True, use_gemv=True)
    g, u = x.float() @ w[:300].float().t(), x.float() @ w[300:].float().t()
    _close(y, torch.nn.functional.silu(g) * u, torch.float16)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("gemma", [False, True])
def test_rmsnorm(dt, gemma):
    from rhinoforge_b200.ops import kernels as K_
    x = torch.randn(37, 1024, device="cuda").to(dt)
    r = torch.randn(37, 1024, device="cuda").to(dt)
    w = (torch.randn(1024, device="cuda") * 0.1 + (0 if gemma else 1)).to(dt)
    ro = torch.empty_like(x)
    y = K_.rmsnorm(x, w, 1e-6, residual=r, residual_out=ro, gemma=gemma)
    h = (x.float() + r.float()).to(dt).float()
    n = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6)
    ref = n * (1 + w.float()) if gemma else w.float() * n.to(dt).float()
    _close(y, ref, dt)
    _close(ro, h, dt)


def test_rmsnorm_adarms_and_gated_residual():
    from rhinoforge_b200.ops import kernels as K_
    dt = torch.float16
    B, T, H = 3, 50, 1024
    x = torch.randn(B * T, H, device="cuda").to(dt)
    mod = (torch.randn(B, 3 * H, device="cuda") * 0.3).to(dt)
    y = K_.rmsnorm(x, None, 1e-6, mod=mod, rows_per_mod=T)
    n = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6)
    sc, sh, gt = mod.float().view(B, 1, 3 * H).chunk(3, -1)
    ref = (n.view(B, T, H) * (1 + sc) + sh).view(B * T, H)
    _close(y, ref, dt)
    x2 = x.clone()
    K_.gated_residual(x2, y, mod, T)
    _close(x2, (x.float().view(B, T, H) + gt * y.float().view(B, T, H)).view(B * T, H), dt)


@pytest.mark.parametrize("dt", DT)
def test_layernorm_l2norm(dt):
    from rhinoforge_b200.ops import kernels as K_
    x = torch.randn(33, 1152, device="cuda").to(dt)
    w, b = torch.randn(1152, device="cuda").to(dt), torch.randn(1152, device="cuda").to(dt)
    y = K_.layernorm(x, w, b, 1e-6)
    _close(y, torch.nn.functional.layer_norm(x.float(), (1152,), w.float(), b.float(), 1e-6), dt)
    z = K_.l2norm(x[:, :128].contiguous(), 1e-6)
    xf = x[:, :128].float()
    _close(z, xf * torch.rsqrt(xf.pow(2).sum(-1, keepdim=True) + 1e-6), dt)


def _rope_tables(max_pos, rot, theta, device):
    inv = 1.0 / (theta ** (torch.arange(0, rot, 2, device=device).float() / rot))
    ang = torch.arange(max_pos, device=device).float()[:, None] * inv[None]
    return ang.cos().contiguous(), ang.sin().contiguous()


def _rot_half(x):
    h = x.shape[-1] // 2
    return torch.cat([-x[..., h:], x[..., :h]], -1)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,rot", [(128, 128), (256, 64), (64, 64)])
def test_qk_norm_rope_kv_insert(dt, hd, rot):
    from rhinoforge_b200.ops import kernels as K_
    Hq, Hkv, T = 6, 2, 21
    seqs = 3
    qkv = torch.randn(T, (Hq + 2 * Hkv) * hd, device="cuda").to(dt)
    orig = qkv.clone()
    qw, kw = (torch.rand(hd, device="cuda") + 0.5).to(dt), (torch.rand(hd, device="cuda") + 0.5).to(dt)
    cos, sin = _rope_tables(512, rot, 1e6, "cuda")
    seq_of_tok = torch.arange(T, device="cuda", dtype=torch.int32) % seqs
    pos = (torch.arange(T, device="cuda", dtype=torch.int32) // seqs + 30).contiguous()
    pages = 16
    k_pool = torch.zeros(pages, Hkv, 16, hd, device="cuda", dtype=dt)
    v_pool = torch.zeros_like(k_pool)
    page_table = torch.arange(seqs * 4, device="cuda", dtype=torch.int32).view(seqs, 4).contiguous()
    K_.qk_norm_rope_kv(qkv, Hq, Hkv, hd, pos=pos, cos=cos, sin=sin, rot_dim=rot, q_norm_w=qw, k_norm_w=kw,
                       k_pool=k_pool, v_pool=v_pool, page_table=page_table, seq_of_tok=seq_of_tok)
    o = orig.float().view(T, Hq + 2 * Hkv, hd)

    def ref(x, w):
        n = (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6)).to(dt).float() * w.float()
        n = n.to(dt).float()
        c = cos[pos.long()][:, None, :].repeat(1, 1, 2)
        s = sin[pos.long()][:, None, :].repeat(1, 1, 2)
        r = n[..., :rot] * c + _rot_half(n[..., :rot]) * s
        return torch.cat([r, n[..., rot:]], -1)

    q_ref, k_ref, v_ref = ref(o[:, :Hq], qw), ref(o[:, Hq:Hq + Hkv], kw), o[:, Hq + Hkv:]
    _close(qkv.view(T, -1, hd)[:, :Hq], q_ref, dt)
    for t in range(T):
        s, p = int(seq_of_tok[t]), int(pos[t])
        page = int(page_table[s, p // 16])
        _close(k_pool[page, :, p % 16], k_ref[t], dt)
        _close(v_pool[page, :, p % 16], v_ref[t], dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,rot,Hq,Hkv", [(64, 64, 6, 6), (128, 128, 5, 2), (256, 64, 3, 1), (128, 64, 4, 4)])
@pytest.mark.parametrize("variant", ["plain", "norm", "gemma_rope_first", "mrope_vnorm", "pool"])
def test_qk_norm_rope_kv_prefill_sized(dt, hd, rot, Hq, Hkv, variant):
    """Launches of 512 tokens or more take the 16-byte kernel: the same rows through one 640-token launch and through
    two launches of 320 (below the switch, the scalar kernel) must agree to one rounding step, in every mode."""
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(3)
    T, half = 640, rot // 2
    W = (Hq + 2 * Hkv) * hd
    qkv = (torch.randn(T, W, device="cuda") * 0.7).to(dt)
    axes = 3 if variant == "mrope_vnorm" else 1
    pos = torch.randint(0, 900, (T, axes), device="cuda", dtype=torch.int32)
    ang = torch.arange(1024, device="cuda", dtype=torch.float32)[:, None] * (1.0 / 10000 ** (torch.arange(half, device="cuda") / half))[None]
    kw = dict(pos=pos, cos=ang.cos().contiguous(), sin=ang.sin().contiguous(), rot_dim=rot)
    if variant in ("norm", "gemma_rope_first", "mrope_vnorm", "pool"):
        kw.update(q_norm_w=(1 + 0.1 * torch.randn(hd, device="cuda")).to(dt), k_norm_w=(1 + 0.1 * torch.randn(hd, device="cuda")).to(dt))
    if variant == "gemma_rope_first":
        kw.update(gemma=True, rope_before_norm=True)
    if variant == "mrope_vnorm":
        kw.update(axis_of_freq=torch.randint(0, 3, (half,), device="cuda", dtype=torch.int8), v_norm=True)
    outs = []
    pt = torch.randperm(T // 16 + 2, device="cuda").to(torch.int32)[None].contiguous()     # one shuffled page table for both runs
    for chunks in (1, 2):
        buf = qkv.clone()
        q_out = torch.zeros(T, Hq * hd, device="cuda", dtype=dt) if variant == "pool" else None
        pools = None
        if variant == "pool":
            pages = T // 16 + 2
            pools = (torch.zeros(pages, Hkv, 16, hd, device="cuda", dtype=dt), torch.zeros(pages, Hkv, 16, hd, device="cuda", dtype=dt))
        n = T // chunks
        for c in range(chunks):
            sl = slice(c * n, (c + 1) * n)
            extra = {}
            if variant == "pool":
                extra = dict(k_pool=pools[0], v_pool=pools[1], page_table=pt, seq_of_tok=torch.zeros(n, device="cuda", dtype=torch.int32),
                             cache_pos=torch.arange(c * n, (c + 1) * n, device="cuda", dtype=torch.int32), q_out=q_out[sl])
            K_.qk_norm_rope_kv(buf[sl], Hq, Hkv, hd, **{**kw, "pos": pos[sl].contiguous()}, **extra)
        torch.cuda.synchronize()
        outs.append((buf, q_out, pools))
    (b1, q1, p1), (b2, q2, p2) = outs

    def same(x, y):            # one rounding step of the 16-bit type at most (the two kernels may contract their FMAs differently)
        tol = (2.0 ** -10 if dt == torch.float16 else 2.0 ** -7) * max(1.0, float(y.float().abs().max()))
        return float((x.float() - y.float()).abs().max()) <= tol
    assert same(b1, b2)
    if variant == "pool":
        assert same(q1, q2) and same(p1[0], p2[0]) and same(p1[1], p2[1])
        assert float(p1[0].abs().max()) > 0 and float(q1.abs().max()) > 0
    else:
        assert not torch.equal(b1, qkv)


def test_mrope_axis_select():
    from rhinoforge_b200.ops import kernels as K_
    dt, hd, T = torch.float16, 128, 9
    qkv = torch.randn(T, 3 * hd, device="cuda").to(dt)
    orig = qkv.clone()
    cos, sin = _rope_tables(256, hd, 1e6, "cuda")
    pos = torch.randint(0, 200, (T, 3), device="cuda", dtype=torch.int32)
    sec = [24, 20, 20]
    axis = torch.zeros(hd // 2, dtype=torch.int8)
    for dim, off in ((1, 1), (2, 2)):
        axis[off:sec[dim] * 3:3] = dim
    K_.qk_norm_rope_kv(qkv, 1, 1, hd, pos=pos, cos=cos, sin=sin, axis_of_freq=axis.cuda(), write_k_inplace=True)
    idx = pos.long()[:, axis.long().cuda()]  # [T, hd/2]
    f = torch.arange(hd // 2, device="cuda")
    c = cos[idx, f].repeat(1, 2)
    s = sin[idx, f].repeat(1, 2)
    for h in range(2):
        x = orig.float().view(T, 3, hd)[:, h]
        _close(qkv.view(T, 3, hd)[:, h], x * c + _rot_half(x) * s, dt)


def _sdpa_ref(q, k, v, mask):
    # q [Hq, Lq, hd], k/v [Hkv, Lk, hd], mask [Lq, Lk] bool
    G = q.shape[0] // k.shape[0]
    k = k.repeat_interleave(G, 0)
    v = v.repeat_interleave(G, 0)
    s = (q.float() @ k.float().transpose(1, 2)) / math.sqrt(q.shape[-1])
    s = s.masked_fill(~mask[None], float("-inf"))
    p = torch.softmax(s, -1)
    p = torch.nan_to_num(p)
    return p @ v.float()


def _paged(Hkv, hd, kv_lens, dt, extra_pages=3):
    seqs = len(kv_lens)
    maxp = max((l + 15) // 16 for l in kv_lens) + 1
    total = seqs * maxp + extra_pages
    perm = torch.randperm(total)[: seqs * maxp].to(torch.int32).view(seqs, maxp)
    k_pool = torch.zeros(total, Hkv, 16, hd, device="cuda", dtype=dt)
    v_pool = torch.zeros_like(k_pool)
    ks, vs = [], []
    for s, L in enumerate(kv_lens):
        k = torch.randn(Hkv, L, hd, device="cuda").to(dt)
        v = torch.randn(Hkv, L, hd, device="cuda").to(dt)
        for t in range(L):
            pg = int(perm[s, t // 16])
            k_pool[pg, :, t % 16] = k[:, t]
            v_pool[pg, :, t % 16] = v[:, t]
        ks.append(k)
        vs.append(v)
    return k_pool, v_pool, perm.cuda().contiguous(), ks, vs


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(128, 8, 2), (64, 4, 4), (256, 8, 1)])
def test_attn_prefill_paged_causal(dt, hd, Hq, Hkv, status):
    from rhinoforge_b200.ops import kernels as K_
    q_lens, kv_lens = [70, 33, 128], [70, 97, 128]
    k_pool, v_pool, pt, ks, vs = _paged(Hkv, hd, kv_lens, dt)
    q_start = [0, 70, 103]
    Tq = sum(q_lens)
    q = torch.randn(Tq, Hq * hd, device="cuda").to(dt)
    out = torch.zeros_like(q)
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    K_.attention_prefill(q, out, Hq=Hq, Hkv=Hkv, hd=hd, q_start=i32(q_start), q_len=i32(q_lens), kv_len=i32(kv_lens),
                         max_q_len=max(q_lens), k_pool=k_pool, v_pool=v_pool, page_table=pt, causal=True,
                         status=status)
    for s in range(3):
        Lq, Lk = q_lens[s], kv_lens[s]
        qs = q[q_start[s]:q_start[s] + Lq].view(Lq, Hq, hd).transpose(0, 1)
        qi = torch.arange(Lq, device="cuda")[:, None] + (Lk - Lq)
        mask = torch.arange(Lk, device="cuda")[None] <= qi
        ref = _sdpa_ref(qs, ks[s], vs[s], mask).transpose(0, 1).reshape(Lq, Hq * hd)
        _close(out[q_start[s]:q_start[s] + Lq], ref, dt)


@pytest.mark.parametrize("mode", ["bidir", "mask", "segments", "window"])
def test_attn_prefill_contiguous_masks(mode, status):
    from rhinoforge_b200.ops import kernels as K_
    dt, hd, H = torch.float16, 64, 4
    L = 201
    qkv = torch.randn(L, 3 * H * hd, device="cuda").to(dt)
    q, k, v = qkv[:, :H * hd], qkv[:, H * hd:2 * H * hd], qkv[:, 2 * H * hd:]
    out = torch.zeros(L, H * hd, device="cuda", dtype=dt)
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    kw = dict(Hq=H, Hkv=H, hd=hd, q_start=i32([0]), q_len=i32([L]), kv_len=i32([L]), max_q_len=L, k=k, v=v,
              kv_start=i32([0]), causal=False, status=status)
    full = torch.ones(L, L, dtype=torch.bool, device="cuda")
    if mode == "bidir":
        mask = full
    elif mode == "mask":
        mask = torch.rand(L, L, device="cuda") > 0.3
        mask[:, 0] = True
        kw["mask"] = mask.contiguous()
    elif mode == "segments":
        seg = (torch.arange(L, device="cuda") // 37).to(torch.int32)
        mask = seg[:, None] == seg[None]
        kw["seg_q"], kw["seg_k"] = seg, seg
    else:
        kw["causal"], kw["window"] = True, 48
        i = torch.arange(L, device="cuda")
        mask = (i[None] <= i[:, None]) & (i[None] > i[:, None] - 48)
    K_.attention_prefill(q, out, **kw)
    tr = lambda t: t.reshape(L, H, hd).transpose(0, 1)
    ref = _sdpa_ref(tr(q), tr(k), tr(v), mask).transpose(0, 1).reshape(L, H * hd)
    _close(out, ref, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(128, 32, 8), (128, 8, 1), (64, 4, 2), (256, 8, 1)])
@pytest.mark.parametrize("split", [False, True])
def test_attn_decode_paged(dt, hd, Hq, Hkv, split, status):
    from rhinoforge_b200.ops import kernels as K_
    kv_lens = [1, 17, 300, 1025, 64]
    k_pool, v_pool, pt, ks, vs = _paged(Hkv, hd, kv_lens, dt)
    B = len(kv_lens)
    q = torch.randn(B, Hq * hd, device="cuda").to(dt)
    out = torch.zeros_like(q)
    ws = K_.attn_decode_scratch(B, Hq, hd, "cuda") if split else None
    K_.attention_decode(q, out, Hq=Hq, Hkv=Hkv, hd=hd, kv_len=torch.tensor(kv_lens, dtype=torch.int32, device="cuda"),
                        max_kv_len=max(kv_lens), k_pool=k_pool, v_pool=v_pool, page_table=pt, ws=ws, status=status)
    for s in range(B):
        L = kv_lens[s]
        ref = _sdpa_ref(q[s].view(Hq, 1, hd), ks[s], vs[s], torch.ones(1, L, dtype=torch.bool, device="cuda"))
        _close(out[s], ref.reshape(Hq * hd), dt)


def test_embedding_scatter_eltwise_cast_argmax():
    from rhinoforge_b200.ops import kernels as K_
    dt = torch.float16
    table = torch.randn(1000, 256, device="cuda").to(dt)
    ids = torch.tensor([3, 999, -1, 0, 17], dtype=torch.int32, device="cuda")
    e = K_.embedding(table, ids, scale=2.0)
    ref = table[ids.clamp(min=0).long()].float() * 2.0
    ref[2] = 0
    _close(e, ref, dt)
    dst = torch.zeros(10, 256, device="cuda", dtype=dt)
    K_.scatter_rows(dst, e, torch.tensor([9, 1, -1, 4, 0], dtype=torch.int32, device="cuda"))
    assert torch.equal(dst[9], e[0]) and torch.equal(dst[0], e[4]) and dst[2].abs().sum() == 0
    a, b = torch.randn(77, 256, device="cuda").to(dt), torch.randn(77, 256, device="cuda").to(dt)
    _close(K_.eltwise("silu_mul", a, b), torch.nn.functional.silu(a.float()) * b.float(), dt)
    _close(K_.eltwise("axpy", a, b, alpha=-0.1), a.float() - 0.1 * b.float(), dt)
    _close(K_.eltwise("mul_row", a, b[0].contiguous()), a.float() * b[0].float(), dt)
    u8 = torch.randint(0, 256, (3, 64), dtype=torch.uint8, device="cuda")
    _close(K_.cast_u8(u8, dt, 1 / 127.5, -1.0), u8.float() / 127.5 - 1.0, dt)
    logits = torch.randn(5, 151936, device="cuda").to(dt)
    logits[2, 77] = 100.0
    logits[3, 151935] = 100.0
    ids2, vals = K_.argmax(logits, offset=10, return_vals=True)
    assert torch.equal(ids2.long() - 10, logits.float().argmax(-1))
    _close(vals, logits.float().max(-1).values, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,swap,splits", [(16, 384, 1024, -1, 0), (64, 1000, 2048, 1, 4), (9, 256, 512, 1, 1),
                                               (300, 640, 1024, 0, 1), (1024, 512, 2048, 0, 1), (130, 256, 4096, 1, 2)])
def test_gemm_w8a16_tensor_core(dt, M, N, K, swap, splits, status):
    """int8 weights widened in the mainloop, (X . Q^T) * scale in the epilogue."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    q = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8)
    sc = (torch.rand(N, device="cuda") * 0.004 + 0.001).to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    y = K_.gemm(x, q, scale=sc, residual=r, status=status, force_swap=swap, force_splits=splits)
    ref = (x.float() @ q.float().t()) * sc.float() + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()) * (4 if dt == torch.bfloat16 else 1))


@pytest.mark.parametrize("M,swap", [(24, 1), (300, 0)])
def test_gemm_w8a16_dual_glu(M, swap, status):
    from rhinoforge_b200.ops import kernels as K_
    dt, N, K = torch.float16, 384, 1024
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    q = torch.randint(-127, 128, (2 * N, K), device="cuda", dtype=torch.int8)
    sc = (torch.rand(2 * N, device="cuda") * 0.002 + 0.0005).to(dt)
    y = K_.gemm(x, q, scale=sc, act="silu_mul", dual=True, status=status, force_swap=swap)
    z = (x.float() @ q.float().t()) * sc.float()
    _close(y, torch.nn.functional.silu(z[:, :N]) * z[:, N:], dt, scale=2.0)


def test_engine_w8a16_matches_dequantised_oracle():
    """Whole decoder with int8 weights: greedy tokens follow the oracle run on the dequantised weights."""
    from rhinoforge_b200.models.decoder import TorchDecoder, random_state_dict, tiny_config
    from rhinoforge_b200.quant._common import dequantize_linear_per_channel, quantize_linear_per_channel
    from rhinoforge_b200.runtime.engine import DecoderEngine
    cfg = tiny_config(num_layers=2)
    sd = random_state_dict(cfg, seed=0, dtype=torch.float16, norm_jitter=0.05)
    deq = {}
    for k, v in sd.items():
        if v.dim() == 2 and "embed" not in k:
            qq, s = quantize_linear_per_channel(v)
            deq[k] = dequantize_linear_per_channel(qq, s)
        else:
            deq[k] = v
    if "lm_head.weight" not in sd:            # tied embeddings: the head is the quantised embedding matrix
        deq["lm_head.weight"] = dequantize_linear_per_channel(*quantize_linear_per_channel(sd["model.embed_tokens.weight"]))
    oracle = TorchDecoder(cfg, deq, dtype=torch.float32, device="cuda")
    eng = DecoderEngine(cfg, lambda n: sd[n] if n in sd else sd["model.embed_tokens.weight"], dtype=torch.float16,
                        max_batch=2, max_seq_len=96, quant="w8a16")
    g = torch.Generator().manual_seed(7)
    prompts = [torch.randint(0, cfg.vocab_size, (L,), generator=g) for L in (19, 40)]
    _, logits = eng.prefill(prompts, return_logits=True)
    for b, p in enumerate(prompts):
        oracle.reset()
        ref = oracle.forward(p[None].cuda())[0, -1]
        torch.testing.assert_close(logits[b].float(), ref.float(), rtol=1e-2, atol=1e-2)
    toks = eng.generate(prompts, 6)
    assert toks.shape == (2, 6)
    eng.check_status()
    eng.close()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,swap,splits", [(16, 384, 1024, -1, 0), (64, 1000, 2048, 1, 4), (9, 200, 520, 1, 1),
                                               (300, 640, 1024, 0, 1), (1024, 512, 2048, 0, 1), (700, 130, 264, 0, 1)])
def test_gemm_packed_weights(dt, M, N, K, swap, splits, status):
    """Tile-major (bulk-copy) weight layout gives the same result as row-major weights."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    b = torch.randn(N, device="cuda").to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    wp = K_.pack_weight(w)
    y = K_.gemm(x, wp, packed_shape=(N, K), bias=b, residual=r, status=status, force_swap=swap, force_splits=splits)
    ref = x.float() @ w.float().t() + b.float() + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))


@pytest.mark.parametrize("M,swap", [(24, 1), (300, 0)])
def test_gemm_packed_dual_and_int8(M, swap, status):
    from rhinoforge_b200.ops import kernels as K_
    dt, N, K = torch.float16, 200, 1024                    # N not a multiple of 128: sections are padded separately
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(2 * N, K, device="cuda") * 0.05).to(dt)
    y = K_.gemm(x, K_.pack_weight(w, 2), packed_shape=(2 * N, K), act="silu_mul", dual=True, status=status, force_swap=swap)
    z = x.float() @ w.float().t()
    _close(y, torch.nn.functional.silu(z[:, :N]) * z[:, N:], dt, scale=2.0)
    q = torch.randint(-127, 128, (2 * N, K), device="cuda", dtype=torch.int8)
    sc = (torch.rand(2 * N, device="cuda") * 0.002 + 0.0005).to(dt)
    y = K_.gemm(x, K_.pack_weight(q, 2), packed_shape=(2 * N, K), scale=sc, act="silu_mul", dual=True, status=status,
                force_swap=swap)
    z = (x.float() @ q.float().t()) * sc.float()
    _close(y, torch.nn.functional.silu(z[:, :N]) * z[:, N:], dt, scale=2.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,dual", [(2500, 2048, 520, False), (4100, 1280, 1024, False), (2304, 2560, 512, True),
                                        (20000, 256, 128, False), (1152, 2560, 512, True), (5000, 2048, 520, False),
                                        (4900, 1152, 256, False), (4900, 2048, 4096, False)])
def test_gemm_persistent_kernel(dt, M, N, K, dual, status):
    """Large token counts take the persistent kernel (one CTA per SM walking tiles): 128-row tiles with two
    accumulator buffers (the first, second, fourth and fifth shapes) and 256-row tiles (the others); ragged M
    (a last half-tile partly or wholly past the end), N not a multiple of the tile, several tiles per CTA,
    a ring shorter and longer than K, bias + residual, GLU epilogue."""
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(M)
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    rows = 2 * N if dual else N
    w = (torch.randn(rows, K, device="cuda") * 0.05).to(dt)
    wp = K_.pack_weight(w, 2 if dual else 1)
    if dual:
        y = K_.gemm(x, wp, packed_shape=(rows, K), act="silu_mul", dual=True, status=status)
        z = x.float() @ w.float().t()
        ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    else:
        b = torch.randn(N, device="cuda").to(dt)
        r = torch.randn(M, N, device="cuda").to(dt)
        y = K_.gemm(x, wp, packed_shape=(rows, K), bias=b, residual=r, status=status)
        ref = x.float() @ w.float().t() + b.float() + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))
    y2 = K_.gemm(x, wp, packed_shape=(rows, K), act="silu_mul", dual=True, status=status) if dual else \
        K_.gemm(x, wp, packed_shape=(rows, K), bias=b, residual=r, status=status)
    assert torch.equal(y, y2), "two launches of the same GEMM must agree bit for bit"
    if not dual:
        # without a residual the results leave through staging tiles and tiled bulk stores
        y3 = K_.gemm(x, wp, packed_shape=(rows, K), bias=b, status=status)
        _close(y3, x.float() @ w.float().t() + b.float(), dt, scale=max(1.0, ref.abs().max().item()))
        view = torch.zeros(M, N + 8, device="cuda", dtype=dt)           # strided output rows
        K_.gemm(x, wp, packed_shape=(rows, K), out=view[:, :N], status=status)
        _close(view[:, :N], x.float() @ w.float().t(), dt, scale=max(1.0, ref.abs().max().item()))
        assert float(view[:, N:].abs().max()) == 0.0, "columns past N must stay untouched"
        # residual already in the output buffer (out == residual): the add happens in the bulk reduce
        acc = r.clone()
        K_.gemm(x, wp, packed_shape=(rows, K), residual=acc, out=acc, status=status)
        _close(acc, x.float() @ w.float().t() + r.float(), dt, scale=max(1.0, ref.abs().max().item()))


def test_manual_graph_capture_replays_with_refilled_inputs(status):
    """``graph.capture``: one recording run, then replays that refill the static input buffers; a changed shape is refused."""
    from rhinoforge_b200.graph import capture
    from rhinoforge_b200.ops import kernels as K_
    w = (1.0 + 0.1 * torch.randn(256, device="cuda")).half()
    x = torch.randn(40, 256, device="cuda").half()
    out = torch.empty_like(x)

    def fn(inp):
        K_.rmsnorm(inp, w, 1e-6, out=out)
        return out

    g = capture(fn, x)
    assert g.replayable, g.non_replayable_reason
    ref = lambda t: (w.float() * (t.float() * torch.rsqrt(t.float().pow(2).mean(-1, keepdim=True) + 1e-6)))
    torch.cuda.synchronize()
    _close(g.cached_output, ref(x), torch.float16)
    x2 = torch.randn(40, 256, device="cuda").half()
    y = g.replay(x2)
    torch.cuda.synchronize()
    _close(y, ref(x2), torch.float16)
    st = g.stats()
    assert st["replays"] == 1 and st["build_count"] == 1 and st["node_count"] >= 1
    with pytest.raises(RuntimeError, match="shape_bucket"):
        g.replay(torch.randn(41, 256, device="cuda").half())
    g.invalidate()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_w8a16_large_m_widens_once_and_matches(dt, dual, status):
    """W8A16 with a prefill-sized token count and caller scratch: the int8 image is widened once and the 16-bit
    (persistent) kernel runs; the result equals ``(x . q^T) * scale`` like the in-loop path without scratch."""
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(3)
    M, N, K = 2304, 2560, 512
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    rows = 2 * N if dual else N
    q = torch.randint(-127, 128, (rows, K), device="cuda", dtype=torch.int8)
    sc = (torch.rand(rows, device="cuda") * 0.002 + 0.0005).to(dt)
    qp = K_.pack_weight(q, 2 if dual else 1)
    scratch = torch.empty(2 * qp.numel(), dtype=torch.uint8, device="cuda")
    kw = dict(packed_shape=(rows, K), scale=sc, status=status)
    if dual:
        kw.update(act="silu_mul", dual=True)
    y = K_.gemm(x, qp, w_scratch=scratch, **kw)
    y0 = K_.gemm(x, qp, **kw)
    z = (x.float() @ q.float().t()) * sc.float()
    ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))
    _close(y0, ref, dt, scale=max(1.0, ref.abs().max().item()))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(64, 4096, 512), (64, 4096, 1024), (50, 1024, 192), (8, 2048, 64)])
def test_gemm_short_k_splits_down_to_one_block_per_cta(dt, M, N, K, status):
    """Short-K weight-streaming shapes (tensor-parallel out-projections): the planner may give every CTA of the
    cluster a single k block (or fewer splits than blocks when K is tiny); bias, residual and the rotated K start are
    all in play."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    b = torch.randn(N, device="cuda").to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    ref = x.float() @ w.float().t() + b.float() + r.float()
    y = K_.gemm(x, K_.pack_weight(w), packed_shape=(N, K), bias=b, residual=r, status=status)
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))
    y2 = K_.gemm(x, w, bias=b, residual=r, status=status)                  # row-major weights, same planner
    _close(y2, ref, dt, scale=max(1.0, ref.abs().max().item()))
    for s in (1, 8):
        if s * 64 <= max(K, 64) or s == 1:
            y3 = K_.gemm(x, K_.pack_weight(w), packed_shape=(N, K), bias=b, residual=r, status=status, force_splits=s)
            _close(y3, ref, dt, scale=max(1.0, ref.abs().max().item()))


def _close_elementwise(y, ref, dt):
    """Every element within fp16 / bf16 rounding of ITS OWN reference value (plus a small absolute floor), so a
    wrong low-magnitude column cannot hide behind the largest entry of the matrix."""
    rel = 2.0 ** -7 if dt == torch.bfloat16 else 2.0 ** -10
    err = (y.float() - ref.float()).abs()
    bound = rel * ref.float().abs() * 2.0 + (6e-2 if dt == torch.bfloat16 else 6e-3)
    bad = (err > bound).nonzero()
    assert bad.numel() == 0, f"{bad.shape[0]} elements off; first {bad[0].tolist()}: {y[tuple(bad[0])].item()} vs {ref[tuple(bad[0])].item()}"


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,dual", [(1, 4096, 4096, False), (7, 384, 2048, False), (16, 1000, 1024, False),
                                        (64, 2048, 4096, True), (64, 4096, 12288, False), (33, 1280, 512, True),
                                        (200, 640, 2560, False), (256, 1152, 1024, False), (96, 8192, 1024, True),
                                        (64, 151936, 1024, False)])
def test_gemm_stream_k(dt, M, N, K, dual, status):
    """The persistent stream-K kernel (tile-major weights, at most 256 tokens): shares that start and end inside a
    tile (partials parked in scratch and added by the tile's finisher), several tiles per CTA, ragged N, one token,
    a full 256-token tile, GLU pairs, a vocabulary-sized N; bias, per-channel scale, per-row scale and residual;
    two launches agree bit for bit."""
    from rhinoforge_b200 import _native as N_
    from rhinoforge_b200.ops import kernels as K_
    old_mode = N_.lib().rf_gemm_streamk_mode(2)          # every shape that fits, not only the large-N ones
    try:
        _stream_k_case(dt, M, N, K, dual, status)
    finally:
        N_.lib().rf_gemm_streamk_mode(old_mode)


def _stream_k_case(dt, M, N, K, dual, status):
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(M * 7 + N)
    rows = 2 * N if dual else N
    plan = K_.gemm_plan(M, N, K, dtype=dt, dual=dual, packed=True)
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(rows, K, device="cuda") * (1.0 / math.sqrt(K))).to(dt)
    wp = K_.pack_weight(w, 2 if dual else 1)
    z = x.float() @ w.float().t()
    if dual:
        y = K_.gemm(x, wp, packed_shape=(rows, K), act="silu_mul", dual=True, status=status)
        ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
        y2 = K_.gemm(x, wp, packed_shape=(rows, K), act="silu_mul", dual=True, status=status)
    else:
        b = torch.randn(N, device="cuda").to(dt)
        sc = (torch.rand(N, device="cuda") + 0.5).to(dt)
        rs = torch.rand(M, device="cuda") + 0.5
        r = torch.randn(M, N, device="cuda").to(dt)
        y = K_.gemm(x, wp, packed_shape=(rows, K), bias=b, scale=sc, row_scale=rs, residual=r, status=status)
        ref = z * rs[:, None] * sc.float() + b.float() + r.float()
        y2 = K_.gemm(x, wp, packed_shape=(rows, K), bias=b, scale=sc, row_scale=rs, residual=r, status=status)
        # in place: the residual already sits in the output buffer
        acc = r.clone()
        K_.gemm(x, wp, packed_shape=(rows, K), residual=acc, out=acc, status=status)
        _close_elementwise(acc, z + r.float(), dt)
    _close_elementwise(y, ref, dt)
    assert torch.equal(y, y2), "two launches of the same GEMM must agree bit for bit"
    assert plan is None or plan["persistent"] in (0, 2)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,group,dual", [(1, 1024, 4096, 64, False), (16, 1000, 1024, 32, False), (64, 384, 2048, 128, False),
                                              (64, 2048, 1024, 0, False), (33, 1280, 512, 64, True), (200, 640, 2560, 32, False),
                                              (300, 512, 1024, 64, False), (300, 768, 512, 128, True), (8, 256, 192, 64, False)])
def test_gemm_w4a16(dt, M, N, K, group, dual, status):
    """int4 weights in the tile-major image: nibbles widened and group scales applied by the converter warps of the
    main loop (per-channel scales in the epilogue when group = 0); reference = x @ dequantised weights in fp32."""
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(N + K + group)
    rows = 2 * N if dual else N
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    q = torch.randint(-8, 8, (rows, K), device="cuda", dtype=torch.int8)
    r = torch.randn(M, N, device="cuda").to(dt)
    kw = dict(packed_shape=(rows, K), w_bits=4, w_group=group, status=status)
    if group:
        sc = (torch.rand(rows, K // group, device="cuda") * 0.03 + 0.005).to(dt)
        img = K_.pack_weight_int4(q, sc, group, sections=2 if dual else 1, dtype=dt)
        wd = q.float().view(rows, K // group, group) * sc.float()[..., None]
        wd = wd.view(rows, K)
    else:
        sc = (torch.rand(rows, device="cuda") * 0.03 + 0.005).to(dt)
        img = K_.pack_weight_int4(q, sections=2 if dual else 1)
        kw["scale"] = sc
        wd = q.float() * sc.float()[:, None]
    assert img.numel() == K_.N.lib().rf_pack_w4_bytes(rows, K, 2 if dual else 1, group)
    z = x.float() @ wd.t()
    if dual:
        y = K_.gemm(x, img, act="silu_mul", dual=True, **kw)
        ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    else:
        y = K_.gemm(x, img, residual=r, **kw)
        ref = z + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()) * (4 if dt == torch.bfloat16 else 1))


@pytest.mark.parametrize("group,from_packed", [(64, False), (32, True), (0, False)])
def test_engine_w4a16_matches_dequantised_oracle(group, from_packed):
    """Whole decoder with int4 projections (lm_head 16-bit): prefill logits follow the oracle run on the dequantised
    weights, whether the engine quantises 16-bit weights itself or reads a packed 4-bit checkpoint."""
    from rhinoforge_b200.models.decoder import TorchDecoder, random_state_dict, tiny_config
    from rhinoforge_b200.quant.int4_pack import pack_int4
    from rhinoforge_b200.runtime.engine import DecoderEngine
    cfg = tiny_config(num_layers=2)
    sd = random_state_dict(cfg, seed=0, dtype=torch.float16, norm_jitter=0.05)

    def quant(w):
        wf = w.float()
        grp = wf.view(wf.shape[0], -1, group) if group else wf.view(wf.shape[0], 1, -1)
        sc = (grp.abs().amax(-1) / 7.0).clamp_min(1e-8)
        q = torch.round(grp / sc[..., None]).clamp_(-8, 7)
        return q.to(torch.int8).view_as(wf), sc, (q * sc[..., None].half().float()).view_as(wf)

    deq, packed, scales = {}, {}, {}
    for k, v in sd.items():
        if v.dim() == 2 and "embed" not in k and "lm_head" not in k:
            q, sc, d = quant(v)
            deq[k], packed[k], scales[k] = d, pack_int4(q), sc.half()
        else:
            deq[k] = v
    oracle = TorchDecoder(cfg, deq, dtype=torch.float32, device="cuda")

    def get(n):
        if n not in sd:
            return sd["model.embed_tokens.weight"]
        return packed[n] if (from_packed and n in packed) else sd[n]
    get.scale = lambda n: scales.get(n)
    eng = DecoderEngine(cfg, get, dtype=torch.float16, max_batch=2, max_seq_len=96, quant="w4a16", w4_group=group)
    g = torch.Generator().manual_seed(7)
    prompts = [torch.randint(0, cfg.vocab_size, (L,), generator=g) for L in (19, 40)]
    _, logits = eng.prefill(prompts, return_logits=True)
    for b, p in enumerate(prompts):
        oracle.reset()
        ref = oracle.forward(p[None].cuda())[0, -1]
        torch.testing.assert_close(logits[b].float(), ref.float(), rtol=2e-2, atol=2e-2)
    toks = eng.generate(prompts, 6)
    assert toks.shape == (2, 6)
    eng.check_status()
    eng.close()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,dual", [(1, 1024, 2048, False), (48, 520, 1024, False), (64, 768, 512, True), (300, 512, 1024, False)])
def test_gemm_nvfp4(dt, M, N, K, dual, status):
    """NVFP4 weights (e2m1 codes, e4m3 block scale per 16 columns, fp32 tensor scale) through the 4-bit main loop;
    reference = x @ the exact fp32 weight the codes stand for."""
    from rhinoforge_b200.ops import kernels as K_
    from rhinoforge_b200.quant.nvfp4_pack import dequantize_nvfp4, quantize_nvfp4
    torch.manual_seed(N + K)
    rows = 2 * N if dual else N
    w = torch.randn(rows, K, device="cuda") * 0.05
    codes, sc, ts = quantize_nvfp4(w)
    wd = dequantize_nvfp4(codes, sc, ts)
    img = K_.pack_weight_nvfp4(codes, sc, ts, sections=2 if dual else 1, dtype=dt)
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    kw = dict(packed_shape=(rows, K), w_bits=4, w_group=16, w_fp4=True, status=status)
    z = x.float() @ wd.t()
    if dual:
        y = K_.gemm(x, img, act="silu_mul", dual=True, **kw)
        ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:]
    else:
        y = K_.gemm(x, img, **kw)
        ref = z
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()) * (4 if dt == torch.bfloat16 else 1))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,H,I,splits", [(1, 1024, 2048, 0), (64, 1024, 3072, 0), (16, 512, 1024, 1), (200, 768, 1536, 0),
                                           (33, 1280, 512, 4)])
def test_gemm_folded_rmsnorm(dt, M, H, I, splits, status):
    """RMSNorm without a kernel of its own: the residual GEMM writes per-tile sums of squares of its finished rows, the
    next projection (norm weights multiplied into its columns) scales its rows by their reciprocal RMS.  Reference:
    rmsnorm(hidden) * w @ W2^T on the rows the first GEMM stored."""
    from rhinoforge_b200.ops import kernels as K_
    torch.manual_seed(M + H)
    x = (torch.randn(M, I, device="cuda") * 0.5).to(dt)
    w1 = (torch.randn(H, I, device="cuda") * 0.05).to(dt)
    resid = torch.randn(M, H, device="cuda").to(dt)
    nw = (1.0 + 0.2 * torch.randn(H, device="cuda")).to(dt)
    w2 = (torch.randn(2 * I, H, device="cuda") * 0.05).to(dt)
    bias = (torch.randn(2 * I, device="cuda") * 0.1).to(dt)
    tiles = (H + 127) // 128
    ss = torch.full((tiles, 256), float("nan"), device="cuda")
    hidden = resid.clone()
    K_.gemm(x, K_.pack_weight(w1), packed_shape=(H, I), residual=hidden, out=hidden, ss_out=ss, status=status,
            force_splits=splits)
    ref_h = (x.float() @ w1.float().t() + resid.float())
    _close(hidden, ref_h, dt, scale=max(1.0, ref_h.abs().max().item()))
    want_ss = hidden.float().pow(2).view(M, tiles, -1).sum(-1).t()             # [tiles, M] of the rows as stored
    torch.testing.assert_close(ss[:, :M], want_ss, rtol=1e-4, atol=1e-3)
    w2f = (w2.float() * nw.float()[None]).to(dt)                                # norm weights folded into the columns
    y = K_.gemm(hidden, K_.pack_weight(w2f, 2), packed_shape=(2 * I, H), bias=bias, act="silu_mul", dual=True, ss_in=ss,
                ss_dim=H, ss_eps=1e-6, status=status)
    hn = hidden.float() * torch.rsqrt(hidden.float().pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()
    z = hn @ w2.float().t() + bias.float()
    ref = torch.nn.functional.silu(z[:, :I]) * z[:, I:]
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()) * (4 if dt == torch.bfloat16 else 1))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(128, 384, 1536), (128, 1536, 384), (41, 1536, 2048), (50, 1024, 4096), (31, 1024, 1024),
                                   (7, 72, 136), (130, 200, 72), (256, 512, 640), (1, 384, 384), (1028, 1152, 384), (600, 384, 1536)])
@pytest.mark.parametrize("packed", [False, True])
def test_gemm_small_latency_kernel(dt, M, N, K, packed, status, monkeypatch):
    """Shapes the latency-bound kernel takes (few rows, small weight): every epilogue option against fp32 PyTorch, and the
    same call with the kernel switched off (the streaming kernel) within rounding."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    b = torch.randn(N, device="cuda").to(dt)
    r = torch.randn(M, N, device="cuda").to(dt)
    wk = K_.pack_weight(w) if packed else w
    kw = dict(packed_shape=(N, K)) if packed else {}
    ref = x.float() @ w.float().t()
    _close(K_.gemm(x, wk, **kw), ref, dt, scale=max(1.0, float(ref.abs().max())))
    full = torch.nn.functional.gelu(ref + b.float(), approximate="tanh") + r.float()
    got = K_.gemm(x, wk, bias=b, act="gelu_tanh", residual=r, **kw)
    _close(got, full, dt, scale=max(1.0, float(full.abs().max())))
    # per-column factor before the bias (the gate of a gated residual): r + (x.w^T * s + b)
    sc = (torch.randn(N, device="cuda") * 0.5).to(dt)
    gated = ref * sc.float() + b.float() + r.float()
    _close(K_.gemm(x, wk, scale=sc, bias=b, residual=r, **kw), gated, dt, scale=max(1.0, float(gated.abs().max())))
    # strided output / input views
    buf = torch.zeros(M, N + 16, device="cuda", dtype=dt)
    K_.gemm(x, wk, out=buf[:, 8:8 + N], **kw)
    _close(buf[:, 8:8 + N], ref, dt, scale=max(1.0, float(ref.abs().max())))
    assert float(buf[:, :8].abs().max()) == 0 and float(buf[:, 8 + N:].abs().max()) == 0


def test_gemm_forced_wide_tile_over_odd_block_count(status):
    """A forced 256-wide tile on a tile-major weight with an odd number of 128-row blocks (N = 1152: nine) falls back to
    128-wide tiles instead of copying a tenth block that is not there; token-row split K (pushed partial slices) on
    the same shape at 2 and 4 splits."""
    from rhinoforge_b200.ops import kernels as K_
    M, N, K = 768, 1152, 1152
    x = (torch.randn(M, K, device="cuda") * 0.5).half()
    w = (torch.randn(N, K, device="cuda") * 0.05).half()
    r = torch.randn(M, N, device="cuda").half()
    wp = K_.pack_weight(w)
    ref = x.float() @ w.float().t() + r.float()
    for kw in (dict(force_bn=256), dict(force_bn=256, force_splits=2), dict(force_bn=128, force_splits=4), dict(force_splits=3)):
        got = K_.gemm(x, wp, packed_shape=(N, K), residual=r, status=status, **kw)
        _close(got, ref, torch.float16, scale=max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(50, 4096, 1024), (128, 1536, 384), (31, 136, 200)])
@pytest.mark.parametrize("packed", [False, True])
def test_gemm_small_dual_glu(dt, M, N, K, packed, status):
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(2 * N, K, device="cuda") * 0.05).to(dt)
    b = (torch.randn(2 * N, device="cuda") * 0.1).to(dt)
    wk = K_.pack_weight(w, sections=2) if packed else w
    kw = dict(packed_shape=(2 * N, K)) if packed else {}
    gte, up = x.float() @ w[:N].float().t() + b[:N].float(), x.float() @ w[N:].float().t() + b[N:].float()
    ref = torch.nn.functional.silu(gte) * up
    got = K_.gemm(x, wk, bias=b, act="silu_mul", dual=True, **kw)
    _close(got, ref, dt, scale=max(1.0, float(ref.abs().max())))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,splits", [(1, 128, 512, 8), (16, 136, 576, 3), (17, 1000, 640, 2), (65, 264, 1024, 4), (93, 300, 1024, 8),
                                          (33, 7, 256, 1), (130, 640, 512, 1), (256, 384, 256, 2)])
@pytest.mark.parametrize("vec", [True, False])
def test_gemm_weight_row_epilogue(dt, M, N, K, splits, vec, status):
    """Few tokens, weights on the MMA rows: parked partials, the splits' sums and the eight-feature finish against fp32 - one split in
    passes of 64 (32 for a GLU) tokens, two to eight splits, token and feature counts that end inside a group, operands that cannot be
    read as 16-byte vectors."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(2 * N, K, device="cuda") * 0.05).to(dt)
    off, pitch = (0, (N + 7) // 8 * 8) if vec else (1, N + 3)
    vector = lambda n, base: (base + 0.2 * torch.randn(n + 1, device="cuda")).to(dt)[off:off + n]
    b, sc, r = vector(N, 0.0), vector(N, 1.0), torch.randn(M, pitch, device="cuda").to(dt)[:, :N]
    out = torch.full((M, pitch), 7.0, device="cuda").to(dt)
    y = K_.gemm(x, K_.pack_weight(w[:N]), packed_shape=(N, K), bias=b, scale=sc, residual=r, out=out[:, :N], status=status, force_splits=splits, force_swap=1)
    z = x.float() @ w.float().t()
    ref = z[:, :N] * sc.float() + b.float() + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))
    assert bool((out[:, N:] == 7.0).all())
    glu = lambda: K_.gemm(x, K_.pack_weight(w, 2), packed_shape=(2 * N, K), act="silu_mul", dual=True, status=status, force_splits=splits, force_swap=1)
    if splits > 1 and (M + 15) // 16 * 16 * 2 * 128 * 4 > 226 * 1024:          # two parked accumulators of fp32 [tokens][128] do not fit shared memory
        with pytest.raises(Exception, match="partial"):
            glu()
    else:
        _close(glu(), torch.nn.functional.silu(z[:, :N]) * z[:, N:], dt, scale=2.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(5000, 1152, 256), (4100, 4304, 128), (2500, 136, 520), (768, 4304, 1152), (825, 2560, 2048), (6000, 328, 64)])
@pytest.mark.parametrize("vec", [True, False])
def test_gemm_persistent_epilogue(dt, M, N, K, vec, status):
    """Persistent kernel: column tiles that end in the middle of a weight block or before their second one, bias and scale from the lanes
    of a warp, the residual added ahead of the staged store, operands that cannot be read as 16-byte vectors."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(dt)
    wp = K_.pack_weight(w)
    off, pitch = (0, N + 8) if vec else (1, N + 3)
    vector = lambda n, base: (base + 0.2 * torch.randn(n + 1, device="cuda")).to(dt)[off:off + n]
    b, sc, r = vector(N, 0.0), vector(N, 1.0), torch.randn(M, pitch, device="cuda").to(dt)
    rs = torch.rand(M, device="cuda") + 0.5
    z = x.float() @ w.float().t()
    ref = z * rs[:, None] * sc.float() + b.float() + r[:, :N].float()
    scale = max(1.0, ref.abs().max().item())
    _close(K_.gemm(x, wp, packed_shape=(N, K), bias=b, scale=sc, row_scale=rs, residual=r[:, :N], status=status), ref, dt, scale=scale)
    acc = r.clone()
    K_.gemm(x, wp, packed_shape=(N, K), bias=b, act="gelu_tanh", residual=acc[:, :N], out=acc[:, :N], status=status)
    ref = torch.nn.functional.gelu(z + b.float(), approximate="tanh") + r[:, :N].float()
    _close(acc[:, :N], ref, dt, scale=scale)
    assert torch.equal(acc[:, N:], r[:, N:])


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(257, 1152, 1152), (511, 2568, 520), (769, 2048, 4104), (2100, 1096, 1160), (9000, 2048, 136), (4097, 8, 1032), (20000, 1032, 264)])
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_cta_pairs(dt, M, N, K, dual, status):
    """Tiles shared by two CTAs: last tiles whose second CTA has no rows or whose second half has no columns, a partial k block, fewer k blocks than
    ring stages, one and several tiles to a pair, 128 and 256 columns, every epilogue option, the residual in the output's place."""
    from rhinoforge_b200.ops import kernels as K_
    assert dual or K_.gemm_plan(M, N, K, dtype=dt)["kernel"] == "persistent"
    rows = 2 * N if dual else N
    x = (torch.randn(M, K + 8, device="cuda") * 0.5).to(dt)[:, :K]
    w = (torch.randn(rows, K, device="cuda") / K ** 0.5).to(dt)
    b, sc = torch.randn(rows, device="cuda").to(dt), (torch.rand(rows, device="cuda") + 0.5).to(dt)
    rs, r = torch.rand(M, device="cuda") + 0.5, torch.randn(M, N + 8, device="cuda").to(dt)[:, :N]
    out = torch.full((M + 1, N + 8), 7.0, device="cuda").to(dt)
    kw = dict(packed_shape=(rows, K), status=status, **(dict(act="silu_mul", dual=True) if dual else {}))
    finish = lambda z: torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    wp, z = K_.pack_weight(w, 2 if dual else 1), x.float() @ w.float().t()
    _close(K_.gemm(x, wp, out=out[:M, :N], **kw), finish(z), dt)
    full = dict(bias=b, scale=sc, row_scale=rs)
    ref = finish(z * rs[:, None] * sc.float() + b.float()) + r.float()
    _close(K_.gemm(x, wp, residual=r, out=out[:M, :N], **full, **kw), ref, dt, scale=2.0)
    assert bool((out[M:] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
    acc = r.clone()
    _close(K_.gemm(x, wp, residual=acc, out=acc, **full, **kw), ref, dt, scale=2.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (1, 1000, 72), (7, 264, 520), (8, 40, 8), (9, 1536, 1024), (16, 5000, 1160), (3, 24, 4096), (16, 7, 2048)])
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_very_few_rows(dt, M, N, K, dual, status):
    """Up to 16 rows over 16-bit weights: strips of 16 features that end inside a weight block or past N, fewer k blocks than warps and
    partial ones, every epilogue option, strided and odd-pitched outputs, a CTA that takes several strips; the RMSNorm that the kernel
    folds in itself, or takes from given sums."""
    from rhinoforge_b200.ops import kernels as K_
    rows = 2 * N if dual else N
    x = (torch.randn(M, K + 8, device="cuda") * 0.5).to(dt)[:, :K]
    w = (torch.randn(rows, K, device="cuda") / K ** 0.5).to(dt)
    wp = K_.pack_weight(w, 2 if dual else 1)
    b, sc = torch.randn(rows, device="cuda").to(dt), (torch.rand(rows, device="cuda") + 0.5).to(dt)
    rs, r = torch.rand(M, device="cuda") + 0.5, torch.randn(M, N, device="cuda").to(dt)
    out = torch.full((M, N + 3), 7.0, device="cuda").to(dt)
    kw = dict(packed_shape=(rows, K), status=status, **(dict(act="silu_mul", dual=True) if dual else {}))
    finish = lambda z: torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    K_.gemm(x, wp, bias=b, scale=sc, row_scale=rs, residual=r, out=out[:, :N], **kw)
    z = x.float() @ w.float().t()
    _close(out[:, :N], finish(z * rs[:, None] * sc.float() + b.float()) + r.float(), dt, scale=2.0)
    assert bool((out[:, N:] == 7.0).all())
    ss = torch.zeros((max(K // 128, 1), 256), device="cuda")
    ss[0, :M] = x.float().pow(2).sum(1)
    normed = finish(z * torch.rsqrt(x.float().pow(2).mean(1, keepdim=True) + 1e-6))
    _close(K_.gemm(x, wp, ss_in=ss, ss_dim=K, ss_eps=1e-6, **kw), normed, dt, scale=4.0)          # the sums are given: another kernel
    # long rows of 8 rows, and large weights of more, are other kernels' (the dispatcher's rule)
    if M * K <= 80 << 10 if M <= 8 and not dual else dual or N * K <= 8 << 20:
        _close(K_.gemm(x, wp, norm_x=True, ss_eps=1e-6, **kw), normed, dt, scale=4.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M", [1, 8, 11, 16])
@pytest.mark.parametrize("N,K,group,fp4", [(264, 320, 0, False), (1000, 1024, 64, False), (40, 2176, 32, False), (128, 192, 16, True), (5008, 512, None, False), (24, 4672, 0, False), (40, 4672, 32, False)])
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_very_few_rows_quantised(dt, M, N, K, group, fp4, dual, status):
    """Up to 16 rows over int8 (``group`` None) and 4-bit weights, against the product with the values that the image holds."""
    from rhinoforge_b200.ops import kernels as K_
    rows = 2 * N if dual else N
    x = (torch.randn(M, K, device="cuda") / K ** 0.5).to(dt)
    sc = (torch.rand(rows, device="cuda") * 0.2 + 0.1).to(dt)
    kw = dict(packed_shape=(rows, K), status=status, **(dict(act="silu_mul", dual=True) if dual else {}))
    sections = 2 if dual else 1
    if group is None:
        q = torch.randint(-127, 128, (rows, K), device="cuda", dtype=torch.int8)
        y, w = K_.gemm(x, K_.pack_weight(q, sections), scale=sc, **kw), q.float() * sc.float()[:, None]
    else:
        q = torch.randint(-8, 8, (rows, K), device="cuda", dtype=torch.int8)
        gs = (torch.rand(rows, K // group, device="cuda") * 0.2 + 0.1).to(dt) if group else None
        value = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6], device="cuda")[(q & 15).long()] if fp4 else q.float()
        img = K_.pack_weight_int4(q, gs, group, sections=sections, dtype=dt)
        y = K_.gemm(x, img, w_bits=4, w_group=group, w_fp4=fp4, scale=None if group else sc, **kw)
        w = (value.view(rows, -1, group) * gs.float()[..., None]).view(rows, K).to(dt).float() if group else value * sc.float()[:, None]
    z = x.float() @ w.t()
    ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 32, 8), (128, 32, 4)])
@pytest.mark.parametrize("mode", ["causal", "window", "full", "mask"])
def test_attn_prefill_two_tiles(dt, hd, Hq, Hkv, mode, status):
    """Enough heads and rows that a CTA takes two query tiles: second tiles that are empty, partial and full, keys ahead of the new rows, tiles that
    stop at different blocks, and the masks that leave a tile's first blocks empty - paged against fp32, contiguous against paged."""
    from rhinoforge_b200.ops import kernels as K_
    q_lens, kv_lens = [257, 100, 384, 129], [257, 420, 400, 129]
    k_pool, v_pool, pt, ks, vs = _paged(Hkv, hd, kv_lens, dt)
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    starts = [sum(q_lens[:i]) for i in range(len(q_lens))]
    q = torch.randn(sum(q_lens), Hq * hd, device="cuda").to(dt)
    kw = dict(Hq=Hq, Hkv=Hkv, hd=hd, q_start=i32(starts), q_len=i32(q_lens), kv_len=i32(kv_lens), max_q_len=max(q_lens), causal=mode in ("causal", "window"),
              window=70 if mode == "window" else 0, status=status)
    given = torch.rand(len(q_lens), max(q_lens), 432, device="cuda") > 0.4
    given[:, :, 0] = True
    if mode == "mask":
        kw["mask"] = given
    out = K_.attention_prefill(q, torch.zeros_like(q), k_pool=k_pool, v_pool=v_pool, page_table=pt, **kw)
    flat = lambda parts: torch.cat([t.transpose(0, 1).reshape(t.shape[1], Hkv * hd) for t in parts])
    rows = K_.attention_prefill(q, torch.zeros_like(q), k=flat(ks), v=flat(vs), kv_start=i32([sum(kv_lens[:i]) for i in range(len(kv_lens))]), **kw)
    assert torch.equal(out, rows)
    for s, (Lq, Lk) in enumerate(zip(q_lens, kv_lens)):
        qs = q[starts[s]:starts[s] + Lq].view(Lq, Hq, hd).transpose(0, 1)
        i, j = torch.arange(Lq, device="cuda")[:, None] + (Lk - Lq), torch.arange(Lk, device="cuda")[None]
        mask = torch.ones(Lq, Lk, dtype=torch.bool, device="cuda") if mode == "full" else given[s, :Lq, :Lk] if mode == "mask" else j <= i
        if mode == "window":
            mask = mask & (j > i - 70)
        ref = _sdpa_ref(qs, ks[s], vs[s], mask).transpose(0, 1).reshape(Lq, Hq * hd)
        _close(out[starts[s]:starts[s] + Lq], ref, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("causal", [False, True])
def test_attn_prefill_of_sequences_without_keys(dt, hd, causal, status):
    """Query rows of a sequence that has no keys come out as zeros, beside one that has; more rows than a tile."""
    from rhinoforge_b200.ops import kernels as K_
    heads, q_lens, kv_lens = 4, [200, 300, 5], [200, 0, 0]
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    q, k, v = (torch.randn(sum(q_lens), heads * hd, device="cuda").to(dt) for _ in range(3))
    out = torch.full_like(q, 7.0)
    K_.attention_prefill(q, out, Hq=heads, Hkv=heads, hd=hd, q_start=i32([0, 200, 500]), q_len=i32(q_lens), kv_len=i32(kv_lens), kv_start=i32([0, 200, 200]),
                         max_q_len=300, k=k, v=v, causal=causal, status=status)
    assert not out[200:].any()
    h = lambda t: t[:200].view(200, heads, hd).transpose(0, 1)
    mask = torch.ones(200, 200, dtype=torch.bool, device="cuda")
    _close(out[:200], _sdpa_ref(h(q), h(k), h(v), mask.tril() if causal else mask).transpose(0, 1).reshape(200, heads * hd), dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("heads,lens", [(2, [16, 1, 65]), (16, [256, 256, 256]), (32, [300, 513, 129, 64])])
@pytest.mark.parametrize("mode", ["full", "causal", "mask"])
def test_attn_prefill_heads_of_80(dt, heads, lens, mode, status):
    """Heads of 80 over rows of one QKV buffer: the second box of a head runs into the next one, of the last head past the row's end."""
    from rhinoforge_b200.ops import kernels as K_
    T, n, hd = sum(lens), heads * 80, 80
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    starts = [sum(lens[:i]) for i in range(len(lens))]
    qkv = torch.randn(T, 3 * n, device="cuda").to(dt)
    kw = dict(Hq=heads, Hkv=heads, hd=hd, q_start=i32(starts), q_len=i32(lens), kv_len=i32(lens), kv_start=i32(starts), max_q_len=max(lens),
              causal=mode == "causal", status=status)
    given = torch.rand(len(lens), max(lens), (max(lens) + 15) // 16 * 16, device="cuda") > 0.4
    given[:, :, 0] = True
    if mode == "mask":
        kw["mask"] = given
    out = K_.attention_prefill(qkv, torch.zeros(T, n, device="cuda", dtype=dt), k=qkv[:, n:2 * n], v=qkv[:, 2 * n:], **kw)
    for s, L in enumerate(lens):
        q, k, v = (qkv[starts[s]:starts[s] + L, i * n:(i + 1) * n].view(L, heads, hd).transpose(0, 1) for i in range(3))
        mask = torch.ones(L, L, dtype=torch.bool, device="cuda")
        mask = mask.tril() if mode == "causal" else given[s, :L, :L] if mode == "mask" else mask
        _close(out[starts[s]:starts[s] + L], _sdpa_ref(q, k, v, mask).transpose(0, 1).reshape(L, n), dt)
    with pytest.raises(Exception, match="80"):
        K_.attention_decode(qkv[:, :n], out, Hq=heads, Hkv=heads, hd=hd, kv_len=i32([1] * T), max_kv_len=16,
                            k_pool=torch.zeros(1, heads, 16, hd, device="cuda", dtype=dt), v_pool=torch.zeros(1, heads, 16, hd, device="cuda", dtype=dt),
                            page_table=i32([[0]] * T), ws=K_.attn_decode_scratch(T, heads, hd, "cuda"))


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K", [(1, 4744, 64), (3, 5000, 1040), (8, 4768, 2048), (9, 9999, 528), (16, 20001, 1024)])
def test_gemm_very_few_rows_int8_wide(dt, M, N, K, status):
    """int8 weights in strips of 32 features: a last strip with one group of 16 or part of it, fewer k blocks than warps, several strips to a CTA, scale,
    bias, residual and an odd output pitch."""
    from rhinoforge_b200.ops import kernels as K_
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    q = torch.randint(-127, 128, (N, K), device="cuda", dtype=torch.int8)
    sc, b = (torch.rand(N, device="cuda") * 0.02 + 0.002).to(dt), torch.randn(N, device="cuda").to(dt)
    r, out = torch.randn(M, N, device="cuda").to(dt), torch.full((M, N + 3), 7.0, device="cuda").to(dt)
    assert K_.gemm_plan(M, N, K, dtype=dt, int8=True)["kernel"] == "rows"
    y = K_.gemm(x, K_.pack_weight(q), packed_shape=(N, K), scale=sc, bias=b, residual=r, out=out[:, :N], status=status)
    ref = x.float() @ q.float().t() * sc.float() + b.float() + r.float()
    _close(y, ref, dt, scale=max(1.0, ref.abs().max().item()))
    assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv,rot", [(64, 8, 8, 64), (64, 32, 2, 32), (128, 16, 8, 128), (128, 14, 1, 0), (256, 8, 1, 64)])
@pytest.mark.parametrize("lens", [[300], [1, 16, 17, 33, 160], [700] * 40, [1500, 15, 16, 3000, 2, 999, 64]])
@pytest.mark.parametrize("mode", [(True, 0, 0), (True, 1, 1), (False, 0, 0)])
def test_attn_decode_inserts(dt, hd, Hq, Hkv, rot, lens, mode, status):
    """Decode attention that normalises, rotates and inserts itself against the two launches, bit for bit, pool included: new tokens in the first and
    last row of a page and in a page of their own, one and several splits, a row whose token goes nowhere, one that lies behind the keys read."""
    import ctypes as C
    from rhinoforge_b200 import _native as N
    from rhinoforge_b200.ops import kernels as K_
    norms, gemma, rope_first = mode
    n, maxp = len(lens), (max(lens) + 15) // 16 + 2
    g = torch.Generator(device="cuda").manual_seed(hd + n)
    qkv = torch.randn(n, (Hq + 2 * Hkv) * hd + 8, device="cuda", generator=g).to(dt)
    pools = torch.randn(2, n * maxp, Hkv, 16, hd, device="cuda", generator=g).to(dt)
    pt = torch.randperm(n * maxp, device="cuda", generator=g).to(torch.int32).view(n, maxp)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    kv_len, pos = i32(lens), i32([l - 1 for l in lens])
    cache_pos = pos.clone()
    if n > 2:
        cache_pos[1], cache_pos[2] = -1, cache_pos[2] + 16
    cos, sin = torch.randn(max(lens), max(rot, 2) // 2, device="cuda"), torch.randn(max(lens), max(rot, 2) // 2, device="cuda")
    qn, kn = (1 + 0.1 * torch.randn(2, hd, device="cuda")).to(dt)
    ws = K_.attn_decode_scratch(n, Hq, hd, "cuda")

    def run(fused):
        rows, kp, vp = qkv.clone(), pools[0].clone(), pools[1].clone()
        out = torch.zeros(n, Hq * hd, device="cuda", dtype=dt)
        r, a = N.RfRopeKv(), N.RfAttn()
        r.qkv, r.ld, r.tokens, r.Hq, r.Hkv, r.hd, r.rot_dim = rows.data_ptr(), rows.stride(0), n, Hq, Hkv, hd, rot
        if norms:
            r.q_norm_w, r.k_norm_w = qn.data_ptr(), kn.data_ptr()
        r.eps, r.norm_mode, r.rope_before_norm, r.dtype = 1e-6, gemma, rope_first, 0 if dt == torch.float16 else 1
        r.cos, r.sin, r.pos, r.pos_stride, r.cache_pos = cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), 1, cache_pos.data_ptr()
        r.k_pool, r.v_pool, r.page_table, r.pt_stride = kp.data_ptr(), vp.data_ptr(), pt.data_ptr(), maxp
        a.q, a.ldq, a.out, a.ldo, a.q_rows_total = rows.data_ptr(), rows.stride(0), out.data_ptr(), out.stride(0), n
        a.k_pool, a.v_pool, a.pool_pages, a.page_table, a.pt_stride = kp.data_ptr(), vp.data_ptr(), n * maxp, pt.data_ptr(), maxp
        a.num_seqs, a.Hq, a.Hkv, a.hd, a.kv_len, a.max_kv_len, a.dtype = n, Hq, Hkv, hd, kv_len.data_ptr(), max(lens), r.dtype
        a.ws, a.ws_bytes, a.status, a.rows_per_seq = ws.data_ptr(), ws.numel() * 4, status.data_ptr(), 1
        L, st = N.lib(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if fused:
            assert L.rf_attn_decode_inserts(C.byref(a), C.byref(r)) == 1
            N.check(L.rf_attn_decode_insert(C.byref(a), C.byref(r), st), "insert")
            assert torch.equal(rows, qkv)
            r.seq_of_tok = pos.data_ptr()                       # a token that may belong elsewhere: two launches, refused here
            assert L.rf_attn_decode_inserts(C.byref(a), C.byref(r)) == 0 and L.rf_attn_decode_insert(C.byref(a), C.byref(r), st) != 0
        else:
            N.check(L.rf_qk_norm_rope_kv(C.byref(r), st), "rope")
            N.check(L.rf_attn_decode(C.byref(a), st), "decode")
        return out, kp, vp

    for x, y in zip(run(True), run(False)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("longest", [40, 1500])
def test_attn_decode_of_a_row_without_pages(dt, hd, longest, status):
    """Rows that see nothing (position -1, no table row: -1) beside rows that do: zeros for them, the others as without them, one and several splits."""
    from rhinoforge_b200.ops import kernels as K_
    Hq, Hkv, maxp = 8, 2, (longest + 15) // 16
    g = torch.Generator(device="cuda").manual_seed(hd)
    q = torch.randn(4, Hq * hd, device="cuda", generator=g).to(dt)
    kp, vp = torch.randn(2, 2 * maxp, Hkv, 16, hd, device="cuda", generator=g).to(dt)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    pt = torch.randperm(2 * maxp, device="cuda", generator=g).to(torch.int32).view(2, maxp)
    pos, slot = [longest - 1, -1, 6, -1], [1, -1, 0, -1]
    run = lambda rows: K_.attention_rows(q[rows].contiguous(), K_.rows(i32([pos[r] for r in rows]), slot=i32([slot[r] for r in rows]), page_table=pt), kp, vp, Hq=Hq,
                                         Hkv=Hkv, hd=hd, scale=hd ** -0.5, max_kv=longest)
    got, want = run([0, 1, 2, 3]), run([0, 2])
    torch.testing.assert_close(got[[0, 2]].float(), want.float(), rtol=0, atol=2e-3 if dt == torch.float16 else 1.6e-2)     # other splits: one rounding of values below 1
    assert not got[[1, 3]].any()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 8, 2), (128, 16, 8), (256, 8, 1)])
@pytest.mark.parametrize("lens", [[33, 16, 7], [1500, 700, 15]])
def test_attn_decode_inserts_nothing_into_a_page_of_nobody(dt, hd, Hq, Hkv, lens, status):
    """A new token whose page number is negative, among the keys read and behind them: nothing is written, not in front of the pool either, and the
    page reads as zeros, bit for bit as with the two launches."""
    import ctypes as C
    from rhinoforge_b200 import _native as N
    from rhinoforge_b200.ops import kernels as K_
    n, maxp = len(lens), (max(lens) + 15) // 16 + 2
    g = torch.Generator(device="cuda").manual_seed(hd)
    qkv = torch.randn(n, (Hq + 2 * Hkv) * hd, device="cuda", generator=g).to(dt)
    room = torch.randn(2, n * maxp + 2, Hkv, 16, hd, device="cuda", generator=g).to(dt)           # a page in front of each pool and one behind
    pt = torch.randperm(n * maxp, device="cuda", generator=g).to(torch.int32).view(n, maxp)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    kv_len, pos = i32(lens), i32([l - 1 for l in lens])
    pt[0, (lens[0] - 1) // 16] = -1
    pos[1] += 16
    pt[1, (lens[1] + 15) // 16] = -1
    cos, sin = torch.randn(2, max(lens) + 16, hd // 2, device="cuda", generator=g)
    ws = K_.attn_decode_scratch(n, Hq, hd, "cuda")

    def run(fused):
        rows, buf, out = qkv.clone(), room.clone(), torch.zeros(n, Hq * hd, device="cuda", dtype=dt)
        r, a = N.RfRopeKv(), N.RfAttn()
        r.qkv, r.ld, r.tokens, r.Hq, r.Hkv, r.hd, r.rot_dim, r.dtype = rows.data_ptr(), rows.stride(0), n, Hq, Hkv, hd, hd, 0 if dt == torch.float16 else 1
        r.cos, r.sin, r.pos, r.pos_stride, r.cache_pos = cos.data_ptr(), sin.data_ptr(), pos.data_ptr(), 1, pos.data_ptr()
        r.k_pool, r.v_pool, r.page_table, r.pt_stride = buf[0, 1:].data_ptr(), buf[1, 1:].data_ptr(), pt.data_ptr(), maxp
        a.q, a.ldq, a.out, a.ldo, a.q_rows_total = rows.data_ptr(), rows.stride(0), out.data_ptr(), out.stride(0), n
        a.k_pool, a.v_pool, a.pool_pages, a.page_table, a.pt_stride = r.k_pool, r.v_pool, n * maxp, pt.data_ptr(), maxp
        a.num_seqs, a.Hq, a.Hkv, a.hd, a.kv_len, a.max_kv_len, a.dtype = n, Hq, Hkv, hd, kv_len.data_ptr(), max(lens), r.dtype
        a.ws, a.ws_bytes, a.status, a.rows_per_seq = ws.data_ptr(), ws.numel() * 4, status.data_ptr(), 1
        L, st = N.lib(), C.c_void_p(torch.cuda.current_stream().cuda_stream)
        if fused:
            assert L.rf_attn_decode_inserts(C.byref(a), C.byref(r)) == 1
            N.check(L.rf_attn_decode_insert(C.byref(a), C.byref(r), st), "insert")
        else:
            N.check(L.rf_qk_norm_rope_kv(C.byref(r), st), "rope")
            N.check(L.rf_attn_decode(C.byref(a), st), "decode")
        return out, buf

    got, buf = run(True)
    want, ref = run(False)
    assert torch.equal(got, want) and torch.equal(buf, ref)
    assert torch.equal(buf[:, :1], room[:, :1]) and torch.equal(buf[:, -1:], room[:, -1:])


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H", [8, 264, 1024, 1152, 2040, 3072, 4096, 4104])
@pytest.mark.parametrize("rows", [295, 1301, 3001])
def test_norms_of_many_rows(dt, H, rows):
    """A warp per row (by rows per SM, length and operands, up to 4096 values): rows that end inside a piece, a last block with idle warps, residual
    and modulation, pitched rows, in place - and sizes past each end of that range on the block kernels."""
    from rhinoforge_b200.ops import kernels as K_
    x = torch.randn(rows, H, device="cuda").to(dt)
    r = torch.randn(rows, H, device="cuda").to(dt)
    w, b = (1 + 0.1 * torch.randn(H, device="cuda")).to(dt), torch.randn(H, device="cuda").to(dt)
    mod = torch.randn((rows + 6) // 7, 3 * H, device="cuda").to(dt)
    rms = lambda t: t.float() * torch.rsqrt(t.float().pow(2).mean(-1, keepdim=True) + 1e-6)
    _close(K_.layernorm(x, w, b, 1e-6), torch.nn.functional.layer_norm(x.float(), (H,), w.float(), b.float(), 1e-6), dt, scale=2.0)
    total, out = torch.empty_like(x), torch.empty(rows, H + 8, device="cuda", dtype=dt)
    K_.rmsnorm(x, w, 1e-6, residual=r, residual_out=total, out=out[:, :H])
    assert torch.equal(total, (x.float() + r.float()).to(dt))
    _close(out[:, :H], rms(total) * w.float(), dt, scale=2.0)
    _close(K_.rmsnorm(x, w, 1e-6, gemma=True), rms(x) * (1 + w.float()), dt, scale=4.0)
    m = mod.float().repeat_interleave(7, 0)[:rows]
    _close(K_.rmsnorm(x, None, 1e-6, mod=mod, rows_per_mod=7), rms(x) * (1 + m[:, :H]) + m[:, H:2 * H], dt, scale=6.0)
    y = x.clone()
    K_.rmsnorm(y, None, 1e-6, out=y)
    _close(y, rms(x), dt, scale=2.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,rot,Hq,Hkv", [(64, 64, 3, 1), (128, 64, 5, 2), (128, 128, 16, 8), (256, 96, 2, 1), (64, 24, 4, 4)])
@pytest.mark.parametrize("T", [1, 3, 77, 600])
def test_rope_kv_few_and_many_tokens_agree(dt, hd, rot, Hq, Hkv, T):
    """Norm, rotation and page insertion of the same rows at every launch size (and on the scalar kernel, which takes rotations that are no multiple
    of 16): heads that do not fill the last warp, tables that are and are not 16-byte aligned, one and three position axes, in place and paged."""
    from rhinoforge_b200.ops import kernels as K_
    width = (Hq + 2 * Hkv) * hd
    qkv = torch.randn(T, width, device="cuda").to(dt)
    w = [(1 + 0.1 * torch.randn(hd, device="cuda")).to(dt) for _ in range(2)]
    ang = torch.rand(T + 9, rot // 2, device="cuda") * 6.0
    table = torch.stack((ang.cos(), ang.sin()))
    shifted = torch.empty(table.numel() + 1, device="cuda")[1:].view_as(table).copy_(table)          # 4-byte aligned only
    pos3 = torch.randint(0, T + 9, (T, 3), dtype=torch.int32, device="cuda")
    axis = (torch.arange(rot // 2) % 3).to(torch.int8).cuda()
    pt = torch.randperm((T + 15) // 16 + 2, device="cuda").to(torch.int32)[None].repeat(T, 1).contiguous()
    seq, cpos = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")

    def ref(pos_of):
        x = qkv.view(T, -1, hd).float()
        parts = []
        for heads, wt in ((x[:, :Hq], w[0]), (x[:, Hq:Hq + Hkv], w[1])):
            n = wt.float() * (heads * torch.rsqrt(heads.pow(2).mean(-1, keepdim=True) + 1e-6)).to(dt).float()
            n = n.to(dt).float()
            c, s = (torch.gather(t, 0, pos_of.long())[:, None] for t in table)
            u, v = n[..., :rot // 2], n[..., rot // 2:rot]
            parts.append(torch.cat((u * c - v * s, v * c + u * s, n[..., rot:]), -1))
        return parts

    for cos_sin, three in ((table, False), (shifted, False), (table, True)):
        pos = pos3 if three else pos3[:, 0].contiguous()
        pos_of = pos3[:, axis.long()] if three else pos3[:, :1].expand(T, rot // 2)
        q_ref, k_ref = ref(pos_of)
        k_pool = torch.zeros(pt.shape[1], Hkv, 16, hd, device="cuda", dtype=dt)
        v_pool, rows = torch.zeros_like(k_pool), qkv.clone()
        K_.qk_norm_rope_kv(rows, Hq, Hkv, hd, pos=pos, cos=cos_sin[0], sin=cos_sin[1], rot_dim=rot, q_norm_w=w[0], k_norm_w=w[1], k_pool=k_pool, v_pool=v_pool,
                           page_table=pt, seq_of_tok=seq, cache_pos=cpos, axis_of_freq=axis if three else None)
        got = rows.view(T, -1, hd)
        at = lambda pool: pool[pt[0][(cpos // 16).long()].long(), :, (cpos % 16).long()]
        _close(got[:, :Hq], q_ref, dt, scale=3.0)
        _close(at(k_pool), k_ref, dt, scale=3.0)
        assert torch.equal(at(v_pool), qkv.view(T, -1, hd)[:, Hq + Hkv:])
        assert torch.equal(got[:, Hq:], qkv.view(T, -1, hd)[:, Hq:])
        flat = qkv.clone()
        K_.qk_norm_rope_kv(flat, Hq, Hkv, hd, pos=pos, cos=cos_sin[0], sin=cos_sin[1], rot_dim=rot, q_norm_w=w[0], k_norm_w=w[1], axis_of_freq=axis if three else None)
        _close(flat.view(T, -1, hd)[:, Hq:Hq + Hkv], k_ref, dt, scale=3.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 6, 2), (128, 32, 8), (128, 40, 2), (256, 8, 1)])
@pytest.mark.parametrize("rows", [1, 2, 7, 50])
@pytest.mark.parametrize("lens", [[1, 300, 131], [5000]])
def test_attn_decode_rows_of_a_sequence(dt, hd, Hq, Hkv, rows, lens, status):
    """Several query rows of a sequence over all its keys: (row, head) pairs that fill, share and end inside a tile of 16, splits merged over a cluster
    (with and without empty ones) and, for 5000 keys, by the second kernel - against fp32 and against the unsplit kernel."""
    from rhinoforge_b200.ops import kernels as K_
    k_pool, v_pool, pt, ks, vs = _paged(Hkv, hd, lens, dt)
    q = torch.randn(len(lens) * rows, Hq * hd, device="cuda").to(dt)
    kw = dict(Hq=Hq, Hkv=Hkv, hd=hd, kv_len=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_kv_len=max(lens), k_pool=k_pool, v_pool=v_pool, page_table=pt,
              status=status, rows_per_seq=rows)
    out = K_.attention_decode(q, torch.full_like(q, float("nan")), ws=K_.attn_decode_scratch(q.shape[0], Hq, hd, "cuda"), **kw)
    whole = K_.attention_decode(q, torch.full_like(q, float("nan")), **kw)
    for s, L in enumerate(lens):
        at = slice(s * rows, (s + 1) * rows)
        ref = _sdpa_ref(q[at].view(rows, Hq, hd).transpose(0, 1), ks[s], vs[s], torch.ones(rows, L, dtype=torch.bool, device="cuda"))
        ref = ref.transpose(0, 1).reshape(rows, Hq * hd)
        _close(out[at], ref, dt)
        _close(whole[at], ref, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,T", [(64, 3), (128, 77), (128, 600), (80, 5)])
def test_rope_kv_without_positions(dt, hd, T):
    """Norm and page insertion by ``cache_pos`` alone: no tables, no positions (a null pointer), on the 16-byte and the scalar kernel."""
    import ctypes as C
    from rhinoforge_b200 import _native as N
    from rhinoforge_b200.ops import kernels as K_
    Hq, Hkv = 3, 2
    qkv = torch.randn(T, (Hq + 2 * Hkv) * hd, device="cuda").to(dt)
    w = (1 + 0.1 * torch.randn(hd, device="cuda")).to(dt)
    pt = torch.arange((T + 15) // 16 + 1, dtype=torch.int32, device="cuda").flip(0).contiguous()[None]
    seq, cpos = torch.zeros(T, dtype=torch.int32, device="cuda"), torch.arange(T, dtype=torch.int32, device="cuda")
    got = []
    for pos in (None, cpos):
        rows = qkv.clone()
        pools = torch.zeros(2, pt.shape[1], Hkv, 16, hd, device="cuda", dtype=dt)
        a = N.RfRopeKv()
        a.qkv, a.ld, a.tokens, a.Hq, a.Hkv, a.hd, a.rot_dim = rows.data_ptr(), rows.stride(0), T, Hq, Hkv, hd, 0
        a.q_norm_w, a.k_norm_w, a.eps, a.dtype = w.data_ptr(), w.data_ptr(), 1e-6, K_.dtype_code(dt)
        a.pos, a.pos_stride = None if pos is None else pos.data_ptr(), 1
        a.k_pool, a.v_pool, a.page_table, a.pt_stride = pools[0].data_ptr(), pools[1].data_ptr(), pt.data_ptr(), pt.stride(0)
        a.seq_of_tok, a.cache_pos = seq.data_ptr(), cpos.data_ptr()
        N.check(N.lib().rf_qk_norm_rope_kv(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "rf_qk_norm_rope_kv")
        got.append((rows, pools))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    rows = qkv.clone()
    a = N.RfRopeKv()                          # neither pool nor positions: norms in place
    a.qkv, a.ld, a.tokens, a.Hq, a.Hkv, a.hd, a.pos_stride = rows.data_ptr(), rows.stride(0), T, Hq, Hkv, hd, 1
    a.q_norm_w, a.k_norm_w, a.eps, a.dtype = w.data_ptr(), w.data_ptr(), 1e-6, K_.dtype_code(dt)
    N.check(N.lib().rf_qk_norm_rope_kv(C.byref(a), C.c_void_p(torch.cuda.current_stream().cuda_stream)), "rf_qk_norm_rope_kv")
    x = qkv.view(T, -1, hd).float()
    ref = w.float() * (x[:, :Hq + Hkv] * torch.rsqrt(x[:, :Hq + Hkv].pow(2).mean(-1, keepdim=True) + 1e-6)).to(dt).float()
    at = lambda pool: pool[pt[0][(cpos // 16).long()].long(), :, (cpos % 16).long()]
    _close(got[0][0].view(T, -1, hd)[:, :Hq], ref[:, :Hq], dt, scale=3.0)
    _close(rows.view(T, -1, hd)[:, :Hq + Hkv], ref, dt, scale=3.0)
    _close(at(got[0][1][0]), ref[:, Hq:], dt, scale=3.0)
    assert torch.equal(at(got[0][1][1]), qkv.view(T, -1, hd)[:, Hq + Hkv:])


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M", [1, 8, 11, 16, 17, 40])
@pytest.mark.parametrize("dual", [False, True])
def test_gemm_scaled_by_given_sums_or_by_its_own_squares(dt, M, dual, status):
    """``ss_in`` scales by the caller's sums at every row count, whatever x holds; ``norm_x`` by the squares of x, where there is a kernel for it."""
    from rhinoforge_b200.ops import kernels as K_
    N, K = 264, 640
    rows = 2 * N if dual else N
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(rows, K, device="cuda") / K ** 0.5).to(dt)
    wp = K_.pack_weight(w, 2 if dual else 1)
    kw = dict(packed_shape=(rows, K), status=status, **(dict(act="silu_mul", dual=True) if dual else {}))
    finish = lambda z: torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    z = x.float() @ w.float().t()
    sums = torch.rand(5, M + 3, device="cuda") * 40 + 1.0                   # nothing to do with x
    rstd = torch.rsqrt(sums[:, :M].sum(0) / 200 + 1e-5)
    ref = finish(z * rstd[:, None])
    _close(K_.gemm(x, wp, ss_in=sums, ss_dim=200, ss_eps=1e-5, **kw), ref, dt, scale=max(1.0, ref.abs().max().item()))
    own = finish(z * torch.rsqrt(x.float().pow(2).sum(1, keepdim=True) / 200 + 1e-5))
    if M <= 16:
        _close(K_.gemm(x, wp, norm_x=True, ss_dim=200, ss_eps=1e-5, **kw), own, dt, scale=max(1.0, own.abs().max().item()))
    else:
        with pytest.raises(Exception, match="squares of its rows"):
            K_.gemm(x, wp, norm_x=True, ss_dim=200, ss_eps=1e-5, **kw)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("hd,Hq,Hkv", [(64, 4, 2), (128, 8, 2), (256, 2, 1)])
@pytest.mark.parametrize("mode", ["full", "causal", "window"])
def test_attn_prefill_scattered_segments(dt, hd, Hq, Hkv, mode, status):
    """Segment ids in no order over sequences that end inside a block of keys, with keys ahead of the new rows, under causal and window masks too."""
    from rhinoforge_b200.ops import kernels as K_
    q_lens, kv_lens = [150, 1, 65, 290], [150, 70, 129, 300]
    i32 = lambda l: torch.tensor(l, dtype=torch.int32, device="cuda")
    starts = lambda lens: [sum(lens[:i]) for i in range(len(lens))]
    q = torch.randn(sum(q_lens), Hq * hd, device="cuda").to(dt)
    k, v = (torch.randn(sum(kv_lens), Hkv * hd, device="cuda").to(dt) for _ in range(2))
    seg_k = torch.randint(0, 4, (sum(kv_lens),), dtype=torch.int32, device="cuda")
    seg_q = torch.cat([seg_k[s + n - m:s + n] for s, n, m in zip(starts(kv_lens), kv_lens, q_lens)]).contiguous()      # a row sees itself
    out = K_.attention_prefill(q, torch.zeros_like(q), Hq=Hq, Hkv=Hkv, hd=hd, q_start=i32(starts(q_lens)), q_len=i32(q_lens), kv_len=i32(kv_lens),
                               max_q_len=max(q_lens), k=k, v=v, kv_start=i32(starts(kv_lens)), causal=mode != "full", window=70 if mode == "window" else 0,
                               seg_q=seg_q, seg_k=seg_k, status=status)
    for a, b, m, n in zip(starts(q_lens), starts(kv_lens), q_lens, kv_lens):
        i, j = torch.arange(m, device="cuda")[:, None] + (n - m), torch.arange(n, device="cuda")[None]
        mask = seg_q[a:a + m, None] == seg_k[None, b:b + n]
        if mode != "full":
            mask = mask & (j <= i) & ((j > i - 70) | torch.tensor(mode == "causal", device="cuda"))
        heads = lambda t, r0, r1: t[r0:r1].view(r1 - r0, -1, hd).transpose(0, 1)
        ref = _sdpa_ref(heads(q, a, a + m), heads(k, b, b + n), heads(v, b, b + n), mask).transpose(0, 1).reshape(m, Hq * hd)
        _close(out[a:a + m], ref, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("n,kv,Hq,Hkv,hd", [(8, 500, 16, 8, 128), (12, 500, 16, 8, 128), (12, 3900, 16, 8, 128), (7, 1500, 16, 8, 128), (9, 2100, 8, 8, 64),
                                            (24, 1400, 8, 1, 256), (3, 4100, 4, 1, 256), (40, 333, 40, 2, 128)])
def test_attn_decode_split_plans(dt, n, kv, Hq, Hkv, hd, status):
    """Batches whose splits fit as clusters, as fewer or smaller clusters, and not (second kernel), with ragged and nearly empty sequences: against the
    unsplit kernel at every sequence and against fp32 at three."""
    from rhinoforge_b200.ops import kernels as K_
    lens = [max(1, kv - 37 * (i * i % 29)) if i % 5 else kv for i in range(n - 1)] + [3]
    k_pool, v_pool, pt, ks, vs = _paged(Hkv, hd, lens, dt)
    q = torch.randn(n, Hq * hd, device="cuda").to(dt)
    kw = dict(Hq=Hq, Hkv=Hkv, hd=hd, kv_len=torch.tensor(lens, dtype=torch.int32, device="cuda"), max_kv_len=kv, k_pool=k_pool, v_pool=v_pool, page_table=pt,
              status=status)
    out = K_.attention_decode(q, torch.full_like(q, float("nan")), ws=K_.attn_decode_scratch(n, Hq, hd, "cuda"), **kw)
    whole = K_.attention_decode(q, torch.full_like(q, float("nan")), **kw)
    _close(out, whole.float(), dt)
    for s in (0, n // 2, n - 1):
        ref = _sdpa_ref(q[s].view(Hq, 1, hd), ks[s], vs[s], torch.ones(1, lens[s], dtype=torch.bool, device="cuda"))
        _close(out[s], ref.reshape(Hq * hd), dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H", [64, 1152, 2048])
@pytest.mark.parametrize("pad,off", [(2, 0), (4, 0), (6, 0), (8, 2), (8, 0)])
def test_layernorm_of_rows_off_their_boundary(dt, H, pad, off):
    """Even pitches that are no multiple of eight values, and rows that begin off a 16-byte boundary, below and above the number of rows from which
    a warp takes each (it reads 16 bytes at a time); odd pitches and offsets are refused."""
    from rhinoforge_b200.ops import kernels as K_
    w, b = (1 + 0.1 * torch.randn(H, device="cuda")).to(dt), torch.randn(H, device="cuda").to(dt)
    for rows in (5, 2000):
        x = torch.randn(rows, H + pad, device="cuda").to(dt)[:, off:off + H]
        out = torch.full((rows, H + pad), 7.0, device="cuda").to(dt)
        _close(K_.layernorm(x, w, b, 1e-6, out=out[:, off:off + H]), torch.nn.functional.layer_norm(x.float(), (H,), w.float(), b.float(), 1e-6), dt, scale=2.0)
        assert bool((out[:, off + H:] == 7.0).all()) and bool((out[:, :off] == 7.0).all())
    odd = torch.zeros(4, H + 1, device="cuda", dtype=dt)[:, :H]
    with pytest.raises(Exception, match="even"):
        K_.layernorm(odd, w, b, 1e-6)
    with pytest.raises(Exception, match="even"):
        K_.layernorm(torch.zeros(4, H + 8, device="cuda", dtype=dt)[:, 1:1 + H], w, b, 1e-6)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H", [8, 248, 256, 1000, 4096, 8192, 8200])
def test_rmsnorm_rows_of_any_width(dt, H):
    """A row of at most 8192 values in the registers of its block, and the first width beyond: whole and ragged warps, every form, in place."""
    from rhinoforge_b200.ops import kernels as K_
    x, r = (torch.randn(5, H, device="cuda").to(dt) for _ in range(2))
    w, mod = (1 + 0.1 * torch.randn(H, device="cuda")).to(dt), (0.3 * torch.randn(5, 3 * H, device="cuda")).to(dt)
    norm = lambda t: t.float() * torch.rsqrt(t.float().pow(2).mean(-1, keepdim=True) + 1e-6)
    total = torch.empty_like(x)
    y = K_.rmsnorm(x, w, 1e-6, residual=r, residual_out=total)
    assert torch.equal(total, (x.float() + r.float()).to(dt))
    _close(y, norm(total) * w.float(), dt, scale=2.0)
    _close(K_.rmsnorm(x, w, 1e-6, gemma=True), norm(x) * (1 + w.float()), dt, scale=2.0)
    _close(K_.rmsnorm(x, None, 1e-6, mod=mod), norm(x) * (1 + mod[:, :H].float()) + mod[:, H:2 * H].float(), dt, scale=2.0)
    z = x.clone()
    K_.rmsnorm(z, None, 1e-6, out=z)
    _close(z, norm(x), dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("H,mod", [(1000, False), (2040, False), (1000, True), (2040, True)])
def test_rmsnorm_around_the_line_between_block_and_warp(dt, H, mod):
    """The last number of rows that a block each takes and the first that a warp each does."""
    from rhinoforge_b200.ops import kernels as K_
    per_sm = {(1000, False): 21600, (2040, False): 34000, (1000, True): 24300, (2040, True): 48600}[H, mod]
    line = -(-per_sm * torch.cuda.get_device_properties(0).multi_processor_count // H)
    x, w = torch.randn(line, H, device="cuda").to(dt), (1 + 0.1 * torch.randn(H, device="cuda")).to(dt)
    m = (0.3 * torch.randn(line, 3 * H, device="cuda")).to(dt)
    n = x.float() * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + 1e-6)
    for rows in (line - 1, line):
        if mod:
            _close(K_.rmsnorm(x[:rows], None, 1e-6, mod=m), (n * (1 + m[:, :H].float()) + m[:, H:2 * H].float())[:rows], dt, scale=2.0)
        else:
            _close(K_.rmsnorm(x[:rows], w, 1e-6), (n * w.float())[:rows], dt, scale=2.0)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("M,N,K,extra,dual,cols", [(257, 1032, 72, True, False, 128), (2087, 4104, 72, False, False, 192), (2087, 4104, 72, True, False, 192), (1538, 1288, 1032, False, False, 192),
                                                   (2819, 4104, 72, False, False, 256), (2819, 4104, 1032, True, False, 256), (129, 2048, 2048, False, False, 128), (200, 2056, 1160, True, False, 128),
                                                   (256, 3080, 1160, True, True, 128), (600, 1288, 520, False, True, 128), (300, 2568, 1032, True, True, 128)])
def test_gemm_cta_pairs_of_every_width(dt, M, N, K, extra, dual, cols, status):
    """Tiles of 128, 192 and 256 columns by name, bare and with scale, bias, row scale and residual: 192 columns begin at all four offsets of a 128-row weight block
    and end inside one; GLU pairs; 129 to 256 rows, which have one row tile."""
    import ctypes as C
    from rhinoforge_b200 import _native as N_
    from rhinoforge_b200.ops import kernels as K_
    rows = 2 * N if dual else N
    x = (torch.randn(M, K, device="cuda") * 0.5).to(dt)
    w = (torch.randn(rows, K, device="cuda") / K ** 0.5).to(dt)
    b, sc, rs = torch.randn(rows, device="cuda").to(dt), (torch.rand(rows, device="cuda") + 0.5).to(dt), torch.rand(M, device="cuda") + 0.5
    r, out = torch.randn(M, N, device="cuda").to(dt), torch.full((M + 1, N + 8), 7.0, device="cuda").to(dt)
    wp = K_.pack_weight(w, 2 if dual else 1)
    g = N_.RfGemm()
    g.x, g.w, g.out, g.M, g.N, g.K, g.ldx, g.ldw, g.ldo, g.force_swap, g.w_packed = x.data_ptr(), wp.data_ptr(), out.data_ptr(), M, N, K, K, K, N + 8, -1, 1
    if extra:
        g.bias, g.scale, g.row_scale, g.residual, g.ldr = b.data_ptr(), sc.data_ptr(), rs.data_ptr(), r.data_ptr(), N
    if dual:
        g.dual_offset, g.act = N, 1
    assert N_.lib().rf_gemm_pair_cols(C.byref(g)) == cols
    z = x.float() @ w.float().t()
    if extra:
        z = z * rs[:, None] * sc.float() + b.float()
    ref = torch.nn.functional.silu(z[:, :N]) * z[:, N:] if dual else z
    if extra:
        ref = ref + r.float()
    kw = dict(bias=b, scale=sc, row_scale=rs, residual=r) if extra else {}
    K_.gemm(x, wp, packed_shape=(rows, K), out=out[:M, :N], status=status, **kw, **(dict(act="silu_mul", dual=True) if dual else {}))
    _close(out[:M, :N], ref, dt, scale=2.0 if extra else 1.0)
    assert bool((out[M:] == 7.0).all()) and bool((out[:, N:] == 7.0).all())
