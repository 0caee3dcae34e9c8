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
