"""Memory-bound sm_100a kernels vs FP32 PyTorch references: norms, embedding, shifted CE,
Philox dropout, gradient norm + AdamW, column sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def close(a, b, tol):
    return (a.float() - b.float()).abs().max().item() <= tol * max(b.float().abs().max().item(), 1e-6) + 1e-6


@pytest.mark.parametrize("rows,cols", [(64, 128), (1000, 768), (4096, 1600)])
def test_layernorm_fwd_bwd(rows, cols):
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    x, res = torch.randn(rows, cols, device=DEV), torch.randn(rows, cols, device=DEV)
    g, b = torch.randn(cols, device=DEV), torch.randn(cols, device=DEV)
    s_out = torch.empty_like(x)
    y, mean, rstd = K.norm_fwd(x, g, b, residual=res, sum_out=s_out, out_dtype=torch.bfloat16)
    xs = x + res
    assert close(y, torch.nn.functional.layer_norm(xs, (cols,), g, b, 1e-5), 1e-2)
    assert close(s_out, xs, 1e-6)
    dy, add = torch.randn(rows, cols, device=DEV).bfloat16(), torch.randn(rows, cols, device=DEV)
    dg, db = torch.zeros(cols, device=DEV), torch.zeros(cols, device=DEV)
    lp = torch.empty(rows, cols, device=DEV, dtype=torch.bfloat16)
    dx = K.norm_bwd(dy, xs, g, mean, rstd, add=add, dx_dtype=torch.float32, dgamma=dg, dbeta=db, dx_lp=lp)
    xs2, g2, b2 = xs.clone().requires_grad_(True), g.clone().requires_grad_(True), b.clone().requires_grad_(True)
    torch.nn.functional.layer_norm(xs2, (cols,), g2, b2, 1e-5).backward(dy.float())
    assert close(dx, xs2.grad + add, 1e-4)
    assert close(lp, xs2.grad + add, 1e-2)
    assert close(dg, g2.grad, 1e-3) and close(db, b2.grad, 1e-3)
    # the same pass can also return the column sums of the BF16 dx (a bias gradient), accumulated like dgamma
    dg2, db2 = torch.zeros(cols, device=DEV), torch.zeros(cols, device=DEV)
    cs = torch.ones(cols, device=DEV)
    lp2 = torch.empty_like(lp)
    dx2 = K.norm_bwd(dy, xs, g, mean, rstd, add=add, dx_dtype=torch.float32, dgamma=dg2, dbeta=db2, dx_lp=lp2,
                     dx_colsum=cs, accumulate_params=True)
    assert torch.equal(dx2, dx) and torch.equal(lp2, lp) and close(dg2, dg, 1e-6)
    assert close(cs, 1.0 + lp.float().sum(0), 1e-4)


@pytest.mark.parametrize("rows,cols", [(1000, 768), (512, 4096)])
def test_rmsnorm_fwd_bwd(rows, cols):
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    x, g = torch.randn(rows, cols, device=DEV), torch.randn(cols, device=DEV)
    y, _, rstd = K.norm_fwd(x, g, None, rms=True, eps=1e-5, out_dtype=torch.float32)
    ref = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * g
    assert close(y, ref, 1e-5)
    dy, dg = torch.randn(rows, cols, device=DEV), torch.zeros(cols, device=DEV)
    dx = K.norm_bwd(dy, x, g, None, rstd, rms=True, dx_dtype=torch.float32, dgamma=dg)
    x2, g2 = x.clone().requires_grad_(True), g.clone().requires_grad_(True)
    (x2 * torch.rsqrt(x2.pow(2).mean(-1, keepdim=True) + 1e-5) * g2).backward(dy)
    assert close(dx, x2.grad, 1e-4) and close(dg, g2.grad, 1e-3)


@pytest.mark.parametrize("deterministic", (True, False))
def test_embedding(deterministic):
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    B, T, C, V = 4, 64, 128, 1000
    tok = torch.randint(0, V, (B, T), device=DEV, dtype=torch.int32)
    wte, wpe = torch.randn(V, C, device=DEV), torch.randn(T, C, device=DEV)
    assert close(K.embedding_pos_fwd(tok, wte, wpe), wte[tok.long()] + wpe[None], 1e-6)
    dx = torch.randn(B, T, C, device=DEV)
    dwte, dwpe = torch.zeros_like(wte), torch.zeros_like(wpe)
    K.embedding_bwd(tok, dx, dwte, dwpe, B, T, deterministic=deterministic)
    ref = torch.zeros_like(wte)
    ref.index_add_(0, tok.reshape(-1).long(), dx.reshape(-1, C))
    assert close(dwte, ref, 1e-5) and close(dwpe, dx.sum(0), 1e-5)


@pytest.mark.parametrize("dtype,ld", [(torch.float32, 1024), (torch.bfloat16, 1024), (torch.float32, 1001)])
def test_cross_entropy_shifted(dtype, ld):
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    B, T, V = 3, 33, 1000
    tok = torch.randint(0, V, (B, T), device=DEV, dtype=torch.int32)
    logits = torch.zeros(B * T, ld, device=DEV, dtype=dtype)
    logits[:, :V] = (torch.randn(B * T, V, device=DEV) * 3).to(dtype)
    ref_in = logits[:, :V].float().clone().requires_grad_(True)
    tg = torch.full((B, T), -100, device=DEV, dtype=torch.long)
    tg[:, :-1] = tok[:, 1:].long()
    sm, z = 0.1, 1e-3
    lse = torch.logsumexp(ref_in, -1)
    valid = tg.reshape(-1) != -100
    nll = lse - ref_in.gather(1, tg.reshape(-1).clamp(min=0)[:, None])[:, 0]
    lossr = ((1 - sm) * nll + sm * (lse - ref_in.mean(-1)) + z * lse * lse)[valid].sum() / valid.sum()
    (lossr * 0.5).backward()
    loss = K.cross_entropy_shifted(logits, tok, vocab=V, smoothing=sm, z_loss=z, grad_scale=0.5)
    bf = dtype == torch.bfloat16
    assert close(loss, lossr.detach().reshape(1), 1e-3 if bf else 1e-5)
    assert close(logits[:, :V], ref_in.grad, 2e-2 if bf else 1e-4)
    assert float(logits[:, V:].float().abs().max()) == 0.0 if ld > V else True


def test_dropout_philox():
    from nexus_b200.ops import _cuda as K
    from nexus_b200.fused.philox import philox_uniform as cpu_uniform
    x = torch.ones(1 << 20, device=DEV)
    y1, y2 = K.dropout(x, 0.25, 1234, 7), K.dropout(x, 0.25, 1234, 7)
    assert torch.equal(y1, y2)
    assert abs((y1 != 0).float().mean().item() - 0.75) < 5e-3
    u = K.philox_uniform(64, 42, 3).cpu()
    assert torch.equal(u, torch.from_numpy(cpu_uniform(64, 42, 3)))


def test_adamw_and_grad_norm():
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    n = 200000
    master, grad = torch.randn(n, device=DEV), torch.randn(n, device=DEV) * 3
    m, v = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV)
    shadow = torch.empty(n, device=DEV, dtype=torch.bfloat16)
    st = K.opt_state_tensor(DEV)
    st.copy_(torch.frombuffer(bytearray(K.pack_opt_state(lr=1e-2, weight_decay=0.1, beta1=0.9, beta2=0.95, eps=1e-8,
                                                         max_grad_norm=1.0, loss_scale=1.0)), dtype=torch.uint8))
    chunks = K.make_chunks([(0, 100000, 1.0, 1.0), (100000, 100000, 0.0, 1.0)], device=DEV)
    p0 = master.clone()
    K.grad_norm(grad, st)
    K.adamw(master, grad, m, v, shadow, chunks, st)
    s = K.unpack_opt_state(bytes(st.cpu().numpy().tobytes()))
    gn = grad.double().norm().item()
    assert abs(s.grad_norm - gn) / gn < 1e-5 and s.step == 1 and s.found_inf == 0
    g = grad * s.clip_coef
    pr = p0.clone()
    pr[:100000] -= 1e-2 * 0.1 * pr[:100000]
    mr, vr = 0.1 * g, 0.05 * g * g
    pr -= 1e-2 * (mr / (1 - 0.9)) / ((vr / (1 - 0.95)).sqrt() + 1e-8)
    assert close(master, pr, 1e-5) and close(shadow, pr, 1e-2)
    # non-finite gradients skip the update
    grad[5] = float("nan")
    before = master.clone()
    K.grad_norm(grad, st)
    K.adamw(master, grad, m, v, shadow, chunks, st)
    s = K.unpack_opt_state(bytes(st.cpu().numpy().tobytes()))
    assert s.found_inf == 1 and s.step == 1 and torch.equal(before, master)


def test_colsum_and_nonfinite():
    from nexus_b200.ops import _cuda as K
    dy = torch.randn(1000, 304, device=DEV).bfloat16()
    assert close(K.colsum(dy), dy.float().sum(0), 1e-4)
    dy = torch.randn(777, 300, device=DEV)
    assert close(K.colsum(dy), dy.sum(0), 1e-5)
    assert K.count_nonfinite(torch.tensor([1.0, float("nan"), float("inf")], device=DEV)).item() == 2


@pytest.mark.parametrize("kind", ["swiglu", "geglu"])
def test_gated_activation_autograd_matches_fp32_formula(kind):
    from nexus_b200.fused import ops as F_
    torch.manual_seed(11)
    h = torch.randn(3, 70, 2 * 96, device="cuda").bfloat16().requires_grad_()
    t = torch.randn(3, 70, 96, device="cuda")
    y = F_.gated_activation(h, kind)
    (y.float() * t).sum().backward()
    h2 = h.detach().float().requires_grad_()
    a, b = h2[..., :96], h2[..., 96:]
    ref = (torch.nn.functional.silu(a) if kind == "swiglu" else torch.nn.functional.gelu(a, approximate="tanh")) * b
    (ref * t).sum().backward()
    assert (y.float() - ref).abs().max() < 2e-2 * ref.abs().max()
    assert (h.grad.float() - h2.grad).abs().max() < 2e-2 * h2.grad.abs().max()


def test_dlpack_exchange_on_the_device_and_pinned_host():
    """The native DLPack producer / consumer on CUDA memory and pinned host memory: zero copy in both directions."""
    from nexus_b200.interop import dlpack
    t = torch.arange(24, dtype=torch.float32, device="cuda").reshape(4, 6)
    assert dlpack.device_type(t) == dlpack.K_CUDA
    u = torch.from_dlpack(dlpack.to_dlpack(t))
    assert u.is_cuda and u.data_ptr() == t.data_ptr()
    v = dlpack.from_dlpack(torch.utils.dlpack.to_dlpack(t))
    v[0, 0] = 5.0
    assert v.is_cuda and v.device == t.device and float(t[0, 0]) == 5.0
    w = dlpack.from_dlpack(dlpack.to_dlpack(t.t()))
    assert tuple(w.shape) == (6, 4) and torch.equal(w, t.t())
    h = torch.ones(8, dtype=torch.float32).pin_memory()
    assert dlpack.device_type(h) == dlpack.K_CUDA_HOST
    g = dlpack.from_dlpack(dlpack.to_dlpack(h))
    g[3] = 2.0
    assert float(h[3]) == 2.0 and not g.is_cuda


@pytest.mark.parametrize("H,Hk,D,rot,T,window,dropout", [(4, 4, 64, 64, 203, 0, 0.0), (6, 2, 128, 96, 130, 50, 0.0), (4, 1, 64, 0, 64, 0, 0.2),
                                                       (2, 2, 64, 16, 1, 0, 0.0)])
def test_packed_qkv_attention_matches_the_separate_operators(H, Hk, D, rot, T, window, dropout):
    """The packed node against apply_rope + attention on views: the same kernels on the same rotated rows (equal outputs), gradients
    that differ only where sums of the zero-padded views were rounded."""
    from nexus_b200.fused import ops as F
    from nexus_b200.lm.rope import apply_rope
    torch.manual_seed(6)
    B, W = 3, (H + 2 * Hk) * D
    qkv = torch.randn(B, T, W, device="cuda").bfloat16().requires_grad_(True)
    ang = torch.rand(T + 5, rot // 2, device="cuda") * 6
    tables = (ang.cos(), ang.sin()) if rot else None
    assert F.qkv_attention_ok(qkv, D, tables)
    kw = dict(window=window, dropout_p=dropout, dropout_seed=3, dropout_offset=8)
    o = F.qkv_attention(qkv, H, Hk, D, tables, **kw)
    do = torch.randn_like(o)
    (got,) = torch.autograd.grad(o, qkv, do)
    q, k, v = (t.view(B, T, -1, D) for t in qkv.split([H * D, Hk * D, Hk * D], -1))
    if rot:
        q, k = (apply_rope(t, *tables) for t in (q, k))
    want = F.attention(q, k, v, **kw)
    assert torch.equal(o, want)
    (ref,) = torch.autograd.grad(want, qkv, do)
    assert (got.float() - ref.float()).norm() <= 1e-2 * ref.float().norm()


def test_packed_qkv_attention_refuses_other_forms():
    from nexus_b200.fused import ops as F
    x = torch.zeros(2, 8, 3 * 128, device="cuda").bfloat16()
    t = torch.zeros(8, 32, device="cuda")
    assert F.qkv_attention_ok(x, 64, (t, t))
    assert not F.qkv_attention_ok(x.float(), 64, (t, t)) and not F.qkv_attention_ok(x, 32, None)
    assert not F.qkv_attention_ok(x[:, ::2], 64, (t, t)) and not F.qkv_attention_ok(x, 64, (t[:7], t[:7]))
    assert not F.qkv_attention_ok(x, 64, (t[:, :12].contiguous(), t[:, :12].contiguous())) and not F.qkv_attention_ok(x, 64, (t.half(), t.half()))


@pytest.mark.parametrize("rows,m,n", [(609, 512, 512), (1, 256, 264), (4097, 768, 768), (64, 8, 16), (3000, 40, 2048)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
def test_weight_grad_any_number_of_rows(rows, m, n, dt):
    """Rows that fill no block of the reduction, sliced and whole.  FP32 sums of exact products: 1e-5 of the norm; BF16 results 2^-8."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(7)
    dy, x = torch.randn(rows, m, device="cuda").bfloat16(), torch.randn(rows, n, device="cuda").bfloat16()
    want = dy.double().t() @ x.double()
    got = K.weight_grad(dy, x, dt)
    assert got.dtype == dt and (got.double() - want).norm() <= (2.0 ** -8 if dt is torch.bfloat16 else 1e-5) * want.norm()
    assert torch.equal(got, K.weight_grad(dy, x, dt))


@pytest.mark.parametrize("n", [1, 7, 8, 4099])
@pytest.mark.parametrize("act", ["gelu", "silu", "relu"])
def test_activation_backward(n, act):
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(8)
    x, dy = (torch.randn(n + 1, device="cuda").bfloat16() for _ in range(2))
    fn = dict(gelu=lambda t: torch.nn.functional.gelu(t, approximate="tanh"), silu=torch.nn.functional.silu, relu=torch.relu)[act]
    for a, b in ((x[:n], dy[:n]), (x[1:], dy[1:])):           # on 16 bytes and beside them
        r = a.double().requires_grad_(True)
        fn(r).backward(b.double())
        assert ((K.act_bwd(a, b, act).double() - r.grad).abs() <= 2.0 ** -8 * r.grad.abs() + 2e-5).all()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_activation_backward_rounds_once(act, dt):
    """FP32 inside: beside the rounding of the result (half a unit in the last place) 2e-6 of the larger of 1 and |x|; tanh to 5e-4
    would show as 1e-4."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(13)
    x = torch.cat([torch.randn(40000, device="cuda") * 2, torch.linspace(-30, 30, 20001, device="cuda"), torch.zeros(1, device="cuda")]).to(dt)
    dy = torch.ones_like(x)
    r = x.double().requires_grad_(True)
    (torch.nn.functional.gelu(r, approximate="tanh") if act == "gelu" else torch.nn.functional.silu(r)).sum().backward()
    half = torch.finfo(dt).eps / 2
    floor = torch.finfo(dt).smallest_normal * torch.finfo(dt).eps
    err = (K.act_bwd(x, dy, act).double() - r.grad).abs()
    assert (err <= half * r.grad.abs() + 2e-6 * x.double().abs().clamp(min=1.0) + floor).all()


@pytest.mark.parametrize("V,ld,dt", [(50, 56, torch.bfloat16), (8192, 8192, torch.bfloat16), (50257, 50304, torch.bfloat16), (101, 101, torch.bfloat16),
                                     (997, 1000, torch.float32), (13, 13, torch.float32)])
@pytest.mark.parametrize("smoothing", [0.0, 0.1])
def test_cross_entropy_gradient_beside_the_logits(V, ld, dt, smoothing):
    """In place and into another matrix give the same bits, the logits stay, entries of -inf get no probability."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(9)
    rows = 6
    logits = (torch.randn(rows, ld, device="cuda") * 3).to(dt)
    if ld % (16 // logits.element_size()) == 0:       # rows of single elements: their kernel's sum of all logits takes finite ones
        logits[:, 0:16:3] = -float("inf")
    targets = torch.tensor([V - 1 if V > 16 else 5, 1, -100, 7, 8, 10], device="cuda", dtype=torch.int32)
    keep, grad, inplace = logits.clone(), torch.empty_like(logits), logits.clone()
    if smoothing:
        keep = logits.nan_to_num(neginf=-30.0)
        logits, inplace = keep.clone(), keep.clone()
    kw = dict(targets=targets, vocab=V, smoothing=smoothing, z_loss=1e-3, seq_len=1)
    a = K.cross_entropy_shifted(logits, None, grad=grad, **kw)
    b = K.cross_entropy_shifted(inplace, None, **kw)
    assert torch.equal(logits, keep) and torch.equal(grad, inplace) and torch.equal(a, b)
    r = keep[:, :V].double().requires_grad_(True)
    lse, ok = r.logsumexp(1), targets >= 0
    nll = lse - r.gather(1, targets.long().clamp(min=0)[:, None])[:, 0]
    per = (1 - smoothing) * nll + (smoothing * (lse - r.mean(1)) if smoothing else 0) + 1e-3 * lse * lse
    want = per[ok].sum() / ok.sum()
    want.backward()
    assert abs(float(a) - float(want)) < 1e-4 * max(1.0, abs(float(want)))
    err = (grad[:, :V].double() - r.grad).abs()
    assert (err <= (2.0 ** -8 if dt is torch.bfloat16 else 1e-5) * r.grad.abs() + 1e-7).all() and (grad[:, V:] == 0).all()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("V", [9000, 8997])
@pytest.mark.parametrize("mask", [-1e9, -1e10, -1e20, -1e30, "lowest"])
def test_cross_entropy_of_masked_vectors(dt, V, mask):
    """Large negative finite logits in whole 16-byte vectors from the first column on: one vector, all vectors of the first thread
    (of 512), all but the target's, none.  Masked entries weigh nothing, as in the 64-bit result: FP32 sums of 9000 terms give 1e-5."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(12)
    mask, ld = torch.finfo(dt).min if mask == "lowest" else mask, 9000
    n = 16 // torch.empty(0, dtype=dt).element_size()
    logits = (torch.randn(4, ld, device="cuda") * 3).to(dt)
    targets = torch.tensor([V - 1, 4500, 4501, 3], device="cuda", dtype=torch.int32)
    logits[0, :n] = mask
    for v in range(0, ld, 512 * n):
        logits[1, v: v + n] = mask
    kept = logits[2, 4501 // n * n: 4501 // n * n + n].clone()
    logits[2] = mask
    logits[2, 4501 // n * n: 4501 // n * n + n] = kept
    for smoothing in (0.0, 0.1) if abs(mask) < 1e30 else (0.0,):      # the mean of all logits is finite
        kw = dict(targets=targets, vocab=V, smoothing=smoothing, z_loss=1e-3, seq_len=1)
        grad, inplace = torch.empty_like(logits), logits.clone()
        a = K.cross_entropy_shifted(logits, None, grad=grad, **kw)
        b = K.cross_entropy_shifted(inplace, None, **kw)
        assert torch.equal(a, b) and torch.equal(grad, inplace)
        r = logits[:, :V].double().requires_grad_(True)
        lse = r.logsumexp(1)
        per = (1 - smoothing) * (lse - r.gather(1, targets.long()[:, None])[:, 0]) + 1e-3 * lse * lse
        want = (per + (smoothing * (lse - r.mean(1)) if smoothing else 0)).mean()
        want.backward()
        assert abs(float(a) - float(want)) <= 1e-5 * max(1.0, abs(float(want)))
        err = (grad[:, :V].double() - r.grad).abs()
        assert (err <= (2.0 ** -8 if dt is torch.bfloat16 else 1e-5) * r.grad.abs() + 1e-7).all()
        if not smoothing:
            assert (grad[:, :V][logits[:, :V] == mask] == 0).all()


def test_loss_gradient_in_batches_and_differentiated():
    """Several gradients of the loss at once, and the derivative of its gradient with respect to the factor in front of it."""
    from nexus_b200.fused import ops
    torch.manual_seed(15)
    logits = torch.randn(6, 40, device="cuda", requires_grad=True)
    targets = torch.arange(6, device="cuda")
    loss = ops.cross_entropy(logits, targets)
    (g,) = torch.autograd.grad(loss, logits, retain_graph=True)
    (many,) = torch.autograd.grad(loss, logits, torch.tensor([1.0, -2.0], device="cuda"), is_grads_batched=True, retain_graph=True)
    assert torch.allclose(many, torch.stack([g, -2 * g]))
    factor = torch.tensor(3.0, device="cuda", requires_grad=True)
    (scaled,) = torch.autograd.grad(loss * factor, logits, create_graph=True)
    (back,) = torch.autograd.grad((scaled * g).sum(), factor)
    assert torch.allclose(scaled, 3 * g) and torch.allclose(back, (g * g).sum())


@pytest.mark.parametrize("rows,pitch,at", [(5, 16, 1), (1, 21, 1), (8, 16, 3)])
def test_linear_weight_gradient_from_any_output_gradient(rows, pitch, at):
    """Gradients that lie beside 16 bytes.  BF16 result of exact products: 2^-8."""
    from nexus_b200.fused import ops
    torch.manual_seed(17)
    x, w = torch.randn(rows, 24, device="cuda").bfloat16(), torch.randn(16, 24, device="cuda").bfloat16().requires_grad_(True)
    dy = torch.randn(rows * pitch + 8, device="cuda").bfloat16()[at:].as_strided((rows, 16), (pitch, 1))
    (dw,) = torch.autograd.grad(ops.fused_linear(x, w), w, dy)
    want = dy.double().t() @ x.double()
    assert ((dw.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


def test_packed_attention_leaves_tables_beside_16_bytes_to_the_general_form():
    from nexus_b200.fused import ops
    qkv = torch.randn(1, 4, 3 * 64, device="cuda").bfloat16()
    flat = torch.randn(4 * 32 + 1, device="cuda")
    on, off = flat[:128].view(4, 32), flat[1:].view(4, 32)
    assert ops.qkv_attention_ok(qkv, 64, (on, on)) and not ops.qkv_attention_ok(qkv, 64, (off, on)) and not ops.qkv_attention_ok(qkv, 64, (on, off))


@pytest.mark.parametrize("rows,cols", [(1, 516), (64, 1600), (3, 1028), (1300, 2048), (5, 4100), (7, 8192), (2, 8196)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("xdt", [torch.float32, torch.bfloat16])
def test_norm_rows_that_a_warp_or_a_block_holds(rows, cols, rms, xdt):
    """Rows of no multiple of 128, on both sides of the widths that a warp's and a block's registers hold, with and without the
    fused sum.  FP32 statistics: results to 2^-8 of values up to about 6 in BF16, 1e-4 in FP32."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(5)
    x, r = (torch.randn(rows, cols, device="cuda").to(xdt) for _ in range(2))
    g, b = torch.randn(cols, device="cuda").to(xdt), torch.randn(cols, device="cuda").to(xdt)
    for res in (None, r):
        s = torch.empty_like(x) if res is not None else None
        y, mean, rstd = K.norm_fwd(x, g, None if rms else b, rms=rms, residual=res, sum_out=s)
        v = (x if res is None else x + r).double()
        if s is not None:
            assert torch.equal(s, x + r)
        mu = 0.0 if rms else v.mean(1, keepdim=True)
        rs = ((v - mu).square().mean(1, keepdim=True) + 1e-5).rsqrt()
        want = (v - mu) * rs * g.double() + (0.0 if rms else b.double())
        assert (y.double() - want).abs().max() < (1e-4 if xdt is torch.float32 else 6e-2)
        # rows too long for a block's registers take the squares of the sum before it is rounded (2^-9 each, averaged over the row)
        assert torch.allclose(rstd.double(), rs[:, 0], rtol=3e-4 if cols > 8192 and res is not None and xdt is torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("rows,cols", [(1, 8), (300, 40), (16384, 3072), (257, 33)])
def test_colsum_lanes(rows, cols):
    """Fewer partials than lanes, more, and the 64 there are at most; FP32 sums of BF16: 1e-5 of the sum of magnitudes."""
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(6)
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    out = torch.ones(cols, device="cuda")
    want = x.double().sum(0)
    assert ((K.colsum(x).double() - want).abs() <= 1e-5 * x.double().abs().sum(0)).all()
    K.colsum(x, out=out, accumulate=True)
    assert ((out.double() - 1 - want).abs() <= 1e-5 * (1 + x.double().abs().sum(0))).all()
