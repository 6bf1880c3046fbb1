import pytest
import torch

pytestmark = pytest.mark.gpu


def test_moe_gpu_forward_backward_matches_reference():
    from nexus_b200.moe import gpu as G
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(0)
    N, d, F, E, k = 300, 128, 256, 8, 2
    cap = 64            # 600 assignments over 8 experts: some overflow and are dropped
    x = (torch.randn(N, d, device="cuda") * 0.5).bfloat16().requires_grad_(True)
    router = (torch.randn(E, d, device="cuda") * 0.2).requires_grad_(True)
    up = (torch.randn(E, 2 * F, d, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    down = (torch.randn(E, d, F, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    y, counts, dropped = G.moe_ffn(x, router, up, down, k, cap)
    dy = torch.randn_like(y)
    y.backward(dy)
    got = [t.grad.float().clone() for t in (x, router, up, down)]
    xr, rr, ur, dr = (t.detach().float().requires_grad_(True) for t in (x, router, up, down))
    yr, idx, gate, keep = G.reference(xr, rr, ur, dr, k, cap)
    yr.backward(dy.float())
    assert int(dropped) == int((~keep).sum()) and int(dropped) > 0
    assert int(counts.sum()) == int(keep.sum())
    assert (y.float() - yr).norm() / yr.norm() < 2e-2
    for g, r, name in zip(got, (xr, rr, ur, dr), ("dx", "drouter", "dup", "ddown")):
        rel = (g - r.grad).norm() / r.grad.norm()
        assert rel < 4e-2, (name, float(rel))
    K.check_status()


def test_moe_routing_kernels_priority_and_ties():
    from nexus_b200.moe import gpu as G
    logits = torch.zeros(10, 4, device="cuda")
    logits[:, 2] = 1.0          # everyone's first choice is expert 2; ties for the second go to expert 0
    expert, gate, slot, counts, dropped = G.route(logits, 2, 8)
    assert expert[:, 0].tolist() == [2] * 10 and expert[:, 1].tolist() == [0] * 10
    assert slot[:, 0].tolist() == [0, 1, 2, 3, 4, 5, 6, 7, -1, -1]
    assert counts.tolist() == [8, 0, 8, 0] and int(dropped) == 4
    assert torch.allclose(gate.sum(-1), torch.ones(10, device="cuda"))


@pytest.mark.parametrize("groups,overflow,noisy", [(2, "drop", False), (1, "reroute", False), (4, "reroute", True)])
def test_moe_gpu_groups_reroute_and_noisy_router_match_the_cpu_core(groups, overflow, noisy):
    """Capacity per token group, the Reroute overflow policy and the noisy top-k router on the GPU (one warp per group
    walks the assignments in (choice, token) order) against the FP32 CPU core `moe.moe_forward` on the same inputs:
    output rows, numbers of dropped and rerouted assignments, and the gradients of the inputs, the router and the noise
    projection."""
    from nexus_b200.moe import gpu as G
    from nexus_b200.moe import moe as M
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(3)
    N, d, E, k, Fd = 128 * max(groups, 2), 64, 8, 2, 64
    spec = M.Spec(experts=E, top_k=k, d_model=d, d_ff=Fd, capacity_factor=0.75, groups=groups, overflow=overflow,
                  noisy=noisy, min_capacity=8)
    cap = M.capacity_of(spec, N // groups)
    assert cap % 8 == 0
    # skewed router: a few experts overflow, so the policy matters
    x = torch.randn(N, d)
    router = torch.randn(E, d) * 0.5
    router[0] *= 3.0
    noise_w = torch.randn(E, d) * 0.3 if noisy else None
    up, down = torch.randn(E, 2 * Fd, d) * 0.1, torch.randn(E, d, Fd) * 0.1
    xb, ub, db = x.bfloat16(), up.bfloat16(), down.bfloat16()
    # CPU core in FP32 on the BF16-rounded operands
    xc = xb.float().requires_grad_(True)
    rc = router.t().contiguous().requires_grad_(True)
    nc = noise_w.t().contiguous().requires_grad_(True) if noisy else None
    yc, r = M.moe_forward(xc, rc, nc, ub.float(), db.float(), spec, training=True, seed=11)
    go = torch.randn(N, d)
    yc.backward(go)
    # GPU
    xg = xb.cuda().requires_grad_(True)
    rg = router.cuda().requires_grad_(True)
    ng = noise_w.cuda().requires_grad_(True) if noisy else None
    out = G.moe_ffn(xg, rg, ub.cuda(), db.cuda(), k, cap, groups=groups, overflow=overflow, noise_w=ng, noise_seed=11,
                    training=True)
    yg, counts, dropped = out[0], out[1], out[2]
    yg.backward(go.cuda().bfloat16())
    torch.cuda.synchronize()
    K.check_status()
    assert int(dropped) == r.dropped
    if len(out) > 3:
        assert int(out[3]) == r.rerouted
        assert int(counts.sum()) == N * k - r.dropped
    if overflow == "reroute":
        assert r.rerouted > 0
    assert (yg.float().cpu() - yc.detach()).abs().max() < 3e-2 * max(1.0, float(yc.detach().abs().max()))
    rel = lambda a, b: float((a - b).norm() / b.norm().clamp_min(1e-6))
    assert rel(xg.grad.float().cpu(), xc.grad) < 4e-2
    assert rel(rg.grad.float().cpu(), rc.grad.t()) < 4e-2
    if noisy:
        assert rel(ng.grad.float().cpu(), nc.grad.t()) < 6e-2


@pytest.mark.parametrize("N,d,E,k,cap,rdt", [(77, 72, 8, 1, 16, "bf16"), (301, 136, 10, 3, 40, "bf16"), (64, 128, 16, 8, 8, "f32"), (513, 264, 64, 2, 24, "bf16")])
def test_moe_router_types_and_odd_sizes(N, d, E, k, cap, rdt):
    """Experts that fill no multiple of eight, every expert over and under its capacity, BF16 and FP32 routers."""
    from nexus_b200.moe import gpu as G
    from nexus_b200.ops import _cuda as K
    torch.manual_seed(N)
    F = 64
    x = torch.randn(N, d, device="cuda").bfloat16().requires_grad_(True)
    router = (torch.randn(E, d, device="cuda") * d ** -0.5).to(torch.bfloat16 if rdt == "bf16" else torch.float32).requires_grad_(True)
    up = (torch.randn(E, 2 * F, d, device="cuda") * d ** -0.5).bfloat16().requires_grad_(True)
    down = (torch.randn(E, d, F, device="cuda") * F ** -0.5).bfloat16().requires_grad_(True)
    y, counts, dropped = G.moe_ffn(x, router, up, down, k, cap)
    dy = torch.randn_like(y)
    got = torch.autograd.grad(y, (x, router, up, down), dy)
    K.check_status()
    xr, rr, ur, dr = (t.detach().double().requires_grad_(True) for t in (x, router, up, down))
    logits = xr @ rr.t()
    val, idx = torch.sort(logits, dim=-1, descending=True, stable=True)
    gate, idx = torch.softmax(val[:, :k], -1), idx[:, :k]
    fill, want, kept = [0] * E, torch.zeros_like(xr), 0
    for j in range(k):
        for t, e in enumerate(idx[:, j].tolist()):
            if fill[e] < cap:
                fill[e] += 1
                kept += 1
                h = ur[e] @ xr[t]
                want = want.index_add(0, torch.tensor([t], device="cuda"),
                                      (gate[t, j] * (dr[e] @ (torch.nn.functional.silu(h[:F]) * h[F:])))[None])
    assert counts.tolist() == fill and int(dropped) == N * k - kept
    ref = (want, *torch.autograd.grad(want, (xr, rr, ur, dr), dy.double()))
    # BF16 activations between the products: 2^-9 each over four roundings, with room for the router's cancelling sums
    for g, r, name in zip((y, *got), ref, ("y", "dx", "drouter", "dup", "ddown")):
        assert (g.double() - r).norm() <= 2e-2 * r.norm(), name


@pytest.mark.parametrize("N,d,E", [(1111, 2048, 64), (200, 1024, 8)])
def test_router_logits_are_fp32_sums(N, d, E):
    """Exact products; d FP32 additions, each rounded to nearest, of partial sums that grow as sqrt(i): about 2.4e-8 sqrt(d / 2) of the
    result where they are added in turn (7.7e-7 at 2048, 5.4e-7 at 1024), less in pieces.  Sums of less than FP32 are beyond that."""
    from nexus_b200.moe import gpu as G
    torch.manual_seed(6)
    x, r = torch.randn(N, d, device="cuda").bfloat16(), (torch.randn(E, d, device="cuda") * d ** -0.5).bfloat16()
    want = x.double() @ r.double().t()
    assert (G.router_logits(x, r).double() - want).norm() <= 2.4e-8 * (d / 2) ** 0.5 * want.norm()


def test_router_delta_pieces_sum_to_the_value():
    """Three BF16 pieces hold an FP32 gradient whole, up to the largest and down to small ones."""
    import ctypes as C
    from nexus_b200.ops import _cuda as K
    big = torch.finfo(torch.float32).max
    torch.manual_seed(14)
    delta = torch.cat([torch.tensor([big, -big, 3.39e38, 1.0, -1.0 / 3.0, 1e-30, 0.0]), torch.randn(249) * 10.0 ** torch.randint(-20, 20, (249,))]).cuda()
    N, E, pitch = delta.numel(), 5, 8
    gate, dgate = torch.ones(N, 2, device="cuda"), torch.stack([delta, -delta], 1).contiguous()      # their inner sum is 0
    expert = torch.tensor([[1, 3]], dtype=torch.int32, device="cuda").repeat(N, 1).contiguous()
    dsel, pieces = torch.empty(N, 2, device="cuda"), torch.empty(N, 3, pitch, device="cuda", dtype=torch.bfloat16)
    K._check(K.lib().nx_moe_router_delta(K._p(gate), K._p(dgate), K._p(expert), K._p(dsel), K._p(pieces), C.c_int(N), C.c_int(2), C.c_int(E),
                                         C.c_int(pitch), K._stream()), "nx_moe_router_delta")
    got = pieces.double().sum(1)
    assert torch.equal(dsel[:, 0], delta) and torch.equal(dsel[:, 1], -delta)
    assert torch.equal(got[:, 1], delta.double()) and torch.equal(got[:, 3], -delta.double()) and (got[:, [0, 2, 4, 5, 6, 7]] == 0).all()
