"""Numerics of every sm_100a kernel against a plain PyTorch fp32 statement of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp(min=1e-12)).item()


def _close(a, b, tol=2e-2, name=""):
    """Norm-wise relative error of the whole tensor, and of every row and every column on its own, so that a
    single wrong row, or one wrong column block, fails although it barely moves the overall norm.  Rows and columns
    are measured against their own norm, floored at a tenth of the typical one (near-zero rows of a reference
    carry no relative information)."""
    err = _rel_err(a, b)
    assert err < tol, f"{name}: relative error {err:.4g} (tolerance {tol})"
    a2, b2 = a.float(), b.float()
    if a2.dim() < 2 or a2.numel() == 0:
        return
    a2, b2 = a2.reshape(-1, a2.shape[-1]), b2.reshape(-1, b2.shape[-1])
    for dim, what in ((1, "row"), (0, "column")):
        ref_norm = b2.norm(dim=dim)
        floor = 0.1 * ref_norm.mean().clamp(min=1e-12)
        rel = (a2 - b2).norm(dim=dim) / ref_norm.clamp(min=floor)
        worst = int(rel.argmax())
        assert float(rel[worst]) < 4 * tol, f"{name}: {what} {worst} relative error {float(rel[worst]):.4g} (tolerance {4 * tol})"


@pytest.fixture(scope="module")
def ops():
    from moe_distributed_training_b200.ops import cuda_ops
    return cuda_ops


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


# ------------------------------------------------------------------------------------------ GEMM family
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 256, 128), (300, 520, 200), (1024, 4096, 4096), (77, 136, 4096)])
def test_gemm_nt(ops, M, N, K):
    torch.manual_seed(0)
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    y = ops.mm_nt(x, w)
    _close(y, x.float() @ w.float().t(), name=f"nt {M}x{N}x{K}")
    ops.check_status(DEV)


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (300, 520, 200), (1024, 4096, 1024)])
def test_gemm_nn(ops, M, N, K):
    torch.manual_seed(1)
    x, w = _rand(M, K), _rand(K, N, scale=0.05)
    _close(ops.mm_nn(x, w), x.float() @ w.float(), name=f"nn {M}x{N}x{K}")
    ops.check_status(DEV)


@pytest.mark.parametrize("R,M,N", [(128, 128, 128), (200, 136, 264), (1000, 1024, 4096), (64, 16, 512), (512, 4096, 16)])
def test_gemm_tn(ops, R, M, N):
    torch.manual_seed(2)
    a, b = _rand(R, M), _rand(R, N, scale=0.05)
    _close(ops.mm_tn(a, b), a.float().t() @ b.float(), name=f"tn {R}x{M}x{N}")
    out32 = torch.ones(M, N, device=DEV)
    ops.mm_tn(a, b, out=out32, alpha=0.5, accumulate=True)
    _close(out32, 1.0 + 0.5 * (a.float().t() @ b.float()), name="tn accumulate fp32")
    ops.check_status(DEV)


def test_gemm_lora_segment(ops):
    torch.manual_seed(3)
    M, N, K, r = 300, 512, 1024, 16
    x, w = _rand(M, K), _rand(N, K, scale=0.03)
    t, b = _rand(M, r), _rand(N, r, scale=0.1)
    y = ops.mm_nt(x, w, lora=(t, b))
    _close(y, x.float() @ w.float().t() + t.float() @ b.float().t(), name="nt + lora")
    w2, b2 = _rand(K, N, scale=0.03), _rand(r, N, scale=0.1)
    y2 = ops.mm_nn(x, w2, lora=(t, b2))
    _close(y2, x.float() @ w2.float() + t.float() @ b2.float(), name="nn + lora")
    ops.check_status(DEV)


def _plan(ops, T, k, E, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    logits = torch.randn(T, E, device=DEV, generator=g)
    top = logits.topk(k, dim=-1).indices.int()
    return top, ops.make_plan(top, E)


@pytest.mark.parametrize("T,k,E", [(64, 2, 4), (1000, 2, 8), (5000, 2, 8), (300, 1, 2)])
def test_make_plan(ops, T, k, E):
    from moe_distributed_training_b200.ops import reference
    top, plan = _plan(ops, T, k, E)
    ref = reference.make_plan(top.cpu(), E)
    assert torch.equal(plan.tokens_per_expert.cpu(), ref.tokens_per_expert)
    assert torch.equal(plan.padded_offsets.cpu(), ref.padded_offsets)
    assert torch.equal(plan.dest_row.cpu(), ref.dest_row)
    assert torch.equal(plan.src_slot.cpu(), ref.src_slot)


def test_gather_combine(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(4)
    T, k, E, H = 700, 2, 8, 512
    top, plan = _plan(ops, T, k, E)
    x = _rand(T, H).requires_grad_(True)
    w = torch.rand(T, k, device=DEV).to(torch.bfloat16).requires_grad_(True)
    xg = ops.gather_rows(x, plan)
    n_used = int(plan.padded_offsets[-1])
    ref_xg = reference.gather_rows(x.detach().float(), plan.src_slot, k)
    _close(xg[:n_used], ref_xg[:n_used], 1e-6, "gather")
    y = ops.combine_rows(xg * 1.0, plan, w)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = reference.combine_rows(reference.gather_rows(xr, plan.src_slot, k), plan.dest_row, wr, k)
    _close(y, yr, 1e-2, "combine")
    go = _rand(T, H)
    y.backward(go)
    yr.backward(go.float())
    _close(x.grad, xr.grad, 1e-2, "combine->gather dx")
    _close(w.grad, wr.grad, 2e-2, "combine dweights")


@pytest.mark.parametrize("T,E,H,F,lora", [(600, 4, 256, 512, False), (1500, 8, 1024, 2048, False), (600, 4, 256, 512, True)])
def test_grouped_swiglu_mlp(ops, T, E, H, F, lora):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(5)
    k, r = 2, 16
    top, plan = _plan(ops, T, k, E)
    x = _rand(T, H)
    ws = [(_rand(E, F, H, scale=0.05)).requires_grad_(True) for _ in range(3)]
    lo, lo_ref, lparams = None, None, []
    if lora:
        lo, lo_ref = {}, {}
        for name in ("w1", "w2", "w3"):
            fin, fout = (F, H) if name == "w2" else (H, F)
            A = _rand(E, fin, r, scale=0.05).requires_grad_(True)
            B = _rand(E, r, fout, scale=0.05).requires_grad_(True)
            lparams += [A, B]
            lo[name] = (A, B, 2.0)
    xg = ops.gather_rows(x, plan).detach().requires_grad_(True)
    y = ops.grouped_swiglu_mlp(xg, ws[0], ws[1], ws[2], plan, lo, 0.5)
    # fp32 reference on the same rows
    xr = xg.detach().float().requires_grad_(True)
    wr = [w.detach().float().requires_grad_(True) for w in ws]
    lr_params = []
    if lora:
        lo_ref = {}
        for i, name in enumerate(("w1", "w2", "w3")):
            A, B = lparams[2 * i].detach().float().requires_grad_(True), lparams[2 * i + 1].detach().float().requires_grad_(True)
            lr_params += [A, B]
            lo_ref[name] = (A, B, 2.0)
    yr = reference.grouped_swiglu_mlp(xr, wr[0], wr[1], wr[2], plan.padded_offsets, plan.tokens_per_expert, lo_ref, 0.5)
    n_used = int(plan.padded_offsets[-1])
    valid = (plan.src_slot[:n_used] >= 0)
    _close(y[:n_used][valid], yr[:n_used][valid], 2e-2, "mlp forward")
    go = torch.zeros_like(y)
    go[:n_used][valid] = _rand(int(valid.sum()), H)
    y.backward(go)
    yr.backward(go.float())
    _close(xg.grad[:n_used][valid], xr.grad[:n_used][valid], 3e-2, "mlp dx")
    for i in range(3):
        _close(ws[i].grad, wr[i].grad, 3e-2, f"mlp dw{i + 1}")
    for i, (p, q) in enumerate(zip(lparams, lr_params)):
        _close(p.grad, q.grad, 4e-2, f"mlp lora grad {i}")
    ops.check_status(DEV)


def _under_pair_policy(ops, policy, fn):
    prev = ops.ext.gemm_set_pair_policy(policy)
    try:
        return fn()
    finally:
        ops.ext.gemm_set_pair_policy(prev)


@pytest.mark.parametrize("policy", [2, 5], ids=["pair", "default"])
def test_gemm_pair_kernel_matches_single_cta_kernel(ops, policy):
    """The CTA-pair (cta_group::2) kernel, forced for every 256-wide tile, and the default choice of kernel against
    the 128-row kernel."""
    torch.manual_seed(21)
    cases = []
    for M, N, K in [(300, 520, 200), (1024, 4096, 4096), (77, 264, 4096), (512, 256, 64)]:
        x, w = _rand(M, K), _rand(N, K, scale=0.05)
        cases.append((f"nt {M}x{N}x{K}", lambda x=x, w=w: ops.mm_nt(x, w), x.float() @ w.float().t()))
    x, w = _rand(300, 200), _rand(200, 520, scale=0.05)
    cases.append(("nn", lambda x=x, w=w: ops.mm_nn(x, w), x.float() @ w.float()))
    for R, M, N in [(1000, 1024, 4096), (200, 136, 264)]:
        a, b = _rand(R, M), _rand(R, N, scale=0.05)
        cases.append((f"tn {R}x{M}x{N}", lambda a=a, b=b: ops.mm_tn(a, b), a.float().t() @ b.float()))

        def acc(a=a, b=b):
            out = torch.ones(a.shape[1], b.shape[1], device=DEV)
            ops.mm_tn(a, b, out=out, alpha=0.5, accumulate=True)
            return out
        cases.append((f"tn accumulate {R}x{M}x{N}", acc, 1.0 + 0.5 * (a.float().t() @ b.float())))
    for name, fn, want in cases:
        single = _under_pair_policy(ops, 0, fn)
        pair = _under_pair_policy(ops, policy, fn)
        ops.check_status(DEV)
        _close(pair, want, 2e-2, f"pair kernel {name} vs fp32")
        _close(pair, single, 1e-3, f"pair kernel {name} vs single-CTA kernel")


@pytest.mark.parametrize("policy", [0, 2, 5], ids=["tile128", "pair", "default"])
@pytest.mark.parametrize("M,N,K", [(1, 136, 64), (127, 264, 72), (129, 200, 640), (257, 520, 128), (2305, 328, 192)])
def test_gemm_epilogue_edges(ops, M, N, K, policy):
    """Remainders of the 64-column chunks, 32-row quarters and 2048-row panels of the epilogue: plain, accumulating
    (bf16 and fp32), with a residual, weight gradients, and the SwiGLU form with its gate / up outputs.  fp32 sums of at
    most 640 products, one bf16 rounding (0.4 %) of each result; 2e-2 as for the other products."""
    def run():
        torch.manual_seed(M * 7 + N)
        x, w, u = _rand(M, K), _rand(N, K, scale=0.05), _rand(N, K, scale=0.05)
        res, old = _rand(M, N), _rand(M, N)
        want = x.float() @ w.float().t()
        _close(ops.mm_nt(x, w), want, name="plain")
        _close(ops.mm_nt(x, w, residual=res), want + res.float(), name="residual")
        out = old.clone()
        ops._gemm(0, x, False, w, False, out, M, N, K, accumulate=True, alpha=0.5)
        _close(out, old.float() + 0.5 * want, name="accumulate")
        out = old.float()
        ops._gemm(0, x, False, w, False, out, M, N, K, accumulate=True)
        _close(out, old.float() + want, name="accumulate fp32")
        d = _rand(M, N)
        dw, old_w = torch.empty(N, K, dtype=torch.bfloat16, device=DEV), _rand(N, K)
        ops.mm_tn(d, x, out=dw)
        _close(dw, d.float().t() @ x.float(), name="weight gradient")
        dw = old_w.clone()
        ops.mm_tn(d, x, out=dw, accumulate=True)
        _close(dw, old_w.float() + d.float().t() @ x.float(), name="weight gradient, accumulated")
        h, g, v = (torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3))
        ops._gemm(0, x, False, w, False, h, M, N, K, B2=u, C2=g, C3=v)
        up = x.float() @ u.float().t()
        _close(g, want, name="gate"); _close(v, up, name="up")
        _close(h, torch.nn.functional.silu(want) * up, name="swiglu")
    _under_pair_policy(ops, policy, run)
    ops.check_status(DEV)


@pytest.mark.parametrize("policy", [0, 2, 5], ids=["tile128", "pair", "default"])
@pytest.mark.parametrize("T,E,H,F", [(5, 2, 64, 72), (300, 3, 192, 520), (1500, 4, 512, 1024)])
def test_swiglu_backward_in_the_product(ops, T, E, H, F, policy):
    """dg and du of silu(g) * u from the down projection's input gradient, remainders of the 64-column chunks and empty
    experts included, against fp64 on the same bf16 g, u, dy, w2: one bf16 rounding of each result; rows past the groups
    stay untouched."""
    torch.manual_seed(T)
    top = (torch.arange(T, device=DEV) % max(E - 1, 1)).int()[:, None]
    plan = ops.make_plan(top, E)
    R, used, offs = plan.src_slot.numel(), int(plan.padded_offsets[-1]), plan.padded_offsets.tolist()
    dy = ops.ext.gather_rows(_rand(T, H), plan.src_slot, plan.padded_offsets, E, None, 1)
    g, u, w2 = _rand(R, F, scale=2.0), _rand(R, F), _rand(E, F, H, scale=0.1)
    dg, du = (torch.full((R, F), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    _under_pair_policy(ops, policy, lambda: ops._g(1, dy, False, w2, False, dg, F, H, plan, C2=du, swiglu=(g, u)))
    for e in range(E):
        a, b = offs[e], offs[e + 1]
        if a == b:
            continue
        g64, u64 = g[a:b].double().requires_grad_(True), u[a:b].double().requires_grad_(True)
        dh = dy[a:b].double() @ w2[e].double().t()
        rg, ru = torch.autograd.grad(torch.nn.functional.silu(g64) * u64, (g64, u64), dh)
        _close(dg[a:b], rg, 1e-2, name=f"dg {e}")
        _close(du[a:b], ru, 1e-2, name=f"du {e}")
    assert bool((dg[used:] == 7.0).all()) and bool((du[used:] == 7.0).all())
    ops.check_status(DEV)


@pytest.mark.parametrize("counts", [[1], [0, 31, 32, 33], [255, 0, 256, 257], [513, 64, 95], [2100, 1, 300]])
@pytest.mark.parametrize("H,F", [(72, 136), (264, 1032), (1024, 768)])
def test_transposed_pair_kernel(ops, counts, H, F):
    """Weights as the 256-row operand, rows of every group counted exactly: remainders of the 32-row units, of 256-row tiles
    and 8-tile panels, of feature tiles and of the depth; gate / up with and without its outputs and with adapters, SwiGLU
    backward, K-major and MN-major weights, two depth segments; shared last rounds (2100 rows).  fp32 reference, one bf16
    rounding of each result (2e-2 as for the other products); padding becomes zeros, rows past the groups stay untouched."""
    torch.manual_seed(sum(counts) + F)
    E, r = len(counts), 16
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(sum(counts))].to(DEV).int()
    plan = ops.make_plan(ids[:, None], E)
    R, used, offs = plan.src_slot.numel(), int(plan.padded_offsets[-1]), plan.padded_offsets.tolist()
    real = plan.src_slot[:used] >= 0
    rows = lambda n, scale=1.0: torch.where((plan.src_slot >= 0)[:, None], _rand(R, n, scale=scale), 0.0).to(torch.bfloat16)
    x, dy, t = rows(H), rows(H), rows(2 * r)
    w1, w3, w2 = (_rand(E, F, H, scale=0.1) for _ in range(3))
    b1, b3 = _rand(E, F, 2 * r, scale=0.1), _rand(E, F, 2 * r, scale=0.1)
    a2 = _rand(E, 2 * r, H, scale=0.1)

    def ref(fn):
        out = []
        for e in range(E):
            out.append(fn(slice(offs[e], offs[e + 1]), e))
        return torch.cat(out)
    new = lambda n: torch.full((R, n), 7.0, dtype=torch.bfloat16, device=DEV)
    check = lambda got, want, name: (_close(got[:used][real], want[real], name=name), _zero_pads(got, name))

    def _zero_pads(got, name):
        assert bool((got[:used][~real] == 0).all()) and bool((got[used:] == 7.0).all()), name
    f = lambda v: v.float()
    gate = ref(lambda s, e: f(x[s]) @ f(w1[e]).t())
    up = ref(lambda s, e: f(x[s]) @ f(w3[e]).t())
    prev = ops.ext.gemm_set_pair_policy(6)
    try:
        h, g, u = new(F), new(F), new(F)
        ops._g(1, x, False, w1, False, h, F, H, plan, B2=w3)
        check(h, torch.nn.functional.silu(gate) * up, "gate and up")
        ops._g(1, x, False, w1, False, h, F, H, plan, B2=w3, C2=g, C3=u, A_l=t, B_l=b1, B2_l=b3, b_mn_l=False, K_l=2 * r)
        gl, ul = gate + ref(lambda s, e: f(t[s]) @ f(b1[e]).t()), up + ref(lambda s, e: f(t[s]) @ f(b3[e]).t())
        check(g, gl, "gate"); check(u, ul, "up"); check(h, torch.nn.functional.silu(gl) * ul, "gate and up with adapters")
        y = new(H)
        ops._g(1, h, False, w2, True, y, H, F, plan, A_l=t, B_l=a2, b_mn_l=True, K_l=2 * r, alpha=0.5)
        hf = f(h)
        check(y, 0.5 * ref(lambda s, e: hf[s] @ f(w2[e]) + f(t[s]) @ f(a2[e])), "down")
        dg, du = new(F), new(F)
        ops._g(1, dy, False, w2, False, dg, F, H, plan, C2=du, swiglu=(g, u))
        gf, uf = f(g[:used]).requires_grad_(True), f(u[:used]).requires_grad_(True)
        want = torch.autograd.grad(torch.nn.functional.silu(gf) * uf, (gf, uf), ref(lambda s, e: f(dy[s]) @ f(w2[e]).t()))
        check(dg, want[0], "dg"); check(du, want[1], "du")
        dx = new(H)
        ops._g(1, dg, False, w1, True, dx, H, F, plan, A_l=du, B_l=w3, b_mn_l=True, K_l=F)
        dgf, duf = f(dg), f(du)
        check(dx, ref(lambda s, e: dgf[s] @ f(w1[e]) + duf[s] @ f(w3[e])), "dx")
        m = sum(counts)                                   # dense, no padding: rows of any number
        x2, out, factor = _rand(m, H), torch.full((m + 1, F), 7.0, dtype=torch.bfloat16, device=DEV), torch.tensor(0.25, device=DEV)
        ops._gemm(0, x2, False, w1[0], False, out, m, F, H, alpha_dev=factor)
        _close(out[:m], 0.25 * (f(x2) @ f(w1[0]).t()), name="dense")
        assert bool((out[m:] == 7.0).all())
    finally:
        ops.ext.gemm_set_pair_policy(prev)
    ops.check_status(DEV)


@pytest.mark.parametrize("counts", [[211, 281, 92, 321, 302, 269, 245, 279], [19, 0, 23, 31, 7, 40, 18, 16], [1024, 700, 513, 65]])
def test_transposed_products_have_one_order_of_sums(ops, counts):
    """Deep products of several rounds of tiles, the last one partly filled: results are the same bits in every run, and those of the
    CTA-pair kernel, which adds the depth up in the same order."""
    torch.manual_seed(sum(counts))
    E, H, F, r = len(counts), 2048, 14336, 16
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(sum(counts))].to(DEV).int()
    plan = ops.make_plan(ids[:, None], E)
    R = plan.src_slot.numel()
    rows = lambda n: torch.where((plan.src_slot >= 0)[:, None], _rand(R, n), 0.0).to(torch.bfloat16)
    x, a, t = rows(H), rows(F), rows(2 * r)
    w1, w3, w2, v = _rand(E, F, H, scale=0.1), _rand(E, F, H, scale=0.1), _rand(E, F, H, scale=0.1), _rand(E, H, F, scale=0.1)
    b1, b3 = _rand(E, F, 2 * r, scale=0.1), _rand(E, F, 2 * r, scale=0.1)

    def products():
        h, g, u, y, z, dg, du, dx = (torch.zeros(R, n, dtype=torch.bfloat16, device=DEV) for n in (F, F, F, H, H, F, F, H))
        ops._g(1, x, False, w1, False, h, F, H, plan, B2=w3, C2=g, C3=u, A_l=t, B_l=b1, B2_l=b3, b_mn_l=False, K_l=2 * r)
        ops._g(1, a, False, w2, True, y, H, F, plan)
        ops._g(1, a, False, v, False, z, H, F, plan)
        ops._g(1, x, False, w2, False, dg, F, H, plan, C2=du, swiglu=(g, u))
        ops._g(1, dg, False, w1, True, dx, H, F, plan, A_l=du, B_l=w3, b_mn_l=True, K_l=F)
        return h, g, u, y, z, dg, du, dx
    prev = ops.ext.gemm_set_pair_policy(6)
    try:
        runs = [products() for _ in range(3)]
        ops.ext.gemm_set_pair_policy(2)
        runs.append(products())
    finally:
        ops.ext.gemm_set_pair_policy(prev)
    for name, first, *others in zip(("h", "g", "u", "y", "z", "dg", "du", "dx"), *runs):
        assert all(torch.equal(first, o) for o in others), name
    ops.check_status(DEV)


@pytest.mark.parametrize("M,N", [(129, 12000), (144, 32008), (300, 32000), (576, 4096), (577, 4100), (1300, 4096)])
@pytest.mark.parametrize("K", [264, 4096])
def test_dense_products_of_odd_row_counts(ops, M, N, K):
    """Row counts at which dense products leave 256-row tiles of tokens: both layouts of the weights, with and without an adapter
    segment, against fp32 (one bf16 rounding: 2e-2 as for the other products)."""
    torch.manual_seed(M)
    N = N // 8 * 8
    x, t = _rand(M, K), _rand(M, 16)
    w, wt, b = _rand(N, K, scale=0.1), _rand(K, N, scale=0.1), _rand(N, 16, scale=0.1)
    _close(ops.mm_nt(x, w), x.float() @ w.float().t(), name="nt")
    _close(ops.mm_nn(x, wt), x.float() @ wt.float(), name="nn")
    _close(ops.mm_nt(x, w, lora=(t, b)), x.float() @ w.float().t() + t.float() @ b.float().t(), name="nt, adapter")
    ops.check_status(DEV)


@pytest.mark.parametrize("counts,depth", [([300] * 9, 4096), ([257, 290, 64, 512, 301, 480, 33, 320, 350], 4100),
                                          ([211, 281, 92, 321, 302, 269, 245, 279], 14336)])
def test_transposed_pair_kernel_with_two_accumulators(ops, counts, depth):
    """Depths and numbers of tiles at which tiles of more than 256 rows are taken (tests/host/tile_enumeration.cu has the choice):
    both accumulators equal and not, beside tiles of one, with and without a last round that is shared, K-major and MN-major weights
    and two depth segments.  fp32 reference, 2e-2 as above; padding becomes zeros."""
    torch.manual_seed(depth)
    E, N, r = len(counts), 4096, 16
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(sum(counts))].to(DEV).int()
    plan = ops.make_plan(ids[:, None], E)
    R, used, offs = plan.src_slot.numel(), int(plan.padded_offsets[-1]), plan.padded_offsets.tolist()
    real = plan.src_slot[:used] >= 0
    rows = lambda n: torch.where((plan.src_slot >= 0)[:, None], _rand(R, n), 0.0).to(torch.bfloat16)
    depth = depth // 8 * 8
    x, t, a = rows(depth), rows(2 * r), _rand(E, 2 * r, N, scale=0.1)
    prev = ops.ext.gemm_set_pair_policy(6)
    try:
        for mn in (True, False):
            w = _rand(E, depth, N, scale=0.1) if mn else _rand(E, N, depth, scale=0.1)
            y = torch.full((R, N), 7.0, dtype=torch.bfloat16, device=DEV)
            ops._g(1, x, False, w, mn, y, N, depth, plan, A_l=t, B_l=a, b_mn_l=True, K_l=2 * r)
            want = torch.cat([x[s:e].float() @ (w[g] if mn else w[g].t()).float() + t[s:e].float() @ a[g].float() for g, (s, e) in enumerate(zip(offs[:-1], offs[1:]))])
            _close(y[:used][real], want[real], name=f"mn {mn}")
            assert bool((y[:used][~real] == 0).all()) and bool((y[used:] == 7.0).all())
    finally:
        ops.ext.gemm_set_pair_policy(prev)
    ops.check_status(DEV)


@pytest.mark.parametrize("counts", [[1, 0, 5], [64, 65, 127, 128], [300, 0, 1], [700], [1600, 900]])
@pytest.mark.parametrize("M,N", [(136, 136), (264, 1032), (1024, 520), (2312, 264)])
def test_weight_gradient_kernel(ops, counts, M, N):
    """Weight gradients whose result moves through shared memory by TMA: written and added to, edges of the 32 x 64 pieces, of
    256-wide tiles and of the panels, groups without rows (zeros, or untouched when adding), depths of 0 to 25 k blocks, the
    gradients as a slice of a larger buffer.  fp32 sums, one bf16 rounding of each result."""
    torch.manual_seed(sum(counts) + M)
    E = len(counts)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(sum(counts))].to(DEV).int()
    plan = ops.make_plan(ids[:, None], E)
    R, offs = plan.src_slot.numel(), plan.padded_offsets.tolist()
    rows = lambda n: torch.where((plan.src_slot >= 0)[:, None], _rand(R, n), 0.0).to(torch.bfloat16)
    a, b = rows(M), rows(N)
    want = torch.stack([a[offs[e]:offs[e + 1]].float().t() @ b[offs[e]:offs[e + 1]].float() for e in range(E)])
    old = _rand(E, M, N, scale=4.0)
    prev = ops.ext.gemm_set_pair_policy(6)
    try:
        for add in (False, True):
            room = torch.full((E, M + 8, N + 8), 7.0, dtype=torch.bfloat16, device=DEV)
            out = room[:, :M, :N]
            out.copy_(old if add else torch.full_like(old, float("nan")))
            ops._g(2, a, True, b, True, out, N, 0, plan, alpha=0.5, accumulate=add)
            _close(out, 0.5 * want + (old.float() if add else 0.0), 1e-2, name=f"add {add}")
            for e in range(E):
                if counts[e] == 0:
                    assert torch.equal(out[e], old[e] if add else torch.zeros_like(old[e]))
            assert bool((room[:, M:] == 7.0).all()) and bool((room[:, :, N:] == 7.0).all())
        x, y, f = _rand(sum(counts), M), _rand(sum(counts), N), torch.tensor(0.25, device=DEV)      # dense, any number of rows
        _close(ops.mm_tn(x, y, alpha_dev=f), 0.25 * (x.float().t() @ y.float()), 1e-2, name="dense")
    finally:
        ops.ext.gemm_set_pair_policy(prev)
    ops.check_status(DEV)


@pytest.mark.parametrize("M,N,K", [(1, 4096, 4096), (77, 1024, 4096), (300, 520, 2056), (129, 64, 8192), (1000, 16, 4096), (33, 128, 1024)])
def test_gemm_few_tiles_shared_by_a_cluster(ops, M, N, K):
    """Products with few output tiles under the default policy (the depth is cut over a cluster): K-major and MN-major
    weights, adapter segment with residual, accumulation, fp32 results, a device scalar as factor, weight gradients; twice,
    bit for bit the same.  fp32 sums, one bf16 rounding of each result."""
    torch.manual_seed(K + M)
    x, w, w2 = _rand(M, K), _rand(N, K, scale=0.05), _rand(K, N, scale=0.05)
    t, b, res, old = _rand(M, 16), _rand(N, 16, scale=0.1), _rand(M, N), _rand(M, N)
    want = x.float() @ w.float().t()
    f = torch.tensor(0.25, device=DEV)

    def run():
        acc = old.clone()
        ops._gemm(0, x, False, w, False, acc, M, N, K, accumulate=True, alpha=0.5)
        acc32 = old.float()
        ops._gemm(0, x, False, w2, True, acc32, M, N, K, accumulate=True, alpha_dev=f)
        g = torch.empty(N, K, dtype=torch.bfloat16, device=DEV)
        ops.mm_tn(res, x, out=g)
        narrow = torch.empty(K, 16, dtype=torch.bfloat16, device=DEV)       # depth M
        ops.mm_tn(x, t, out=narrow, alpha_dev=f)
        return [ops.mm_nt(x, w), ops.mm_nt(x, w, lora=(t, b), residual=res), ops.mm_nn(x, w2), acc, acc32, g, narrow]
    got, again = run(), run()
    refs = [want, want + t.float() @ b.float().t() + res.float(), x.float() @ w2.float(), old.float() + 0.5 * want,
            old.float() + 0.25 * (x.float() @ w2.float()), res.float().t() @ x.float(), 0.25 * (x.float().t() @ t.float())]
    for i, (a, r, c) in enumerate(zip(got, refs, again)):
        _close(a, r, name=f"product {i}")
        assert torch.equal(a, c), f"product {i} differs between two runs"
    ops.check_status(DEV)


@pytest.mark.parametrize("T,E,r,F", [(40, 4, 16, 2048), (700, 8, 32, 4096), (3, 2, 8, 1024)])
def test_grouped_adapter_products_shared_by_a_cluster(ops, T, E, r, F):
    """Row-grouped and depth-grouped products with a rank-wide side, some experts without rows, against fp32."""
    torch.manual_seed(T)
    top = (torch.arange(T, device=DEV) % max(E - 1, 1)).int()[:, None]
    plan = ops.make_plan(top, E)
    offs, R = plan.padded_offsets.tolist(), plan.src_slot.numel()
    xg = ops.ext.gather_rows(_rand(T, F), plan.src_slot, plan.padded_offsets, E, None, 1)
    A, B = _rand(E, F, r, scale=0.05), _rand(E, r, F, scale=0.05)
    t, u = (torch.empty(R, r, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops._g(1, xg, False, A, True, t, r, F, plan, alpha=2.0)
    ops._g(1, xg, False, B, False, u, r, F, plan)
    dA, dB = torch.full_like(A, 7.0), torch.full_like(B, 7.0)
    ops._g(2, xg, True, t, True, dA, r, 0, plan)
    ops._g(2, t, True, xg, True, dB, F, 0, plan)
    for e in range(E):
        a, b = offs[e], offs[e + 1]
        if b > a:
            _close(t[a:b], 2.0 * xg[a:b].float() @ A[e].float(), name=f"x A, expert {e}")
            _close(u[a:b], xg[a:b].float() @ B[e].float().t(), name=f"dy B, expert {e}")
        _close(dA[e], xg[a:b].float().t() @ t[a:b].float(), name=f"dA {e}")
        _close(dB[e], t[a:b].float().t() @ xg[a:b].float(), name=f"dB {e}")
    ops.check_status(DEV)


@pytest.mark.parametrize("T,H,E", [(1, 64, 4), (33, 4096, 8), (450, 1032, 8), (97, 256, 16), (70, 512, 40)])
def test_router_backward_odd_sizes(ops, T, H, E):
    """Token pairs of a warp, token chunks and column blocks that do not divide, and frozen weights, against fp64."""
    torch.manual_seed(T + E)
    x, w = _rand(T, H), _rand(E, H, scale=0.05)
    k = 2
    scores, wts, idx = ops.ext.router_fwd(x, w, k, True)
    x64, w64 = x.double().requires_grad_(True), w.double().requires_grad_(True)
    p = (x64 @ w64.t()).softmax(-1)
    sel = p.gather(1, idx.long())
    gw = sel / sel.sum(1, keepdim=True)
    _close(wts, gw, 1e-2, name="weights")
    d = _rand(T, k)
    rx, rw = torch.autograd.grad(gw, (x64, w64), d.double())
    dx, dw = ops.ext.router_bwd(x, w, idx, d, None, True)
    _close(dx, rx, 2e-2, name="dx")
    assert _rel_err(dw, rw) < 1e-3, _rel_err(dw, rw)
    base = _rand(T, H)
    acc = base.clone()
    _, none = ops.ext.router_bwd(x, w, idx, d, None, True, acc, False)
    assert none.numel() == 0
    _close(acc, base.float() + dx.float(), name="dx accumulate")


@pytest.mark.parametrize("T,H,E", [(50, 4104, 8), (3700, 4104, 8), (4001, 6144, 3), (300, 8192, 8)])
def test_router_rows_wider_than_4096_columns(ops, T, H, E):
    """The general kernels, one token per warp and (from 3552 tokens on 148 SMs) two, with the statistics, against fp64."""
    test_router_backward_odd_sizes(ops, T, H, E)
    x, w = _rand(T, H), _rand(E, H, scale=0.05)
    scores, wts, idx, stats = ops.ext.router_fwd(x, w, 2, True, True)
    p = (x.double() @ w.double().t()).softmax(-1)
    _close(scores, p, 1e-2, name="scores")
    assert torch.equal(stats[:E], torch.bincount(idx.reshape(-1).long(), minlength=E).float())
    assert torch.allclose(stats[E:], scores.float().sum(0), rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("T,H,E", [(40, 512, 8), (37, 4104, 8), (29, 256, 20)])
def test_router_with_nan_and_infinite_tokens(ops, T, H, E):
    """A token with a NaN or an infinity gets NaN scores, indices that are experts, and a NaN gradient; the others' scores,
    choices and gradients are what they are without it."""
    torch.manual_seed(H)
    x, w, d = _rand(T, H), _rand(E, H, scale=0.05), _rand(T, 2)
    clean = ops.ext.router_fwd(x, w, 2, True)
    clean_dx = ops.ext.router_bwd(x, w, clean[2], d, None, True, None, False)[0]
    bad = x.clone()
    bad[3, 5], bad[T - 1, H - 1] = float("nan"), float("inf")
    rest = [t for t in range(T) if t not in (3, T - 1)]
    scores, wts, idx = ops.ext.router_fwd(bad, w, 2, True)
    assert bool(scores[[3, T - 1]].isnan().all()) and bool(((idx >= 0) & (idx < E)).all())
    for a, b in zip((scores, wts, idx), clean):
        assert torch.equal(a[rest], b[rest])
    dx = ops.ext.router_bwd(bad, w, idx, d, None, True, None, False)[0]
    assert torch.equal(dx[rest], clean_dx[rest]) and bool(dx[[3, T - 1]].isnan().all())


@pytest.mark.parametrize("rows,cols", [(1, 64), (700, 4096), (301, 2056), (40, 8192), (9, 16384)])
def test_rmsnorm_backward_widths(ops, rows, cols):
    torch.manual_seed(cols)
    x, w, dy, dres = _rand(rows, cols), _rand(cols), _rand(rows, cols), _rand(rows, cols)
    y, rstd = ops.ext.rmsnorm_fwd(x, w, 1e-5)
    x64, w64 = x.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = x64 * (x64.square().mean(1, keepdim=True) + 1e-5).rsqrt() * w64
    rx, rw = torch.autograd.grad(ref, (x64, w64), dy.double())
    dx, part = ops.ext.rmsnorm_bwd(x, w, dy, rstd, dres)
    _close(dx, rx + dres.double(), 1e-2, name="dx")
    _close(ops.ext.rmsnorm_dw(part, w)[None], rw[None], 1e-2, name="dw")
    dx2, part = ops.ext.rmsnorm_bwd(x, w, dy, rstd, dres, False)
    assert part.numel() == 0 and torch.equal(dx, dx2)


@pytest.mark.parametrize("heads,d", [(1, 16), (3, 24), (5, 64), (32, 128), (8, 256)])
def test_rope_head_sizes(ops, heads, d):
    T = 37
    x = _rand(T, heads, d)
    pos = torch.randint(0, 9000, (T,), device=DEV, dtype=torch.int32)
    ang = pos.double()[:, None] * 1e6 ** (-2.0 * torch.arange(d // 2, device=DEV).double() / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x.double().split(d // 2, -1)
    # fp32 angles of up to 9000 rad: 9000 * 2^-24 = 5e-4; bf16 results
    _close(ops.ext.rope(x, pos, 1e6, False).flatten(1), torch.cat([a * c - b * s, b * c + a * s], -1).flatten(1), 1e-2, name="rope")
    _close(ops.ext.rope(ops.ext.rope(x, pos, 1e6, False), pos, 1e6, True).flatten(1), x.float().flatten(1), 1e-2, name="rope and back")


@pytest.mark.parametrize("policy", [2, 5], ids=["pair", "default"])
@pytest.mark.parametrize("T,E,H,F,lora", [(600, 4, 256, 512, True), (1500, 8, 1024, 2048, False), (333, 3, 512, 1024, False)])
def test_grouped_mlp_pair_kernel_matches_single_cta_kernel(ops, T, E, H, F, lora, policy):
    """Row groups with odd and even numbers of 128-row blocks (idle second halves), forward and backward."""
    torch.manual_seed(22)
    k, r = 2, 16
    top, plan = _plan(ops, T, k, E)
    x = _rand(T, H)
    ws = [_rand(E, F, H, scale=0.05) for _ in range(3)]
    lo_t = None
    if lora:
        lo_t = {}
        for name in ("w1", "w2", "w3"):
            fin, fout = (F, H) if name == "w2" else (H, F)
            lo_t[name] = (_rand(E, fin, r, scale=0.05), _rand(E, r, fout, scale=0.05), 2.0)
    n_used = int(plan.padded_offsets[-1])
    valid = (plan.src_slot[:n_used] >= 0)
    go = torch.zeros(plan.capacity, H, device=DEV, dtype=torch.bfloat16)
    go[:n_used][valid] = _rand(int(valid.sum()), H)

    def run():
        w = [t.clone().requires_grad_(True) for t in ws]
        lo = None if lo_t is None else {n: (A.clone().requires_grad_(True), B.clone().requires_grad_(True), sc) for n, (A, B, sc) in lo_t.items()}
        xg = ops.gather_rows(x, plan).detach().requires_grad_(True)
        y = ops.grouped_swiglu_mlp(xg, w[0], w[1], w[2], plan, lo, 0.5)
        y.backward(go[:y.shape[0]])
        outs = [y.detach()[:n_used][valid], xg.grad[:n_used][valid]] + [t.grad for t in w]
        if lo is not None:
            for n in ("w1", "w2", "w3"):
                outs += [lo[n][0].grad, lo[n][1].grad]
        return outs
    single = _under_pair_policy(ops, 0, run)
    pair = _under_pair_policy(ops, policy, run)
    ops.check_status(DEV)
    for i, (a, b) in enumerate(zip(pair, single)):
        _close(a, b, 2e-3, f"grouped mlp output {i}: pair vs single-CTA kernel")


# ------------------------------------------------------------------------------------------ small ops
@pytest.mark.parametrize("M,K,r", [(576, 4096, 16), (77, 1024, 8), (1000, 4096, 32), (5, 264, 12)])
def test_skinny_mm(ops, M, K, r):
    torch.manual_seed(30)
    x, A, B = _rand(M, K), _rand(r, K, scale=0.05), _rand(K, r, scale=0.05)
    _close(ops.ext.skinny_mm(x, A, False, 0.5), 0.5 * (x.float() @ A.float().t()), 1e-2, "skinny x A^T")
    _close(ops.ext.skinny_mm(x, B, True, 2.0), 2.0 * (x.float() @ B.float()), 1e-2, "skinny x B")
    xs = _rand(M, K + 64)[:, :K]          # row stride larger than K
    _close(ops.ext.skinny_mm(xs, A, False, 1.0), xs.float() @ A.float().t(), 1e-2, "skinny strided x")


def test_linear_lora_backward(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(6)
    M, K, N, r = 200, 512, 1024, 16
    x = _rand(M, K).requires_grad_(True)
    w = _rand(N, K, scale=0.05).requires_grad_(True)
    A = _rand(r, K, scale=0.05).requires_grad_(True)
    B = _rand(N, r, scale=0.05).requires_grad_(True)
    y = ops.linear(x, w, (A, B, 2.0))
    ref_in = [t.detach().float().requires_grad_(True) for t in (x, w, A, B)]
    yr = reference.linear(ref_in[0], ref_in[1], (ref_in[2], ref_in[3], 2.0))
    _close(y, yr, 2e-2, "linear+lora fwd")
    go = _rand(M, N)
    y.backward(go); yr.backward(go.float())
    for t, rt, name in zip((x, w, A, B), ref_in, "x w A B".split()):
        _close(t.grad, rt.grad, 3e-2, f"linear+lora d{name}")


def test_rmsnorm(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(7)
    x = _rand(333, 4096).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(4096, device=DEV)).to(torch.bfloat16).requires_grad_(True)
    y = ops.rmsnorm(x, w, 1e-5)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    yr = reference.rmsnorm(xr, wr, 1e-5)
    _close(y, yr, 1e-2, "rmsnorm fwd")
    go = _rand(333, 4096)
    y.backward(go); yr.backward(go.float())
    _close(x.grad, xr.grad, 1e-2, "rmsnorm dx")
    _close(w.grad, wr.grad, 2e-2, "rmsnorm dw")


def test_rope(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(8)
    x = _rand(500, 8, 128).requires_grad_(True)
    pos = torch.arange(500, device=DEV, dtype=torch.int32)
    y = ops.rope(x, pos, 1e6)
    xr = x.detach().float().requires_grad_(True)
    yr = reference.rope(xr, pos, 1e6)
    _close(y, yr, 1e-2, "rope fwd")
    go = _rand(500, 8, 128)
    y.backward(go); yr.backward(go.float())
    _close(x.grad, xr.grad, 1e-2, "rope bwd")


def test_router(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(9)
    T, H, E, k = 777, 1024, 8, 2
    x = _rand(T, H).requires_grad_(True)
    w = _rand(E, H, scale=0.05).requires_grad_(True)
    s, wt, idx = ops.router(x, w, k, True)
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    sr, wtr, idxr = reference.router(xr, wr, k, True)
    assert (idx == idxr).float().mean() > 0.995
    _close(s, sr, 1e-2, "router scores")
    same = (idx == idxr).all(dim=1)
    _close(wt[same], wtr[same], 1e-2, "router weights")
    go = torch.rand(T, k, device=DEV).to(torch.bfloat16)
    go = go * same[:, None]
    wt.backward(go)
    wtr.backward(go.float())
    _close(x.grad, xr.grad, 3e-2, "router dx")
    _close(w.grad, wr.grad, 3e-2, "router dw")


@pytest.mark.parametrize("T,V,H,repeat", [(1, 8, 8, 1), (300, 40, 264, 1), (700, 2048, 4096, 1), (64, 4, 1032, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_gradient_written_and_added(ops, T, V, H, repeat, dtype):
    """Table gradients by lists of equal ids: fp32 sums, one rounding (bf16: 0.4 %; fp32: the order of up to T additions)."""
    torch.manual_seed(T + V)
    ids = torch.randint(0, max(V // repeat, 1), (T,), device=DEV)
    d = _rand(T, H)
    old = _rand(V, H).to(dtype)
    want = torch.zeros(V, H, device=DEV, dtype=torch.float64).index_add_(0, ids, d.double())
    out = torch.full((V, H), float("nan"), device=DEV, dtype=dtype)
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    ops.ext.embedding_bwd(d, ids, out, False)
    _close(out, want, tol, "written")
    out = old.clone()
    ops.ext.embedding_bwd(d, ids, out, True)
    _close(out, old.double() + want, tol, "added")
    untouched = torch.ones(V, dtype=torch.bool, device=DEV)
    untouched[ids] = False
    assert torch.equal(out[untouched], old[untouched])


@pytest.mark.parametrize("T,V,H,hot", [(1, 8, 8, 0.0), (300, 40, 264, 0.0), (700, 2048, 4096, 0.0), (64, 4, 1032, 0.0), (32, 3, 16, 1.0), (33, 3, 2048, 1.0),
                                       (34, 3, 2056, 1.0), (257, 5, 520, 0.3), (2000, 7, 264, 0.0), (8192, 1000, 4096, 0.9)])
def test_embedding_gradient(ops, T, V, H, hot):
    """Table gradients by lists of equal ids, and by sums past the length of a list (32 tokens): fp32 sums, one bf16 rounding (0.4 %)
    of each; rows of other ids are zero.  `hot`: share of the tokens that have one id."""
    torch.manual_seed(T + V)
    ids = torch.randint(0, V, (T,), device=DEV)
    ids[torch.rand(T, device=DEV) < hot] = V // 2
    d = _rand(T, H)
    want = torch.zeros(V, H, device=DEV, dtype=torch.float64).index_add_(0, ids, d.double())
    out = torch.full((V, H), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.ext.embedding_bwd(d, ids, out)
    _close(out, want, 1e-2, "gradient")
    # by elements: half a unit in the last place of bf16, and an fp32 sum of n terms in any order (n 2^-24 times the sum of the sizes)
    bound = want.abs() * 2.0 ** -8 + T * 2.0 ** -23 * torch.zeros_like(want).index_add_(0, ids, d.double().abs()) + 1e-30
    assert bool(((out.double() - want).abs() <= bound).all())
    untouched = torch.ones(V, dtype=torch.bool, device=DEV)
    untouched[ids] = False
    assert not bool(out[untouched].any())
    with pytest.raises(RuntimeError):
        ops.ext.embedding_bwd(_rand(T + 1, H), ids, out)


@pytest.mark.parametrize("recompute", [True, False])
def test_weight_gradients_collected_in_place(recompute):
    """One rank: products write or add the dense weights' gradients in the flat gradient; the same step through ordinary gradient
    tensors, two micro-batches (each of the latter's gradients is rounded once more, 0.4 % each), and again after a backward pass that
    failed in a block."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.ops import fused_blocks
    from moe_distributed_training_b200.train.engine import build_engine
    cfg = MixtralConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                        head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    mbs = list(batches(SyntheticInstructionDataset(cfg.vocab_size, 2, 60, 150), 1))

    def step(place, fail=False):
        eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0, activation_checkpointing=recompute)
        assert eng.runner.recompute == recompute
        groups = [u.trainable_group for u in eng.runner.all_units()]
        for g in groups:
            assert g.collect_in_place
            g.collect_in_place = place
        def run():
            for mb in mbs:
                mb = {k: (v.to(DEV) if torch.is_tensor(v) else v) for k, v in mb.items()}
                out = eng.model(mb["input_ids"], labels=mb["labels"], cu_seqlens=mb["cu_seqlens"], max_seqlen=mb["max_seqlen"])
                out.loss.backward()
                eng.runner.finish_microbatch()
        if fail:
            class Failing:
                def __getattr__(self, name):
                    return getattr(fused_blocks_ext, name)

                def attention_block_bwd(self, *a):
                    raise RuntimeError("refused")
            fused_blocks_ext, fused_blocks.ext = fused_blocks.ext, Failing()
            try:
                with pytest.raises(RuntimeError, match="refused"):
                    run()
            finally:
                fused_blocks.ext = fused_blocks_ext
            for leaf in eng.runner._root_leaves:
                leaf.grad = None
            groups[-1]._collecting = None
            for p in eng.model.parameters():
                p.grad = None
        run()
        return [g.shard.grad.clone() for g in groups], [p.grad.clone() for p in eng.model.parameters() if p.grad is not None]
    flat, every = step(True)
    want, want_every = step(False)
    assert len(every) == len(want_every)
    for a, b in zip(flat + every, want + want_every):
        _close(a, b, 1.5e-2, "gradient")
    if recompute:
        again, _ = step(True, fail=True)
        for a, b in zip(again, flat):
            _close(a, b, 1e-3, "gradient after a failure")


def _small_engine(recompute):
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.train.engine import build_engine
    cfg = MixtralConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                        head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    mbs = [{k: (v.to(DEV) if torch.is_tensor(v) else v) for k, v in mb.items()} for mb in batches(SyntheticInstructionDataset(cfg.vocab_size, 2, 60, 150), 1)]
    eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0, activation_checkpointing=recompute)
    assert eng.runner.recompute == recompute
    return eng, mbs, [u.trainable_group for u in eng.runner.all_units()]


def _forward(eng, mb):
    return eng.model(mb["input_ids"], labels=mb["labels"], cu_seqlens=mb["cu_seqlens"], max_seqlen=mb["max_seqlen"])


def _all_grads(eng, groups):
    return [g.shard.grad.clone() for g in groups] + [p.grad.clone() for p in eng.model.parameters() if p.grad is not None]


@pytest.mark.parametrize("recompute", [True, False])
def test_first_weight_gradients_are_written_in_place(recompute):
    """One rank: products write the dense weights' first gradients in the flat gradient; the same step through ordinary gradient
    tensors, two micro-batches (sums in another order, one bf16 rounding: 0.4 %), and again after a backward pass that failed in a
    block, with the head's gradient written already: nothing of the failed one is left."""
    from moe_distributed_training_b200.ops import fused_blocks

    def step(place, fail=None):
        eng, mbs, groups = _small_engine(recompute)
        for g in groups:
            assert g.collect_in_place
            g.collect_in_place = place

        def run(engine_call):
            for mb in mbs:
                if engine_call:
                    eng.forward_backward(mb, 1.0)
                else:
                    _forward(eng, mb).loss.backward()
                    eng.runner.finish_microbatch()
        if fail is not None:
            class Failing:
                def __getattr__(self, name):
                    return getattr(fused_blocks_ext, name)

                def attention_block_bwd(self, *a):
                    raise RuntimeError("refused")
            fused_blocks_ext, fused_blocks.ext = fused_blocks.ext, Failing()
            try:
                with pytest.raises(RuntimeError, match="refused"):
                    run(fail == "engine")
            finally:
                fused_blocks.ext = fused_blocks_ext
            if fail == "loop":
                eng.runner.zero_grad()
            else:
                eng.optimizer.zero_grad(set_to_none=True)
        run(False)
        return _all_grads(eng, groups)
    flat, want = step(True), step(False)
    assert len(flat) == len(want)
    for a, b in zip(flat, want):
        _close(a, b, 4e-3, "gradient")
    for fail in ("engine", "loop"):
        for a, b in zip(step(True, fail), flat):
            _close(a, b, 1e-3, f"gradient after a failure ({fail})")


@pytest.mark.parametrize("recompute", [True, False])
@pytest.mark.parametrize("second", [False, True])
def test_partial_backward_passes_leave_weight_gradients_alone(recompute, second):
    """A backward pass that is asked for something else, before the one for the weights, does not count towards them, whether there is
    a flat gradient already or not; and a weight's gradient that is asked for by itself stays what it was."""
    grads = []
    for partial in (False, True):
        eng, mbs, groups = _small_engine(recompute)
        if second:
            _forward(eng, mbs[1]).loss.backward()
            eng.runner.finish_microbatch()
        out = _forward(eng, mbs[0])
        if partial:
            (dh,) = torch.autograd.grad(out.loss, out.hidden_states, retain_graph=True)
            assert bool(dh.any())
            head = eng.model.lm_head.weight
            (dw,) = torch.autograd.grad(out.loss, head, retain_graph=True)
            kept = dw.clone()
        out.loss.backward()
        eng.runner.finish_microbatch()
        if partial:
            assert head.grad is None and torch.equal(dw, kept)
            if not second:
                place = groups[-1].specs[[m is eng.model.lm_head for m, *_ in groups[-1].specs].index(True)]
                _close(groups[-1].shard.grad[place[4]:place[4] + place[3]].view(place[2]), kept, 4e-3, "lm_head")
        grads.append(_all_grads(eng, groups))
    assert len(grads[0]) == len(grads[1])
    for a, b in zip(*grads):
        _close(a, b, 4e-3, "gradient")


@pytest.mark.parametrize("recompute", [True, False])
def test_gradients_of_dense_weights_pass_through_autograd(recompute):
    """On one rank too: hooks on a weight see its gradient and may change it, and .grad holds the micro-batch's gradient until the
    micro-batch is finished; the flat gradient is the buffer that the products wrote to where nobody else has a part of it."""
    eng, mbs, groups = _small_engine(recompute)
    _forward(eng, mbs[0]).loss.backward()
    root = [eng.model.lm_head.weight, eng.model.model.embed_tokens.weight]
    kept = [] if recompute else [getattr(layer.self_attn, n).weight for layer in eng.model.model.layers for n in ("q_proj", "k_proj", "v_proj", "o_proj")]
    assert all(w.grad is not None and bool(w.grad.any()) for w in root + kept)
    pointer = root[0].grad.data_ptr()
    eng.runner.finish_microbatch()
    flat = groups[-1].shard.grad
    assert flat.data_ptr() <= pointer < flat.data_ptr() + flat.numel() * flat.element_size()          # (no copy)
    want = _all_grads(eng, groups)
    eng, mbs, groups = _small_engine(recompute)
    with torch.no_grad():
        _forward(eng, mbs[0])                        # (the weights' views exist from here on)
    seen = []
    hooked = [eng.model.lm_head.weight, eng.model.model.embed_tokens.weight, eng.model.model.layers[0].self_attn.q_proj.weight]
    for w in hooked:
        w.register_hook(lambda g: (seen.append(g), 2 * g)[1])
    _forward(eng, mbs[0]).loss.backward()
    eng.runner.finish_microbatch()
    assert len(seen) == 3
    got = _all_grads(eng, groups)
    for unit, g in enumerate(groups):
        for i, (mod, name, shape, n, o) in enumerate(g.specs):
            factor = 2.0 if any(getattr(mod, name) is w for w in hooked) else 1.0
            _close(got[unit][o:o + n], factor * want[unit][o:o + n].float(), 4e-3, g.qualnames[i])


@pytest.mark.parametrize("recompute", [True, False])
def test_gradients_that_somebody_keeps_stay_what_they_were(recompute):
    """What a hook or a reader of .grad has kept of the first micro-batch is not changed by the second one."""
    eng, mbs, groups = _small_engine(recompute)
    with torch.no_grad():
        _forward(eng, mbs[0])                        # (the weights' views exist from here on)
    kept = []
    q = eng.model.model.layers[0].self_attn.q_proj.weight
    handle = q.register_hook(lambda g: kept.append(g))
    _forward(eng, mbs[0]).loss.backward()
    kept += [eng.model.lm_head.weight.grad, eng.model.model.embed_tokens.weight.grad.detach()]
    handle.remove()
    want = [t.clone() for t in kept]
    eng.runner.finish_microbatch()
    first = _all_grads(eng, groups)
    _forward(eng, mbs[1]).loss.backward()
    eng.runner.finish_microbatch()
    assert len(kept) == 3 and all(torch.equal(a, b) for a, b in zip(kept, want))
    assert not all(torch.equal(a, b) for a, b in zip(first, _all_grads(eng, groups)))


def test_adapter_blocks_store_gate_and_up_only_for_a_graph(ops, monkeypatch):
    """Passes without a graph (evaluation, the first pass of recomputed blocks) leave the inputs of SwiGLU unwritten, trainable adapters or not."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.train.engine import build_engine
    cfg = MixtralConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                        head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0, use_lora="all")
    (mb,) = list(batches(SyntheticInstructionDataset(cfg.vocab_size, 1, 60, 150), 1))
    stored, real = [], ops._gemm

    def spy(*a, **kw):
        if kw.get("B2") is not None:
            stored.append(kw.get("C2") is not None)
        return real(*a, **kw)
    monkeypatch.setattr(ops, "_gemm", spy)
    before = eng.eval_loss(mb)
    assert stored == [False, False]
    stored.clear()
    loss = eng.forward_backward(mb, 1.0)
    assert stored == [False, False, True, True]
    _close(before, loss, 1e-5, "loss")
    assert all(bool(p.grad.any()) for n, p in eng.model.named_parameters() if "lora_B" in n and p.grad is not None)
    ops.check_status(DEV)


@pytest.mark.parametrize("lora", ["none", "attn-only", "all"])
@pytest.mark.parametrize("keep", [True, False])
def test_two_micro_batches_before_their_backward_pass(lora, keep):
    """Recomputed blocks keep routing and expert results of their own first pass, also where another batch has gone through the
    layer since: the gradient of a sum of two losses is the sum of the two gradients (bf16 gradients, rounded twice)."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.train.engine import build_engine
    cfg = MixtralConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                        head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    mbs = list(batches(SyntheticInstructionDataset(cfg.vocab_size, 2, 60, 150), 1))

    def grads(together):
        eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0, use_lora=lora)
        torch.manual_seed(5)
        for n, p in eng.model.named_parameters():
            if "lora_B" in n:
                p.data.normal_(0.0, 0.05)
        eng.runner.stash_exchange = keep
        losses = []
        for mb in mbs:
            mb = {k: (v.to(DEV) if torch.is_tensor(v) else v) for k, v in mb.items()}
            loss = eng.model(mb["input_ids"], labels=mb["labels"], cu_seqlens=mb["cu_seqlens"], max_seqlen=mb["max_seqlen"]).loss
            if not together:
                loss.backward()
                eng.runner.finish_microbatch()
            losses.append(loss)
        if together:
            sum(losses).backward()
            eng.runner.finish_microbatch()
        return [p.grad for p in eng.model.parameters() if p.grad is not None]
    apart, together = grads(False), grads(True)
    assert len(apart) == len(together) > 0
    for a, b in zip(apart, together):
        _close(a.reshape(-1), b.reshape(-1), 1.5e-2, "gradient")


def test_recomputed_adapter_blocks_keep_results_only_where_there_is_room(ops, monkeypatch):
    """A step that fits in memory without what blocks with expert adapters keep for their recomputation fits with it: nothing is kept
    where an eighth of the GPU, or 24 times what a block keeps, is not free beside it.  Gradients are the same either way."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.ops import fused_blocks
    from moe_distributed_training_b200.train.engine import build_engine
    real = fused_blocks.ext
    free, total = real.memory_room(0)
    big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
    after, same = real.memory_room(0)
    assert free - after >= big.numel() and total == same == torch.cuda.get_device_properties(0).total_memory
    room = [0, 0]

    class Ext:
        def __getattr__(self, name):
            return getattr(real, name)

        def memory_room(self, device):
            return room
    monkeypatch.setattr(fused_blocks, "ext", Ext())
    small = torch.empty(1000, dtype=torch.bfloat16, device=DEV)
    for room[:], fits in (((48000, 80000), True), ((47999, 80000), False), ((48000, 384000), True), ((48000, 384008), False), ((10**11, 18 * 10**10), True)):
        assert fused_blocks._room_to_keep((small, None)) == fits, room
    room[:] = (120, 800)
    assert not fused_blocks._room_to_keep((None, small))
    cfg = MixtralConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, num_key_value_heads=1,
                        head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    (mb,) = list(batches(SyntheticInstructionDataset(cfg.vocab_size, 1, 60, 150), 1))
    grads, plans = [], []
    make_plan = ops.make_plan
    monkeypatch.setattr(ops, "make_plan", lambda *a, **kw: (plans.append(1), make_plan(*a, **kw))[1])
    for room[:], times in (((10**11, 18 * 10**10), 1), ((10**9, 18 * 10**10), 2)):
        eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0, use_lora="all")
        for n, p in eng.model.named_parameters():
            if "lora_B" in n:
                p.data.fill_(0.01)
        plans.clear()
        eng.forward_backward(mb, 1.0)
        assert len(plans) == times * cfg.num_hidden_layers          # (routed again where nothing was kept)
        grads.append([p.grad for p in eng.model.parameters() if p.grad is not None])
    assert len(grads[0]) == len(grads[1]) > 0
    for a, b in zip(*grads):
        _close(a, b, 4e-3, "gradient")
    ops.check_status(DEV)


def test_blocks_keep_nothing_under_an_allocator_without_statistics(ops, monkeypatch):
    from moe_distributed_training_b200.ops import fused_blocks

    class Ext:
        def memory_room(self, device):
            raise RuntimeError("the allocator does not support getDeviceStats")
    monkeypatch.setattr(fused_blocks, "ext", Ext())
    assert not fused_blocks._room_to_keep((torch.empty(8, device=DEV),))


@pytest.mark.parametrize("E,H,F,r", [(1, 8, 8, 4), (3, 72, 200, 12), (8, 256, 1032, 16), (2, 64, 136, 100)])
def test_adapter_pack(ops, E, H, F, r):
    A1, A3, B1, B3 = _rand(E, H, r), _rand(E, H, r), _rand(E, r, F), _rand(E, r, F)
    a13, b1, b3 = ops.ext.adapter_pack(A1, A3, 1.5, 2.0, B1, B3)
    z = torch.zeros_like(B1.transpose(1, 2))
    assert torch.equal(a13, torch.cat([A1 * 1.5, A3 * 2.0], dim=2))
    assert torch.equal(b1, torch.cat([B1.transpose(1, 2), z], dim=2)) and torch.equal(b3, torch.cat([z, B3.transpose(1, 2)], dim=2))
    with pytest.raises(RuntimeError):
        ops.ext.adapter_pack(A1[:, :, :3], A3[:, :, :3], 1.0, 1.0, B1[:, :3], B3[:, :3])


def test_embedding_and_cross_entropy(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(10)
    T, H, V = 300, 256, 2048
    table = _rand(V, H).requires_grad_(True)
    ids = torch.randint(0, V, (T,), device=DEV)
    e = ops.embedding(ids, table)
    assert torch.equal(e, table.detach()[ids])
    e.backward(torch.ones_like(e))
    ref = torch.zeros(V, H, device=DEV)
    ref.index_add_(0, ids, torch.ones(T, H, device=DEV))
    _close(table.grad, ref, 1e-3, "embedding bwd")
    hidden = _rand(T, H).requires_grad_(True)
    head = _rand(V, H, scale=0.05).requires_grad_(True)
    labels = torch.randint(0, V, (T,), device=DEV)
    labels[: T // 3] = -100
    ls, n = ops.cross_entropy_sum(hidden, head, labels)
    loss = ls / n
    hr, wr = hidden.detach().float().requires_grad_(True), head.detach().float().requires_grad_(True)
    lsr, nr = reference.cross_entropy_sum(hr, wr, labels)
    lossr = lsr / nr
    assert abs(loss.item() - lossr.item()) < 2e-2 * abs(lossr.item())
    assert int(n.item()) == int(nr.item())
    (loss * 3.0).backward(); (lossr * 3.0).backward()
    _close(hidden.grad, hr.grad, 3e-2, "ce dhidden")
    _close(head.grad, wr.grad, 3e-2, "ce dhead")


def test_adamw(ops):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(11)
    shapes = [(1000,), (257, 33), (4096, 512)]
    ps = [_rand(*s) for s in shapes]
    gs = [_rand(*s, scale=0.1) for s in shapes]
    ms = [torch.zeros_like(p) for p in ps]
    vs = [torch.zeros_like(p) for p in ps]
    ref = [[t.clone().float() for t in group] for group in (ps, gs, ms, vs)]
    for step in (1, 2, 3):
        ops.adamw_multi(ps, gs, ms, vs, 1e-2, 0.9, 0.999, 1e-8, 0.01, step, 0.5)
        for p, g, m, v in zip(*ref):
            reference.adamw_step(p, g, m, v, 1e-2, 0.9, 0.999, 1e-8, 0.01, step, 0.5)
    for p, pr in zip(ps, ref[0]):
        _close(p, pr, 1e-2, "adamw param")


def test_adamw_tails_and_fp32_states(ops):
    """Sizes that are not multiples of 8, misaligned views and fp32 moments take the element-wise path."""
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(12)
    base = _rand(8 * 1024 + 13)
    edge = base.clone()
    ps = [base[3:8 * 1024 + 5], _rand(100003), _rand(77)]
    gs = [_rand(p.numel(), scale=0.1) for p in ps]
    ms = [torch.zeros(p.numel(), device=DEV, dtype=torch.float32 if i == 1 else torch.bfloat16) for i, p in enumerate(ps)]
    vs = [torch.zeros_like(m) for m in ms]
    ref = [[t.clone().float() for t in group] for group in (ps, gs, ms, vs)]
    for step in (1, 2):
        ops.adamw_multi(ps, gs, ms, vs, 1e-2, 0.9, 0.999, 1e-8, 0.01, step, 1.0)
        for p, g, m, v in zip(*ref):
            reference.adamw_step(p, g, m, v, 1e-2, 0.9, 0.999, 1e-8, 0.01, step, 1.0)
    for p, pr in zip(ps, ref[0]):
        _close(p, pr, 1e-2, "adamw param (tail)")
    assert torch.equal(base[:3], edge[:3]) and torch.equal(base[8 * 1024 + 5:], edge[8 * 1024 + 5:])  # neighbours untouched


def test_sumsq_and_axpby(ops):
    torch.manual_seed(13)
    for n, dt in ((100003, torch.bfloat16), (8 * 4096, torch.bfloat16), (50001, torch.float32)):
        x = torch.randn(n, device=DEV, dtype=dt)
        out = torch.zeros(1, device=DEV, dtype=torch.float32)
        ops.ext.sumsq(x, out)
        ref = x.double().pow(2).sum().item()
        assert abs(out.item() - ref) <= 1e-3 * ref, (n, dt, out.item(), ref)
    y, x = _rand(100003), _rand(100003)
    want = (0.5 * y.float() + 2.0 * x.float())
    ops.ext.axpby(y, x, 0.5, 2.0)
    _close(y, want, 1e-2, "axpby")


def test_end_to_end_matches_reference_path(ops):
    """One training step of a small bf16 model: CUDA kernels vs the PyTorch statement of every op."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.data.synthetic import SyntheticInstructionDataset, batches
    from moe_distributed_training_b200.train.engine import build_engine
    cfg = MixtralConfig(vocab_size=1024, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                        num_attention_heads=2, num_key_value_heads=1, head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    ds = SyntheticInstructionDataset(cfg.vocab_size, 2, 100, 200)
    mbs = list(batches(ds, 1))
    eng = build_engine(cfg, dtype=torch.bfloat16, device_type="cuda", learning_rate=1e-3, seed=0)
    l_gpu = [float(eng.train_step(mbs)["loss"]) for _ in range(3)]
    ref = build_engine(cfg, dtype=torch.float32, device_type="cpu", learning_rate=1e-3, seed=0)
    l_ref = [float(ref.train_step(mbs)["loss"]) for _ in range(3)]
    ops.check_status(DEV)
    for a, b in zip(l_gpu, l_ref):
        assert abs(a - b) < 0.05 * abs(b), (l_gpu, l_ref)
    assert l_gpu[-1] < l_gpu[0]


@pytest.mark.parametrize("T,Hq,Hkv", [(2, 1, 1), (77, 2, 2), (128, 4, 1), (300, 4, 2), (613, 8, 2)])
def test_attention_backward_rounds_ds_with_its_scale(ops, T, Hq, Hkv):
    """dQ and dK against the same sums in fp64 with dS = P (dP - delta) scale rounded to bf16 once, as the operand of their products.  The
    kernel's own errors (fp32 sums, 1e-6) move 1 in 2000 of these roundings and as many of the result's, 1e-4 of the 2-norm together; dS rounded
    without the factor, which is no power of two, is 2.4e-3 away: 1e-3 lies between."""
    torch.manual_seed(T)
    q, k, v, do = (_rand(T, h, 128) for h in (Hq, Hkv, Hkv, Hq))
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    o = ops.attention(*leaves, torch.tensor([0, T], dtype=torch.int32, device=DEV), T)
    dq, dk, dv = torch.autograd.grad(o, leaves, do)
    scale = 128 ** -0.5
    groups = Hq // Hkv
    Q, K, V, dO, O = (t.detach().double().transpose(0, 1) for t in (q, k.repeat_interleave(groups, 1), v.repeat_interleave(groups, 1), do, o))
    S = Q @ K.transpose(1, 2) * scale
    P = torch.softmax(S.masked_fill(torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1), float("-inf")), -1)
    dS = (P * (dO @ V.transpose(1, 2) - (dO * O).sum(-1, keepdim=True)) * scale).bfloat16().double()
    per_kv = lambda t: t.view(Hkv, groups, T, 128).sum(1).transpose(0, 1)
    for name, got, want in (("dq", dq, (dS @ K).transpose(0, 1)), ("dk", dk, per_kv(dS.transpose(1, 2) @ Q)),
                            ("dv", dv, per_kv(P.bfloat16().double().transpose(1, 2) @ dO))):
        want = want.bfloat16().double()
        off, norm = float((got.double() - want).norm()), float(want.norm())
        assert off <= 1e-3 * norm + 1e-6, (name, off, norm)
    ops.check_status(DEV)


@pytest.mark.parametrize("lens", [[128], [200], [577], [1024], [100, 300, 77], [256, 256]])
def test_attention(ops, lens):
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(12)
    T, Hq, Hkv, d = sum(lens), 8, 2, 128
    q, k, v = (_rand(T, h, d).requires_grad_(True) for h in (Hq, Hkv, Hkv))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    o = ops.attention(q, k, v, cu, max(lens))
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    orf = reference.attention(qr, kr, vr, cu)
    _close(o, orf, 2e-2, f"attention fwd {lens}")
    go = _rand(T, Hq, d)
    o.backward(go); orf.backward(go.float())
    _close(q.grad, qr.grad, 3e-2, "attention dq")
    _close(k.grad, kr.grad, 3e-2, "attention dk")
    _close(v.grad, vr.grad, 3e-2, "attention dv")
    ops.check_status(DEV)


def test_attention_node_in_the_graph(ops):
    """The node is part of autograd as any other: hooks on what it saves, inputs of other layouts, a frozen input, no graph without
    gradients; transforms that it has no rule for refuse it."""
    from moe_distributed_training_b200 import ops as front
    torch.manual_seed(3)
    q, k, v, do = (_rand(96, h, 128) for h in (4, 2, 2, 4))
    cu = torch.tensor([0, 40, 96], device=DEV)                    # (any integer type)
    want = None
    for layout in ("plain", "strided", "hooks"):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        ins = [t.transpose(0, 1).contiguous().transpose(0, 1) if layout == "strided" else t for t in leaves]
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(1), t.cpu())[1], lambda t: t.to(DEV)) if layout == "hooks" else torch.enable_grad():
            o = front.attention(*ins, cu, 56)
        assert o.requires_grad and (layout != "hooks" or len(packed) >= 5)
        got = [o.detach()] + list(torch.autograd.grad(o, leaves, do))
        want = want or got
        for a, b in zip(got, want):
            _close(a, b, 2e-3, layout)                            # (the same kernels; one bf16 rounding)
    kf = k.clone().requires_grad_(True)
    (front.attention(q, kf, v, cu, 56) * do).sum().backward()
    _close(kf.grad, want[2], 2e-3, "only k")
    with torch.no_grad():
        assert not front.attention(q, kf, v, cu, 56).requires_grad
    with pytest.raises(Exception):
        torch.func.vmap(lambda a: front.attention(a, k, v, cu, 56))(torch.stack([q, q]))
    with pytest.raises(Exception):
        torch.func.jvp(lambda a: front.attention(a, k, v, cu, 56), (q,), (q,))
    ops.check_status(DEV)


@pytest.mark.parametrize("lens,heads,kv", [([1], 2, 2), ([127, 1, 129], 4, 2), ([255, 257, 128], 6, 2), ([640, 33, 1100, 5], 8, 2),
                                           ([130] * 40, 4, 4), ([2500, 1300], 32, 8), ([3000], 4, 1)])
def test_attention_ragged_blocks_and_head_sets(ops, lens, heads, kv):
    """Edges of the 128-row blocks, sequences of one row, more sequences than a warp has lanes, and both ways of adding a
    kv head's query heads up (in one CTA, over partial sums), against fp64 attention.  bf16 inputs, probabilities and dS
    rounded to bf16 before the second products: 1e-2 on whole tensors is about three times what is seen."""
    T, d = sum(lens), 128
    g = torch.Generator(device=DEV).manual_seed(T + heads)
    q, k, v, do = (torch.randn(T, h, d, device=DEV, generator=g).to(torch.bfloat16) for h in (heads, kv, kv, heads))
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    for t in (q, k, v):
        t.requires_grad_(True)
    from moe_distributed_training_b200.ops.attention_cuda import attention
    o = attention(q, k, v, cu, max(lens))
    grads = torch.autograd.grad(o, (q, k, v), do)
    q2, k2, v2 = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    outs = []
    for s, n in zip(cu.tolist(), lens):
        qs, ks, vs = (t[s:s + n].transpose(0, 1) for t in (q2, k2.repeat_interleave(heads // kv, 1), v2.repeat_interleave(heads // kv, 1)))
        sc = (qs @ ks.transpose(1, 2)) * d ** -0.5
        sc = sc.masked_fill(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
        outs.append((sc.softmax(-1) @ vs).transpose(0, 1))
    ref = torch.cat(outs)
    for name, a, b in zip(("o", "dq", "dk", "dv"), (o,) + grads, (ref,) + torch.autograd.grad(ref, (q2, k2, v2), do.double())):
        if float(b.norm()) == 0.0:            # one key: the softmax is constant
            assert float(a.float().abs().max()) < 1e-2, name
        else:
            assert _rel_err(a, b) < 1e-2, (name, _rel_err(a, b))
    ops.check_status(DEV)


@pytest.mark.parametrize("lens,heads,kv", [([8] * 200, 8, 2), ([1, 3, 0, 127, 2] * 30, 4, 2), ([64, 200] * 10, 4, 4),
                                           ([5] * 31, 4, 2), ([150] * 32, 4, 2), ([9] * 33, 2, 1), ([0] * 40 + [300, 0, 20], 4, 2), ([130, 0] * 33, 2, 2)])
def test_attention_many_short_sequences(ops, lens, heads, kv):
    """Blocks with few rows: their dQ tiles take just those rows, and neighbours must not touch.  Blocks are looked up 32
    sequences at a time: one window less one, one, one more, and windows of empty sequences."""
    test_attention_ragged_blocks_and_head_sets(ops, lens, heads, kv)


@pytest.mark.parametrize("lens,heads,kv", [([128], 12, 2), ([257], 16, 1), ([129, 2, 640], 16, 1), ([384, 1], 8, 1), ([300], 6, 2),
                                           ([1], 24, 3), ([513], 22, 2), ([2, 900], 24, 1)])
def test_attention_backward_clusters_of_head_sets(ops, lens, heads, kv):
    """The query heads of a kv head over clusters of 2 to 8 CTAs and, where the group has no divisor that leaves at most 8, over one,
    at whole blocks, one row more and one block; the loops' first turns (one to three blocks), whose operands' places are not yet in
    rotation.  Bounds as in the test above; every sum has one order, so two runs are the same bit for bit."""
    test_attention_ragged_blocks_and_head_sets(ops, lens, heads, kv)
    T = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(T)
    q, k, v, do = (torch.randn(T, h, 128, device=DEV, generator=g).to(torch.bfloat16) for h in (heads, kv, kv, heads))
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    o, lse = ops.ext.attention_fwd(q, k, v, cu, max(lens), 128 ** -0.5)
    runs = [ops.ext.attention_bwd(q, k, v, o, do, lse, cu, max(lens), 128 ** -0.5, ops.status_tensor(DEV)) for _ in range(2)]
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("scale", [0.3, 0.0, -0.08])
def test_attention_scale_of_any_sign(ops, scale):
    """Forward and backward against fp64, 1e-2 as for the other attention tests."""
    lens, heads, kv, d = [200, 77, 1, 130], 4, 2, 128
    T = sum(lens)
    torch.manual_seed(9)
    q, k, v, do = (_rand(T, h, d) for h in (heads, kv, kv, heads))
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    o, lse = ops.ext.attention_fwd(q, k, v, cu, max(lens), scale, ops.status_tensor(DEV))
    grads = ops.ext.attention_bwd(q, k, v, o, do, lse, cu, max(lens), scale, ops.status_tensor(DEV))
    q2, k2, v2 = (t.double().requires_grad_(True) for t in (q, k, v))
    outs = []
    for s, n in zip(cu.tolist(), lens):
        qs, ks, vs = (t[s:s + n].transpose(0, 1) for t in (q2, k2.repeat_interleave(heads // kv, 1), v2.repeat_interleave(heads // kv, 1)))
        sc = (qs @ ks.transpose(1, 2)) * scale
        sc = sc.masked_fill(torch.ones(n, n, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
        outs.append((sc.softmax(-1) @ vs).transpose(0, 1))
    ref = torch.cat(outs)
    for name, a, b in zip(("o", "dq", "dk", "dv"), [o] + list(grads), (ref,) + torch.autograd.grad(ref, (q2, k2, v2), do.double())):
        if float(b.norm()) == 0.0:            # scale 0: the scores do not depend on q and k
            assert float(a.float().abs().max()) == 0.0, name
        else:
            assert _rel_err(a, b) < 1e-2, (name, _rel_err(a, b))
    ops.check_status(DEV)


@pytest.mark.parametrize("T", [100, 700])
def test_attention_with_nan_and_infinite_rows(ops, T):
    """NaN in a query row and infinities in a key row reach what they reach in fp64 attention, and nothing else: the other rows
    and heads are bit for bit those of the clean call.  In the backward pass, a NaN in a row of dO makes that row of dQ NaN and
    leaves the other rows and the other heads' gradients as they were (dQ: fp32 sums in another order)."""
    torch.manual_seed(T)
    heads, kv, d, bad, hot = 4, 2, 128, 70, 33
    q, k, v, do = (_rand(T, h, d) for h in (heads, kv, kv, heads))
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)

    def fwd(q, k):
        return ops.ext.attention_fwd(q, k, v, cu, T, d ** -0.5, ops.status_tensor(DEV))
    o, lse = fwd(q, k)
    q2 = q.clone()
    q2[bad, 1] = float("nan")
    o2, _ = fwd(q2, k)
    assert bool(o2[bad, 1].isnan().all())
    keep = torch.ones(T, heads, dtype=torch.bool, device=DEV)
    keep[bad, 1] = False
    assert torch.equal(o2[keep], o[keep])
    k2 = k.clone()
    k2[hot, 0, 7] = float("inf")
    o3, _ = fwd(q, k2)
    qs, ks, vs = (t.double().transpose(0, 1) for t in (q, k2.repeat_interleave(2, 1), v.repeat_interleave(2, 1)))
    sc = (qs @ ks.transpose(1, 2)) * d ** -0.5
    ref = (sc.masked_fill(torch.ones(T, T, device=DEV, dtype=torch.bool).triu(1), float("-inf")).softmax(-1) @ vs).transpose(0, 1)
    nan = ref.isnan()
    assert bool(nan.any()) and torch.equal(o3.isnan(), nan)
    assert float((o3.double() - ref)[~nan].norm()) < 1e-2 * float(ref[~nan].norm())
    assert torch.equal(o3[:hot], o[:hot]) and torch.equal(o3[:, 2:], o[:, 2:])
    grads = ops.ext.attention_bwd(q, k, v, o, do, lse, cu, T, d ** -0.5, ops.status_tensor(DEV))
    do2 = do.clone()
    do2[bad, 1] = float("nan")
    grads2 = ops.ext.attention_bwd(q, k, v, o, do2, lse, cu, T, d ** -0.5, ops.status_tensor(DEV))
    assert bool(grads2[0][bad, 1].isnan().all())
    _close(grads2[0][keep], grads[0][keep], 1e-3, name="dq")
    for i in (1, 2):
        assert torch.equal(grads2[i][:, 1], grads[i][:, 1])          # the other kv head
    ops.check_status(DEV)


@pytest.mark.parametrize("T,first,end,heads,kv", [(512, 5, 300, 4, 4), (512, 5, 300, 32, 8), (700, 0, 1, 8, 2), (300, 290, 300, 4, 2), (4000, 1000, 1600, 4, 1)])
def test_attention_gradients_of_rows_outside_the_sequences_are_zero(ops, T, first, end, heads, kv):
    """Rows before the first and after the last sequence (a padded stream) get zero gradients, whatever the memory held, with
    dK / dV added up in one CTA and over partial sums; the rows inside are those of the call without the padding."""
    torch.manual_seed(T + first)
    q, k, v, do = (_rand(T, h, 128) for h in (heads, kv, kv, heads))

    def cu(*values):
        return torch.tensor(values, dtype=torch.int32, device=DEV)
    o, lse = ops.ext.attention_fwd(q, k, v, cu(first, end), T, 128 ** -0.5)
    poison = [torch.full((T * h * 128 * mult,), float("nan"), dtype=dt, device=DEV)
              for h in (heads, kv, kv) for mult, dt in ((1, torch.bfloat16), (1, torch.float32), (3, torch.float32))]
    del poison                                   # what the next allocations find
    grads = ops.ext.attention_bwd(q, k, v, o, do, lse, cu(first, end), T, 128 ** -0.5, ops.status_tensor(DEV))
    inside = [t[first:end].contiguous() for t in (q, k, v, o, do, lse)]
    ref = ops.ext.attention_bwd(*inside, cu(0, end - first), end - first, 128 ** -0.5, ops.status_tensor(DEV))
    for name, a, b in zip(("dq", "dk", "dv"), grads, ref):
        assert bool((a[:first] == 0).all()) and bool((a[end:] == 0).all()), name
        assert float((a[first:end].float() - b.float()).norm()) <= 1e-2 * float(b.float().norm()) + 1e-3, name
    ops.check_status(DEV)


@pytest.mark.parametrize("bounds", [[0, 150, 300], [0, 150, 40000], [0, 150, 200, 90, 260]])
def test_attention_reports_sequences_outside_its_rows(ops, bounds):
    """cu_seqlens that go past the tensors (by a little, by far, or on a detour): what lies outside is left out and the status
    word says so, in the forward and in the backward pass; the sequence inside is as without the others."""
    from moe_distributed_training_b200.ops.attention_cuda import attention
    torch.manual_seed(83)
    T, n = 200, 150
    q, k, v, do = (_rand(T, h, 128) for h in (4, 2, 2, 4))
    for t in (q, k, v):
        t.requires_grad_(True)

    def cu(values):
        return torch.tensor(values, dtype=torch.int32, device=DEV)
    want = attention(q, k, v, cu([0, n, T]), T)
    want_grads = torch.autograd.grad(want, (q, k, v), do)
    ops.check_status(DEV)
    with torch.no_grad():
        got = attention(q, k, v, cu(bounds), T)
        with pytest.raises(RuntimeError, match="status code 7"):
            ops.check_status(DEV)
        lse = ops.ext.attention_fwd(q, k, v, cu([0, n, T]), T, 128 ** -0.5)[1]
        grads = ops.ext.attention_bwd(q, k, v, want, do, lse, cu(bounds), T, 128 ** -0.5, ops.status_tensor(DEV))
    with pytest.raises(RuntimeError, match="status code 7"):
        ops.check_status(DEV)
    if max(bounds) > 260:
        assert torch.equal(got[:n], want[:n])
        for a, b in zip(grads, want_grads):
            _close(a[:n].flatten(1), b[:n].flatten(1), 1e-3)


@pytest.mark.parametrize("lora", [False, True])
def test_fused_attention_block_matches_composed_ops(ops, lora):
    """The single-node attention sub-block against the same layer evaluated op by op."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.models.mixtral import MixtralDecoderLayer, PackedBatch, moe_args_from_config
    from moe_distributed_training_b200.ops import fused_blocks
    torch.manual_seed(13)
    cfg = MixtralConfig(vocab_size=512, hidden_size=512, intermediate_size=512, num_hidden_layers=1, num_attention_heads=4,
                        num_key_value_heads=2, head_dim=128, num_local_experts=2, num_experts_per_tok=1)
    layer = MixtralDecoderLayer(cfg, moe_args_from_config(cfg, torch.bfloat16, DEV), torch.bfloat16, DEV)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            if "layernorm" in n:
                p.copy_(1 + 0.1 * torch.randn_like(p))
            else:
                p.normal_(0, 0.05)
    if lora:
        for lin in (layer.self_attn.q_proj, layer.self_attn.k_proj, layer.self_attn.v_proj, layer.self_attn.o_proj):
            lin.add_lora(16, 32)
            with torch.no_grad():
                lin.lora_B["default"].weight.normal_(0, 0.05)
    lens = [150, 300]
    T = sum(lens)
    cu = torch.tensor([0, 150, 450], dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens]).int()
    batch = PackedBatch(cu, pos, max(lens))
    x1 = _rand(T, 512).requires_grad_(True)
    x2 = x1.detach().clone().requires_grad_(True)
    params = [p for n, p in layer.named_parameters() if "block_sparse_moe" not in n and "post_attention" not in n and p.requires_grad]
    y1 = fused_blocks.attention_block(layer, x1, batch)
    y2 = x2 + layer.self_attn(layer.input_layernorm(x2), batch)
    _close(y1, y2, 1e-2, "fused attention block fwd")
    go = _rand(T, 512)
    g1 = torch.autograd.grad(y1, [x1] + params, go)
    g2 = torch.autograd.grad(y2, [x2] + params, go)
    for a, b, n in zip(g1, g2, ["x"] + [str(i) for i in range(len(params))]):
        _close(a, b, 2e-2, f"fused attention block grad {n}")
    ops.check_status(DEV)


@pytest.mark.parametrize("T,r", [(1, 16), (130, 8), (257, 64), (700, 72), (1100, 32)])
@pytest.mark.parametrize("which", ["all", "q and v", "frozen o"])
def test_adapter_products_of_a_block_together(ops, T, r, which):
    """The adapters' x A^T, dy B and gradients as one launch for several projections, against the block issued product by product:
    the same fp32 sums in another order and one bf16 rounding each (5e-3).  Rank 72 and partial adapters keep single launches."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.models.mixtral import MixtralDecoderLayer, PackedBatch, moe_args_from_config
    from moe_distributed_training_b200.ops import fused_blocks
    torch.manual_seed(T + r)
    cfg = MixtralConfig(vocab_size=64, hidden_size=384, intermediate_size=128, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=1,
                        head_dim=128, num_local_experts=2, num_experts_per_tok=1)
    layer = MixtralDecoderLayer(cfg, moe_args_from_config(cfg, torch.bfloat16, DEV), torch.bfloat16, DEV)
    attn = layer.self_attn
    lins = [attn.q_proj, attn.v_proj] if which == "q and v" else [attn.q_proj, attn.k_proj, attn.v_proj, attn.o_proj]
    for lin in lins:
        lin.add_lora(r, 2 * r)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p)) if "layernorm" in n else p.normal_(0, 0.05)
            p.requires_grad_("lora" in n)
    if which == "frozen o":
        attn.o_proj.lora_A["default"].weight.requires_grad_(False)
    batch = PackedBatch(torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.arange(T, device=DEV).int(), T)
    x, go = _rand(T, 384), _rand(T, 384)
    params = [p for p in attn.parameters() if p.requires_grad]
    res = []
    for native in (True, False):
        xi = x.clone().requires_grad_(True)
        fused_blocks.NATIVE_ISSUE = native
        try:
            y = fused_blocks.attention_block(layer, xi, batch)
        finally:
            fused_blocks.NATIVE_ISSUE = True
        res.append([y] + list(torch.autograd.grad(y, [xi] + params, go)))
    for i, (a, b) in enumerate(zip(*res)):
        _close(a, b, 5e-3, f"output or gradient {i}")
    ops.check_status(DEV)


@pytest.mark.parametrize("lora", [False, True])
def test_fused_moe_block_matches_composed_ops(ops, lora):
    """The single-node MoE sub-block (local experts) against the same layer evaluated op by op."""
    from moe_distributed_training_b200 import MixtralConfig
    from moe_distributed_training_b200.models.mixtral import MixtralDecoderLayer, moe_args_from_config
    from moe_distributed_training_b200.ops import fused_blocks
    from moe_distributed_training_b200.peft.lora import add_expert_lora
    torch.manual_seed(14)
    cfg = MixtralConfig(vocab_size=512, hidden_size=512, intermediate_size=1024, num_hidden_layers=1, num_attention_heads=4,
                        num_key_value_heads=2, head_dim=128, num_local_experts=4, num_experts_per_tok=2)
    layer = MixtralDecoderLayer(cfg, moe_args_from_config(cfg, torch.bfloat16, DEV), torch.bfloat16, DEV)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            if "layernorm" in n:
                p.copy_(1 + 0.1 * torch.randn_like(p))
            else:
                p.normal_(0, 0.05)
    if lora:
        add_expert_lora(layer.block_sparse_moe.experts, 16, 32)
        with torch.no_grad():
            for p in layer.block_sparse_moe.experts.lora.lora_B.values():
                p.normal_(0, 0.05)
    T = 700
    x1 = _rand(T, 512).requires_grad_(True)
    x2 = x1.detach().clone().requires_grad_(True)
    params = [p for n, p in layer.named_parameters() if ("block_sparse_moe" in n or "post_attention" in n) and p.requires_grad]
    assert fused_blocks.moe_block_supported(layer, x1)
    y1 = fused_blocks.moe_block(layer, x1)
    g1 = torch.autograd.grad(y1, [x1] + params, torch.ones_like(y1) * 0.01, allow_unused=True)
    direct = {id(p): p.grad.clone() for p in params if p.grad is not None}     # expert weights accumulate straight into .grad
    for p in params:
        p.grad = None
    moe_out, _ = layer.block_sparse_moe(layer.post_attention_layernorm(x2))
    y2 = x2 + moe_out
    _close(y1, y2, 1e-2, "fused moe block fwd")
    g2 = torch.autograd.grad(y2, [x2] + params, torch.ones_like(y2) * 0.01, allow_unused=True)
    for i, (a, b, p) in enumerate(zip(g1, g2, [None] + params)):
        if a is None and p is not None:
            a = direct.get(id(p))
        if b is None and p is not None and p.grad is not None:
            b = p.grad
        assert (a is None) == (b is None), i
        if a is not None:
            _close(a, b, 3e-2, f"fused moe block grad {i}")
    ops.check_status(DEV)


def test_group_bwd_ab_direct_products_match_fp32():
    """The reference-named LoRA gradient entry point: four grouped-GEMM launches, full reductions over K and N."""
    from scattermoe_utils.kernels.ops import group_bwd_AB, padded_block_indices
    torch.manual_seed(21)
    E, K, N, r, s = 3, 384, 640, 16, 2.0
    counts = [300, 0, 212]
    M = sum(counts)
    X = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    DY = torch.randn(M, N, device=DEV).to(torch.bfloat16)
    A = (torch.randn(E, K, r, device=DEV) * 0.1).to(torch.bfloat16)
    B = (torch.randn(E, r, N, device=DEV) * 0.1).to(torch.bfloat16)
    offs = torch.tensor(counts, device=DEV).cumsum(0)
    dA, dB = group_bwd_AB(DY, X, A, B, s, offs, E)
    lo = 0
    for e, c in enumerate(counts):
        xe, dye = X[lo:lo + c].float(), DY[lo:lo + c].float()
        wantA = s * xe.t() @ (dye @ B[e].float().t()).to(torch.bfloat16).float()
        wantB = s * (xe @ A[e].float()).to(torch.bfloat16).float().t() @ dye
        if c == 0:
            assert float(dA[e].float().abs().max()) == 0 and float(dB[e].float().abs().max()) == 0
        else:
            _close(dA[e], wantA, 3e-2, f"dA[{e}]")
            _close(dB[e], wantB, 3e-2, f"dB[{e}]")
        lo += c
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    pbi, eo = padded_block_indices(ids, E)
    assert pbi.tolist() == [0, 128, 256, 300, 428] and eo.tolist() == [300, 300, 512]


def test_residual_connections_fused_into_their_producers(ops):
    """x + f(x) without a separate add: the GEMM epilogue, the gate-weighted combine and the RMSNorm backward take the
    residual (or its gradient) as an extra input; the router backward adds into an existing gradient."""
    torch.manual_seed(31)
    ext = ops.ext
    M, K, N = 333, 512, 768
    x, w, res = _rand(M, K), _rand(N, K, scale=0.05), _rand(M, N)
    for policy in (0, 2, 5):                                # 128-row tiles, the CTA pair, the default choice
        prev = ext.gemm_set_pair_policy(policy)
        try:
            got = ops.mm_nt(x, w, residual=res)
        finally:
            ext.gemm_set_pair_policy(prev)
        _close(got, x.float() @ w.float().t() + res.float(), name=f"gemm + residual (policy {policy})")
    # combine
    T, k, H = 200, 2, 256
    y = _rand(T * k + 56, H)
    dest = torch.randperm(T * k + 56, device=DEV)[:T * k].int()
    wts = torch.rand(T, k, device=DEV).to(torch.bfloat16)
    r2 = _rand(T, H)
    got = ext.combine_rows(y, dest, wts, k, r2)
    want = (y.float()[dest.long()].view(T, k, H) * wts.float()[:, :, None]).sum(1) + r2.float()
    _close(got, want, name="combine + residual")
    # rmsnorm backward + residual gradient, and the weight gradient finished in one launch
    R, C = 300, 512
    xx, ww, dy, dres = _rand(R, C), (1 + 0.1 * torch.randn(C, device=DEV)).to(torch.bfloat16), _rand(R, C), _rand(R, C)
    _, rstd = ext.rmsnorm_fwd(xx, ww, 1e-5)
    dx, dwp = ext.rmsnorm_bwd(xx, ww, dy, rstd, dres)
    xf = xx.float().requires_grad_(True)
    wf = ww.float().requires_grad_(True)
    yf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    yf.backward(dy.float())
    _close(dx, xf.grad + dres.float(), name="rmsnorm dx + residual gradient")
    _close(ext.rmsnorm_dw(dwp, ww)[None], wf.grad[None], 3e-2, name="rmsnorm dw")
    # router backward accumulating into an existing gradient
    Tk, Hh, E = 150, 256, 8
    xr, wr = _rand(Tk, Hh), _rand(E, Hh, scale=0.1)
    _, _, idx = ext.router_fwd(xr, wr, 2, True)
    dwts = _rand(Tk, 2)
    dx_plain, _ = ext.router_bwd(xr, wr, idx, dwts, None, True)
    base = _rand(Tk, Hh)
    acc = base.clone()
    ext.router_bwd(xr, wr, idx, dwts, None, True, acc)
    _close(acc, base.float() + dx_plain.float(), name="router dx accumulate")


def test_deterministic_kernels_are_bitwise_reproducible(ops):
    """Routing plan, row gather, the GEMM family (dense, row-grouped with fused SwiGLU, depth-grouped), RMSNorm and
    the gate-weighted combine use no atomics on their results: two runs on the same inputs agree bit for bit."""
    torch.manual_seed(41)
    ext = ops.ext
    T, k, E, H, F = 900, 2, 4, 512, 1024
    x = _rand(T, H)
    top = torch.randn(T, E, device=DEV).topk(k, -1).indices.int()
    w1, w2, w3 = (_rand(E, F, H, scale=0.05) for _ in range(3))
    wts = torch.rand(T, k, device=DEV).to(torch.bfloat16)

    def run():
        plan = ops.make_plan(top, E)
        xg = ext.gather_rows(x, plan.src_slot, plan.padded_offsets, E, None, k)
        y = ops.grouped_swiglu_mlp(xg, w1, w2, w3, plan)
        out = ext.combine_rows(y, plan.dest_row, wts, k, x)
        dw = torch.empty(E, F, H, dtype=torch.bfloat16, device=DEV)
        ops._g(2, y.new_zeros(xg.shape[0], F) + 1, True, xg, True, dw, H, 0, plan)
        dense = ops.mm_nt(x, w1[0])
        xn, rstd = ext.rmsnorm_fwd(x, torch.ones(H, dtype=torch.bfloat16, device=DEV), 1e-5)
        used = int(plan.padded_offsets[-1])      # rows past the padded groups are never written
        return [plan.tokens_per_expert, plan.padded_offsets, plan.dest_row, plan.src_slot, xg[:used], y[:used], out, dw, dense, xn, rstd]

    a, b = run(), run()
    torch.cuda.synchronize()
    for i, (p, q) in enumerate(zip(a, b)):
        assert torch.equal(p, q), f"output {i} differs between two runs"
    ops.check_status(DEV)


def test_router_kernel_histogram_and_score_sums(ops):
    """The router kernel's optional statistics (per-expert slot counts and score sums, the f_e and P_e of the
    load-balancing loss) against a count and a sum over its own outputs; the loss built from them equals the plain one."""
    from moe_distributed_training_b200.ops.reference import load_balancing_loss
    torch.manual_seed(51)
    for (T, H, E, k) in [(700, 512, 8, 2), (37, 256, 16, 4)]:
        x, w = _rand(T, H), _rand(E, H, scale=0.2)
        scores, weights, idx, stats = ops.ext.router_fwd(x, w, k, True, True)
        counts = torch.bincount(idx.reshape(-1).long(), minlength=E).float()
        assert torch.equal(stats[:E], counts)
        assert torch.allclose(stats[E:], scores.float().sum(0), rtol=1e-4, atol=1e-3)
        s2, w2, i2 = ops.ext.router_fwd(x, w, k, True)
        assert torch.equal(s2, scores) and torch.equal(i2, idx) and torch.equal(w2, weights)
        f = stats[:E] / (T * k)
        loss = E * torch.sum(f * scores.float().mean(0))
        assert torch.allclose(loss, load_balancing_loss(scores.float(), idx, E, k), rtol=1e-5)


def test_gemm_last_round_shared_along_the_depth(ops):
    """Products whose last round of 128-row tiles would leave most SMs idle: the k blocks of that round are cut into one
    piece per SM, partial sums meet in an fp32 workspace, the last contributor of each tile quarter finishes it.  Checked
    against fp32 and against the same product with the sharing switched off, for the epilogue variants that can meet it
    (plain, LoRA segment, residual, fp32 accumulation, MN-major weights, row groups), twice in a row (the workspace
    must come back clean)."""
    ext = ops.ext
    torch.manual_seed(61)
    prev_policy = ext.gemm_set_pair_policy(0)          # the 128-row kernel
    try:
        for (M, N, K) in [(1280, 4096, 2048), (576, 4096, 1024), (576, 1024, 4096), (200, 2048, 8192)]:
            x, w = _rand(M, K), _rand(N, K, scale=0.05)
            want = x.float() @ w.float().t()
            for rep in range(2):
                _close(ops.mm_nt(x, w), want, name=f"split nt {M}x{N}x{K} run {rep}")
            old = ext.gemm_set_split(0)
            try:
                unsplit = ops.mm_nt(x, w)
            finally:
                ext.gemm_set_split(old)
            _close(ops.mm_nt(x, w), unsplit.float(), 1e-2, name=f"split vs unsplit {M}x{N}x{K}")
        M, N, K, r = 576, 4096, 1024, 16
        x, w, res = _rand(M, K), _rand(N, K, scale=0.05), _rand(M, N)
        t, b = _rand(M, r), _rand(N, r, scale=0.1)
        _close(ops.mm_nt(x, w, lora=(t, b), residual=res), x.float() @ w.float().t() + t.float() @ b.float().t() + res.float(),
               name="split + lora + residual")
        w2 = _rand(K, N, scale=0.05)
        out32 = torch.ones(M, N, device=DEV)
        ops._gemm(0, x, False, w2, True, out32, M, N, K, accumulate=True, alpha=0.5)
        _close(out32, 1.0 + 0.5 * (x.float() @ w2.float()), name="split + fp32 accumulate, MN-major weights")
        # row groups (expert down projection): 3 experts
        E, F, H = 3, 2048, 4096
        top = (torch.arange(700, device=DEV) % E).int()[:, None]
        plan = ops.make_plan(top, E)
        hg = _rand(int(plan.src_slot.numel()), F)
        w2g = _rand(E, F, H, scale=0.03)
        y = torch.empty(hg.shape[0], H, dtype=torch.bfloat16, device=DEV)
        ops._g(1, hg, False, w2g, True, y, H, F, plan)
        offs = plan.padded_offsets.tolist()
        for e in range(E):
            a, bnd = offs[e], offs[e + 1]
            _close(y[a:bnd], hg[a:bnd].float() @ w2g[e].float(), name=f"split grouped rows, expert {e}")
    finally:
        ext.gemm_set_pair_policy(prev_policy)
    ops.check_status(DEV)


def test_shared_last_round_first_used_on_a_stream_beside_a_busy_default_stream(ops):
    """The fp32 workspace of the shared last round is made on a stream's first such product.  It has to be clean for that
    product and for the next ones although the default stream, against which pool streams are not ordered, is busy."""
    ext = ops.ext
    torch.manual_seed(62)
    M, N, K = 1280, 4096, 2048                          # 160 tiles of 128 rows: 12 of them shared on 148 SMs
    x, w = _rand(M, K), _rand(N, K, scale=0.05)
    prev_policy, prev_split = ext.gemm_set_pair_policy(0), ext.gemm_set_split(0)
    try:
        unsplit = ops.mm_nt(x, w).float()
        ext.gemm_set_split(1)
        for priority in (0, -1, 0, -1):
            side = torch.cuda.Stream(priority=priority)
            side.wait_stream(torch.cuda.current_stream())
            torch.cuda._sleep(20_000_000)               # about 10 ms of the default stream
            with torch.cuda.stream(side):
                got = [ops.mm_nt(x, w) for _ in range(6)]
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                got.append(ops.mm_nt(x, w))
            torch.cuda.synchronize()
            for i, y in enumerate(got):                 # the same products, their fp32 sums in another order: one bf16 rounding apart
                _close(y, unsplit, 1e-2, name=f"shared last round on a fresh stream, product {i}")
    finally:
        ext.gemm_set_split(prev_split)
        ext.gemm_set_pair_policy(prev_policy)
    ops.check_status(DEV)


@pytest.mark.parametrize("where", ["number", "gpu", "cpu tensor", "fp64 gpu"])
def test_clipping_factor_in_the_update(ops, where):
    """AdamW with the factor as a number and as a scalar on the GPU: the same update, against the fp32 statement; a scalar that
    the kernel cannot read there is read by the host.  bf16 results: one rounding (0.4 %)."""
    from moe_distributed_training_b200.ops import reference
    torch.manual_seed(5)
    for n in (1, 7, 4096, 33333):
        p, g = _rand(n), _rand(n)
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        want = [t.float().clone() for t in (p, m, v)]
        reference.adamw_step(want[0], g.float(), want[1], want[2], 1e-2, 0.9, 0.999, 1e-8, 0.01, 1, 0.125)
        scale = {"number": 0.125, "gpu": torch.tensor(0.125, device=DEV), "cpu tensor": torch.tensor(0.125),
                 "fp64 gpu": torch.tensor(0.125, device=DEV, dtype=torch.float64)}[where]
        ops.adamw_multi([p], [g], [m], [v], 1e-2, 0.9, 0.999, 1e-8, 0.01, 1, scale)
        for name, a, b in zip(("p", "m", "v"), (p, m, v), want):
            torch.testing.assert_close(a.float(), b, rtol=8e-3, atol=1e-6, msg=lambda t: f"{name} of {n}, {where}: {t}")


def test_clipping_factor_set_on_the_gpu_reads_as_a_number(ops):
    from moe_distributed_training_b200.optim.adamw import FusedAdamW
    from moe_distributed_training_b200.optim.clip import clip_grad_norm_
    lin = torch.nn.Linear(64, 8, bias=False, device=DEV, dtype=torch.bfloat16)
    opt = FusedAdamW(lin.parameters(), lr=0.1)
    lin.weight.grad = torch.ones_like(lin.weight)
    clip_grad_norm_(lin, 1.0, optimizer=opt)
    assert type(opt.grad_scale) is float and abs(opt.grad_scale - 1.0 / 512 ** 0.5) < 1e-5


@pytest.mark.parametrize("bounds_on", ["cuda", "cpu"])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_shifted_labels_with_bounds_on_either_device(bounds_on, dtype):
    from moe_distributed_training_b200.models.mixtral import shift_labels
    labels = torch.arange(10, 21, device=DEV)
    cu = torch.tensor([0, 0, 4, 5, 11], dtype=dtype, device=bounds_on)        # an empty first sequence, and one of a single token
    want = [11, 12, 13, -100, -100, 16, 17, 18, 19, 20, -100]
    assert shift_labels(labels, cu).tolist() == want


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("layout", ["plain", "strided", "odd start"])
def test_parallel_linear_lora_slot_order_on_the_gpu(ops, gated, layout):
    """Slot-ordered calls (plan from the slots, no permutation) against fp64 of the definition: experts without rows, tokens and
    output gradients that are strided or that start between two 16-byte pieces (a view into a larger buffer).  bf16 inputs,
    intermediates (hidden rank products, gate weights) and results: 2e-2 as for the other products, gradients of gates and
    factors included."""
    from scattermoe_utils.parallel_linear_lora import parallel_linear_lora
    torch.manual_seed(17)
    T, K, N, E, r, k = 203, 264, 136, 5, 16, 2

    def place(t):
        if layout == "plain":
            return t
        if layout == "strided":
            return torch.stack([t, t], -1)[..., 0]
        buf = torch.empty(t.numel() + 3, dtype=t.dtype, device=DEV)[3:]
        return buf.copy_(t.reshape(-1)).view(t.shape)
    experts = torch.randint(0, E - 1, (T, k), device=DEV)                   # the last expert gets nothing
    ids, order = torch.sort(experts.reshape(-1), stable=True)
    x = place(_rand(T, K)).requires_grad_(True)
    W = _rand(E, K, N, scale=0.05)
    A, B = _rand(E, K, r, scale=0.05).requires_grad_(True), _rand(E, r, N, scale=0.05).requires_grad_(True)
    g = torch.rand(T, k, device=DEV).to(torch.bfloat16).requires_grad_(True) if gated else None
    dy = place(_rand(T if gated else T * k, N))
    if layout == "odd start":
        assert x.is_contiguous() and x.data_ptr() % 16 != 0 and dy.data_ptr() % 16 != 0
    y = parallel_linear_lora(x, W, A, B, r, 32.0, k, ids, order, gates=g)
    wrt = [x, A, B] + ([g] if gated else [])
    grads = torch.autograd.grad(y, wrt, dy)
    x64, A64, B64 = (t.detach().double().requires_grad_(True) for t in (x, A, B))
    g64 = g.detach().double().requires_grad_(True) if gated else None
    eff = W.double() + 2.0 * A64 @ B64                                      # lora_alpha / r = 2
    slots = torch.einsum("tk,tckn->tcn", x64, eff[experts])
    ref = (slots * g64[..., None]).sum(1) if gated else slots.reshape(T * k, N)
    ref_grads = torch.autograd.grad(ref, [x64, A64, B64] + ([g64] if gated else []), dy.double())
    _close(y, ref, name="y")
    for name, a, b in zip(("x", "A", "B", "gates"), grads, ref_grads):
        assert a.shape == b.shape and _rel_err(a, b) < 2e-2, (name, _rel_err(a, b))
    ops.check_status(DEV)


def test_row_kernels_refuse_rows_that_start_between_two_pieces(ops):
    """The kernels move 16 bytes at a time: the bindings answer with an error instead of a misaligned access."""
    top = torch.zeros(8, 1, dtype=torch.int32, device=DEV)
    plan = ops.make_plan(top, 1)
    odd = torch.zeros(8 * 64 + 1, dtype=torch.bfloat16, device=DEV)[1:].view(8, 64)
    with pytest.raises(RuntimeError, match="16-byte"):
        ops.ext.gather_rows(odd, plan.src_slot, plan.padded_offsets, 1, None, 1)
    with pytest.raises(RuntimeError, match="16-byte"):
        ops.ext.combine_rows(odd, plan.dest_row, None, 1)
    with pytest.raises(RuntimeError, match="16-byte"):
        ops.ext.combine_wgrad(torch.zeros(8, 64, dtype=torch.bfloat16, device=DEV), plan.dest_row, odd, 1)


@pytest.mark.parametrize("block", [False, True])
def test_expert_gradients_written_then_added(ops, block):
    """Two micro-batches into fresh `.grad`s (the first product writes, the second adds), for the experts on their own and for
    the decoder layers' MoE sub-block, against the same module on torch's operators.  bf16 gradients, rounded after each
    micro-batch on both sides: 2e-2 as for the other products."""
    from moe_distributed_training_b200 import MixtralConfig, ops as front
    from moe_distributed_training_b200.config import MoEArguments
    from moe_distributed_training_b200.models.mixtral import MixtralForCausalLM
    from moe_distributed_training_b200.moe.layer import dMoE
    torch.manual_seed(23)
    if block:
        cfg = MixtralConfig(vocab_size=256, hidden_size=256, intermediate_size=384, num_hidden_layers=1, num_attention_heads=2,
                            num_key_value_heads=1, head_dim=128, num_local_experts=4, num_experts_per_tok=2)
        module = MixtralForCausalLM(cfg, dtype=torch.bfloat16, device=DEV)
        batches = [torch.randint(0, 256, (1, n), device=DEV) for n in (150, 211)]
    else:
        module = dMoE(MoEArguments(hidden_size=256, ffn_hidden_size=384, moe_num_experts=4, moe_top_k=2, bf16=True, device=DEV))
        batches = [_rand(1, n, 256) for n in (150, 211)]
    with torch.no_grad():
        for name, p in module.named_parameters():
            if "norm" not in name:
                p.normal_(0.0, 0.2 if "router" in name else 0.05)

    def run():
        module.zero_grad(set_to_none=True)
        for b in batches:
            if block:
                module(b, labels=b).loss.backward()
            else:
                y, _ = module(b)
                (y.float() * torch.linspace(-1, 1, y.numel(), device=DEV).view_as(y)).sum().backward()
        return {n: p.grad.clone() for n, p in module.named_parameters() if n.endswith((".w1", ".w2", ".w3"))}
    got = run()
    front.set_backend("library")
    try:
        want = run()
    finally:
        front.set_backend("native")
    assert len(got) == 3 and got.keys() == want.keys()
    for n in got:
        assert _rel_err(got[n], want[n]) < 2e-2, (n, _rel_err(got[n], want[n]))
    ops.check_status(DEV)


def test_shared_last_round_on_a_stream_first_used_under_capture(ops):
    """A capture can neither allocate the workspace nor clear it: the product runs unsplit, in the capture and in every replay."""
    ext = ops.ext
    torch.manual_seed(63)
    x, w = _rand(1280, 2048), _rand(4096, 2048, scale=0.05)
    prev_policy, prev_split = ext.gemm_set_pair_policy(0), ext.gemm_set_split(0)
    try:
        unsplit = ops.mm_nt(x, w)
        ext.gemm_set_split(1)
        out = torch.empty_like(unsplit)
        side = [torch.cuda.Stream(priority=-1) for _ in range(7)][-1]        # further on in the pool than the other tests
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            ops.mm_nt(x, w, out=out)
        for _ in range(2):
            out.fill_(float("nan"))
            graph.replay()
            torch.cuda.synchronize()
            _close(out, unsplit.float(), 1e-2, name="captured product")
    finally:
        ext.gemm_set_split(prev_split)
        ext.gemm_set_pair_policy(prev_policy)
    ops.check_status(DEV)


def test_multi_tensor_gradient_accumulate(ops):
    """fp32 accumulators += bf16 / fp32 gradients of many tensors in one launch per 16."""
    torch.manual_seed(71)
    shapes = [(16, 4096), (4096, 16), (1024, 16), (16, 1024), (7,), (3, 5, 11)] * 4      # 24 tensors: two launches
    dst = [torch.randn(*s_, device=DEV) for s_ in shapes]
    src = [(torch.randn(*s_, device=DEV).to(torch.bfloat16) if i % 3 else torch.randn(*s_, device=DEV)) for i, s_ in enumerate(shapes)]
    want = [d + s_.float() for d, s_ in zip(dst, src)]
    ops.ext.multi_add(dst, src)
    for got, w in zip(dst, want):
        assert torch.equal(got, w)
