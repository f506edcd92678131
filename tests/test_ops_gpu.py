"""Numerics of the sm_100a kernels against plain fp32 PyTorch references of the same ops."""


import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def bf16(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


def rel_err(a, b):
    """Largest element error relative to the largest reference element (catches a single bad tile)."""
    return (a.float() - b.float()).abs().max().item() / max(b.float().abs().max().item(), 1e-6)


def norm_err(a, b):
    """Frobenius norm of the error over the Frobenius norm of the reference.  Rounding a correct
    fp32 result to bf16 gives about 2e-3 here; an element-wise bug in a few percent of the entries,
    which the max-based measure above lets through, does not."""
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("impl", ["single", "pair"])
@pytest.mark.parametrize("a_k,b_k", [(True, True), (True, False), (False, False), (False, True)])
@pytest.mark.parametrize("shape", [(128, 256, 64), (384, 520, 328), (1024, 1024, 512), (2304, 19200, 192)])
def test_gemm_all_layouts(a_k, b_k, shape, impl):
    """(2304, 19200, 192): 9 x 75 tiles of 256 x 256 = 675 = 9 waves of 74 pairs + 9, so the pair
    kernel's split tail (halves of the last tiles) is exercised; 520 and 328 are ragged edges."""
    import functools

    from torchft_b200.ops import _lib
    from torchft_b200.ops.gemm import gemm as _gemm

    gemm = functools.partial(_gemm, impl=impl)

    M, N, K = shape
    a = bf16(M, K) if a_k else bf16(K, M)
    b = bf16(N, K) if b_k else bf16(K, N)
    A = a.float() if a_k else a.float().t()
    B = b.float().t() if b_k else b.float()
    ref = A @ B
    out = gemm(a, b, a_kmajor=a_k, b_kmajor=b_k)
    assert rel_err(out, ref) < 1e-2 and norm_err(out, ref) < 4e-3
    out32 = gemm(a, b, a_kmajor=a_k, b_kmajor=b_k, out_dtype=torch.float32)
    assert rel_err(out32, ref) < 1e-4 and norm_err(out32, ref) < 1e-5
    acc = bf16(M, N)
    ref2 = ref + acc.float()
    gemm(a, b, acc, a_kmajor=a_k, b_kmajor=b_k, accumulate=True)
    assert rel_err(acc, ref2) < 1e-2 and norm_err(acc, ref2) < 4e-3
    _lib.check_status("gemm")


# The products of one Llama-3-8B layer and of the head at the benchmark's 4096 tokens:
# (name, layout, M, N, K) with layout = (A is K-major, B is K-major).
LLAMA_GEMMS = [
    ("wqkv forward", (True, True), 4096, 6144, 4096),
    ("w13 forward", (True, True), 4096, 28672, 4096),
    ("w2 forward", (True, True), 4096, 4096, 14336),
    ("head forward", (True, True), 4096, 128256, 4096),
    ("w13 input gradient", (True, False), 4096, 4096, 28672),
    ("w13 weight gradient", (False, False), 28672, 4096, 4096),
    ("w2 weight gradient", (False, False), 4096, 14336, 4096),
]


@pytest.mark.parametrize("name,layout,M,N,K", LLAMA_GEMMS, ids=[g[0].replace(" ", "_") for g in LLAMA_GEMMS])
def test_gemm_at_benchmark_shapes(name, layout, M, N, K):
    from torchft_b200.ops import _lib
    from torchft_b200.ops.gemm import gemm

    a_k, b_k = layout
    torch.manual_seed(M + N + K)
    a = bf16(M, K, scale=0.5) if a_k else bf16(K, M, scale=0.5)
    b = bf16(N, K, scale=0.05) if b_k else bf16(K, N, scale=0.05)
    ref = (a.float() if a_k else a.float().t()) @ (b.float().t() if b_k else b.float())  # fp32, no TF32
    for impl in ("single", "pair"):
        out = gemm(a, b, a_kmajor=a_k, b_kmajor=b_k, impl=impl)
        assert rel_err(out, ref) < 1e-2 and norm_err(out, ref) < 4e-3, (name, impl)
        del out
    out32 = gemm(a, b, a_kmajor=a_k, b_kmajor=b_k, out_dtype=torch.float32, impl="pair")
    # fp32 output: what is left is the order of the fp32 summation over K (up to 28672 terms here)
    assert norm_err(out32, ref) < 1e-4, name
    _lib.check_status("gemm")


def test_linear_autograd_and_main_grad():
    from torchft_b200.ops.functional import linear

    x = bf16(4, 96, 256, scale=0.5).requires_grad_()
    w = bf16(512, 256, scale=0.05).requires_grad_()
    y = linear(x, w)
    dy = bf16(4, 96, 512)
    y.backward(dy)
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = xf @ wf.t()
    yf.backward(dy.float())
    assert rel_err(y, yf) < 1e-2 and norm_err(y, yf) < 4e-3
    assert rel_err(x.grad, xf.grad) < 1e-2 and norm_err(x.grad, xf.grad) < 4e-3
    assert rel_err(w.grad, wf.grad) < 1e-2 and norm_err(w.grad, wf.grad) < 4e-3

    # gradient accumulation straight into a preallocated buffer
    w2 = w.detach().clone().requires_grad_()
    w2.main_grad = torch.empty_like(w2)
    for _ in range(2):
        linear(x.detach(), w2).backward(dy)
    assert w2.grad is None
    assert rel_err(w2.main_grad, 2 * wf.grad) < 1e-2


@pytest.mark.parametrize("dim", [2048, 4096, 768])
def test_rmsnorm_fwd_bwd(dim):
    from torchft_b200.ops.functional import add_rmsnorm, rmsnorm

    rows = 300
    x = bf16(rows, dim).requires_grad_()
    w = (1 + 0.1 * torch.randn(dim, device=DEV)).to(torch.bfloat16).requires_grad_()
    y = rmsnorm(x, w, 1e-5)
    dy = bf16(rows, dim)
    y.backward(dy)

    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    yf.backward(dy.float())
    assert rel_err(y, yf) < 1e-2 and norm_err(y, yf) < 4e-3
    assert rel_err(x.grad, xf.grad) < 2e-2 and norm_err(x.grad, xf.grad) < 5e-3
    assert rel_err(w.grad, wf.grad) < 2e-2 and norm_err(w.grad, wf.grad) < 5e-3

    # fused residual add
    a, r = bf16(rows, dim).requires_grad_(), bf16(rows, dim).requires_grad_()
    w2 = w.detach().clone().requires_grad_()
    y2, h2 = add_rmsnorm(a, r, w2, 1e-5)
    dh = bf16(rows, dim)
    (y2.float() * dy.float()).sum().add((h2.float() * dh.float()).sum()).backward()
    af, rf, w2f = a.detach().float().requires_grad_(), r.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    hf = (af + rf).to(torch.bfloat16).float() + 0 * (af + rf)  # forward value rounded like the kernel
    hf = (af + rf)
    yf2 = hf * torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + 1e-5) * w2f
    ((yf2 * dy.float()).sum() + (hf * dh.float()).sum()).backward()
    assert rel_err(h2, hf) < 1e-2 and rel_err(y2, yf2) < 2e-2
    assert rel_err(a.grad, af.grad) < 2e-2 and torch.equal(a.grad, r.grad)
    assert rel_err(w2.grad, w2f.grad) < 2e-2


@pytest.mark.parametrize("hd", [64, 128])
def test_rope_matches_reference_and_inverts(hd):
    from torchft_b200.ops.functional import rope_, rope_table

    T, H = 200, 6
    theta = 500000.0
    cs = rope_table(256, hd, theta, torch.device(DEV))
    x = bf16(T, H * hd)
    ref = x.float().view(T, H, hd)
    pos = torch.arange(T, device=DEV, dtype=torch.float32)
    inv = theta ** (-torch.arange(hd // 2, device=DEV, dtype=torch.float32) / (hd // 2))
    ang = pos[:, None] * inv[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]
    a, b = ref[..., : hd // 2], ref[..., hd // 2 :]
    expect = torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1).view(T, H * hd)
    y = x.clone()
    rope_(y, cs, H, hd)
    assert rel_err(y, expect) < 1e-2
    rope_(y, cs, H, hd, inverse=True)
    assert rel_err(y, x) < 2e-2
    # view into a wider fused buffer
    wide = bf16(T, 3 * H * hd)
    q = wide[:, : H * hd]
    keep = wide[:, H * hd :].clone()
    expect_q = wide[:, : H * hd].clone()
    rope_(expect_q.contiguous(), cs, H, hd)
    e2 = wide[:, : H * hd].contiguous()
    rope_(e2, cs, H, hd)
    rope_(q, cs, H, hd)
    assert torch.equal(wide[:, : H * hd], e2) and torch.equal(wide[:, H * hd :], keep)


def test_swiglu():
    from torchft_b200.ops.functional import swiglu

    gu = bf16(130, 2 * 1024).requires_grad_()
    out = swiglu(gu)
    d = bf16(130, 1024)
    out.backward(d)
    gf = gu.detach().float().requires_grad_()
    g, u = gf[:, :1024], gf[:, 1024:]
    of = torch.nn.functional.silu(g) * u
    of.backward(d.float())
    assert rel_err(out, of) < 1e-2 and norm_err(out, of) < 4e-3
    assert rel_err(gu.grad, gf.grad) < 2e-2 and norm_err(gu.grad, gf.grad) < 5e-3


@pytest.mark.parametrize("rows", [64, 4096])  # 4096 x 128256 is the benchmark's logits matrix
def test_cross_entropy_loss_and_grad(rows):
    from torchft_b200.ops.functional import cross_entropy

    V = 128256
    logits = bf16(rows, V, scale=2.0)
    targets = torch.randint(V, (rows,), device=DEV)
    lf = logits.float().requires_grad_()
    ref = torch.nn.functional.cross_entropy(lf, targets)
    ref.backward()
    work = logits.clone().requires_grad_()
    loss = cross_entropy(work, targets)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * abs(ref.item())
    assert (work.grad.float() - lf.grad).abs().max().item() < 2e-2 * lf.grad.abs().max().item() + 1e-6
    assert norm_err(work.grad, lf.grad) < 5e-3

    # ignore_index
    targets2 = targets.clone()
    targets2[::3] = -100
    lf2 = logits.float().requires_grad_()
    ref2 = torch.nn.functional.cross_entropy(lf2, targets2, ignore_index=-100)
    work2 = logits.clone().requires_grad_()
    loss2 = cross_entropy(work2, targets2, ignore_index=-100)
    assert abs(loss2.item() - ref2.item()) < 2e-3 * abs(ref2.item())


def test_embedding_fwd_bwd():
    from torchft_b200.ops.functional import embedding

    V, D = 1000, 256
    table = bf16(V, D).requires_grad_()
    tokens = torch.randint(V, (4, 50), device=DEV)
    tokens[0, :10] = 7  # repeated rows exercise the atomics
    out = embedding(tokens, table)
    assert torch.equal(out, table.detach()[tokens])
    d = bf16(4, 50, D)
    out.backward(d)
    ref = torch.zeros(V, D, device=DEV)
    ref.index_add_(0, tokens.reshape(-1), d.float().view(-1, D))
    assert rel_err(table.grad, ref) < 3e-2


def test_adamw_matches_torch():
    from torchft_b200.ops.functional import adamw_step_

    n = 8 * 1000 + 5
    p = bf16(n)
    m = torch.zeros(n, device=DEV)
    v = torch.zeros(n, device=DEV)
    ref_p = p.float().clone().requires_grad_()
    opt = torch.optim.AdamW([ref_p], lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        g = bf16(n)
        ref_p.grad = g.float()
        opt.step()
        adamw_step_(p, g, m, v, lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
        # the kernel rounds the parameter to bf16 each step; keep the reference in lockstep
        assert (p.float() - ref_p.detach()).abs().max().item() < 1e-2 * ref_p.detach().abs().max().item()
        ref_p.data.copy_(p.float())
    st = opt.state[ref_p]
    assert rel_err(m, st["exp_avg"]) < 1e-4 and rel_err(v, st["exp_avg_sq"]) < 1e-4


def test_fused_adamw_optimizer_on_bf16_parameters():
    """``FusedAdamW`` (one kernel per bf16 parameter, fp32 moments) against ``torch.optim.AdamW`` on fp32 copies."""
    from torchft_b200.optim import FusedAdamW

    params = [torch.nn.Parameter(bf16(257, 33)), torch.nn.Parameter(bf16(1000))]
    refs = [torch.nn.Parameter(p.detach().float().clone()) for p in params]
    kw = dict(lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    ours, theirs = FusedAdamW(params, **kw), torch.optim.AdamW(refs, **kw)
    for _ in range(3):
        for p, q in zip(params, refs):
            g = bf16(*p.shape)
            p.grad, q.grad = g, g.float()
        ours.step()
        theirs.step()
        for p, q in zip(params, refs):
            assert (p.float() - q.detach()).abs().max().item() < 1e-2 * q.detach().abs().max().item()
            q.data.copy_(p.float())  # the kernel rounds the parameter to bf16 each step
    for p, q in zip(params, refs):
        assert ours.state[p]["exp_avg"].dtype == torch.float32
        assert rel_err(ours.state[p]["exp_avg"], theirs.state[q]["exp_avg"]) < 1e-4
        assert rel_err(ours.state[p]["exp_avg_sq"], theirs.state[q]["exp_avg_sq"]) < 1e-4


def test_diloco_fused_outer_step_matches_sgd():
    from torchft_b200.local_sgd import _FlatBuckets
    from torchft_b200.ops.outer_step import FusedOuterStep

    torch.manual_seed(0)
    params = [torch.nn.Parameter(bf16(33, 7)), torch.nn.Parameter(bf16(129))]
    ref_params = [torch.nn.Parameter(p.detach().float().clone()) for p in params]
    outer = torch.optim.SGD(params, lr=0.7, momentum=0.9, nesterov=True)
    ref_outer = torch.optim.SGD(ref_params, lr=0.7, momentum=0.9, nesterov=True)
    backup = _FlatBuckets(params, None, False)
    backup.copy_from_params()
    comm = _FlatBuckets(params, None, False)
    fused = FusedOuterStep.maybe_create(params, backup, comm, outer)
    assert fused is not None
    for _ in range(3):
        global_ref = [p.detach().clone() for p in ref_params]
        deltas = [torch.randn_like(p).mul(0.01).to(torch.bfloat16) for p in params]
        with torch.no_grad():
            for p, d in zip(params, deltas):
                p.add_(d)
        fused.compute_pseudogradients()
        fused.apply_outer_update()
        for rp, gp, p, d in zip(ref_params, global_ref, params, deltas):
            rp.data.copy_(gp)
            rp.grad = (p.detach().float() * 0 + d.float())
        ref_outer.step()
        for p, rp, i in zip(params, ref_params, range(2)):
            assert (p.detach().float() - rp.detach()).abs().max().item() < 3e-2 * rp.detach().abs().max().item()
            assert torch.equal(backup.views[i], p.detach())
            rp.data.copy_(p.detach().float())
            ref_outer.state[rp]["momentum_buffer"].copy_(outer.state[p]["momentum_buffer"])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("momentum,nesterov", [(0.9, True), (0.9, False), (0.0, False)])
def test_outer_step_reads_and_writes_the_parameters_in_place(dtype, momentum, nesterov):
    """Sizes around a vector and a block's chunk, a strided parameter, one at an odd address, more tensors than one table
    holds.  The expected values follow the kernels' arithmetic (fp32, one rounding to ``dtype`` of the pseudo-gradient and
    of the new weight), so a result may differ by one rounding of ``dtype`` where a multiply-add was contracted."""
    from torchft_b200.local_sgd import _FlatBuckets
    from torchft_b200.ops.outer_step import FusedOuterStep

    chunk = 256 * 4 * (16 // torch.empty(0, dtype=dtype).element_size())
    sizes = [1, 7, 8, 9, chunk - 1, chunk, chunk + 1, 3 * chunk + 5] + [3] * 125
    base = torch.randn(sum(sizes) + 1, device=DEV).to(dtype)
    params, at = [], 1  # from element 1 on: most of these views start at no 16-byte boundary
    for n in sizes[:4]:
        params.append(torch.nn.Parameter(base[at : at + n]))
        at += n
    params += [torch.nn.Parameter(torch.randn(n, device=DEV).to(dtype)) for n in sizes[4:]]
    params.append(torch.nn.Parameter(torch.randn(48, 80, device=DEV).to(dtype).t()))
    assert not params[-1].is_contiguous()
    opt = torch.optim.SGD(params, lr=0.7, momentum=momentum, nesterov=nesterov)
    backup, comm = _FlatBuckets(params, None, False), _FlatBuckets(params, None, False)
    backup.copy_from_params()
    fused = FusedOuterStep.maybe_create(params, backup, comm, opt)
    old = [p.detach().clone() for p in params]
    bufs = [None] * len(params)
    ulp = 2.0**-7 if dtype == torch.bfloat16 else 2.0**-22
    for _ in range(2):
        with torch.no_grad():
            for p in params:
                p.add_((torch.randn(p.shape, device=DEV) * 0.05).to(dtype))
        local = [p.detach().clone() for p in params]
        fused.compute_pseudogradients()
        for i, (p, q) in enumerate(zip(local, old)):
            assert torch.equal(comm.views[i], (p.float() - q.float()).to(dtype))
            assert torch.equal(params[i].detach(), p)
        fused.apply_outer_update()
        for i, p in enumerate(params):
            g = comm.views[i].float() if p.is_contiguous() else (local[i].float() - old[i].float()).to(dtype).float()
            bufs[i] = g if bufs[i] is None else momentum * bufs[i] + g
            step = g if momentum == 0 else (g + momentum * bufs[i] if nesterov else bufs[i])
            want = old[i].float() - 0.7 * step
            assert ((p.detach().float() - want).abs() <= ulp * want.abs() + 1e-6).all()
            assert torch.equal(backup.views[i], p.detach())
            if momentum:
                got = opt.state[p]["momentum_buffer"]
                assert ((got - bufs[i]).abs() <= 2.0**-22 * (bufs[i].abs() + g.abs())).all()
                bufs[i] = got.clone()
            old[i] = p.detach().clone()


@pytest.mark.parametrize("shape", [(8, 6), (48,), (7, 8), (5, 8)])
def test_outer_step_refuses_a_parameter_of_another_shape(shape):
    """The buckets are laid out once: a weight that was replaced by one of another shape, larger, smaller or of the same size,
    raises as the copies between parameters and buckets do, and the buckets' other parts keep their values."""
    from torchft_b200.local_sgd import _FlatBuckets
    from torchft_b200.ops.outer_step import FusedOuterStep

    params = [torch.nn.Parameter(torch.randn(s, device=DEV)) for s in ((6, 8), (16,))]
    opt = torch.optim.SGD(params, lr=0.7, momentum=0.9)
    backup, comm = _FlatBuckets(params, None, False), _FlatBuckets(params, None, False)
    backup.copy_from_params()
    comm.copy_from_params()
    fused = FusedOuterStep.maybe_create(params, backup, comm, opt)
    old = params[0].data
    params[0].data = torch.randn(shape, device=DEV)
    kept = [t.clone() for t in (comm.views[1], backup.views[0], backup.views[1])]
    with pytest.raises(RuntimeError):
        fused.compute_pseudogradients()
    assert all(torch.equal(a, b) for a, b in zip((comm.views[1], backup.views[0], backup.views[1]), kept))
    params[0].data = old
    fused.compute_pseudogradients()
    params[0].data = torch.randn(shape, device=DEV)
    with pytest.raises(RuntimeError):
        fused.apply_outer_update()


@pytest.mark.parametrize("V", [8, 248, 256, 264, 2056, 32768, 32776, 49144, 49152, 49160, 65536, 65544, 128256, 262144, 262152])
def test_cross_entropy_around_the_sizes_of_a_row_in_registers(V):
    """Rows held in the registers of one warp and of blocks of up to 512 threads (up to 32768 columns), and rows read twice, in
    rounds of 16384 columns; targets at both ends of the row and around its halves and quarters, logits of -inf (also a whole
    first vector of them) and an ignored row."""
    from torchft_b200.ops.functional import cross_entropy

    torch.manual_seed(V)
    marks = sorted({t for t in (0, 7, 8, 255, V // 8, V // 4 - 1, V // 4, V // 2 - 1, V // 2, V // 2 + 3, V - 8, V - 1) if 0 <= t < V})
    targets = torch.tensor(marks + [-100], device=DEV)
    logits = bf16(len(targets), V, scale=3.0)
    kept = torch.zeros(len(targets), V, dtype=torch.bool, device=DEV)
    kept[torch.arange(len(marks)), targets[:-1]] = True
    logits[torch.rand(len(targets), V, device=DEV).lt(0.1) & ~kept] = float("-inf")
    if V > 8 and 0 not in marks[-3:]:
        logits[-3, :8] = float("-inf")
    x = logits.double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(x, targets, ignore_index=-100)
    ref.backward()
    work = logits.clone().requires_grad_()
    loss = cross_entropy(work, targets, ignore_index=-100)
    loss.backward()
    # fp32 sums of exponentials good to 2e-6 each, and one rounding to bf16 of every gradient
    assert abs(loss.item() - ref.item()) < 2e-5 * max(1.0, abs(ref.item()))
    assert ((work.grad.double() - x.grad).abs() <= 2.0**-8 * x.grad.abs() + 4e-6 / len(marks)).all()
    assert (work.grad[-1] == 0).all()


@pytest.mark.parametrize("V,bad", [(1000, 8), (1000, 992), (32768, 64), (32768, 32760), (49152, 8), (49152, 16384), (49152, 49144)])
def test_cross_entropy_keeps_nan(V, bad):
    """Vectors, threads and whole rounds of nothing but NaN (beside -inf in one row) do not vanish: the loss and the row's
    gradient are NaN, as for a NaN among finite logits, and the other rows keep their values."""
    from torchft_b200.ops.functional import cross_entropy

    torch.manual_seed(V)
    logits, targets = bf16(4, V, scale=2.0), torch.tensor([1, V - 1, 2, V - 1], device=DEV)
    clean = logits.clone()
    cross_entropy(clean, targets)
    logits[1, :bad] = float("nan")
    logits[3, :bad] = float("-inf")
    logits[3, bad // 2] = float("nan")
    loss = cross_entropy(logits, targets)
    assert torch.isnan(loss)
    assert torch.isnan(logits[1]).all() and torch.isnan(logits[3]).all()
    assert torch.equal(logits[::2], clean[::2])


@pytest.mark.parametrize("shift", [0.0, 1e3, -1e6, 1e30, -3e38, torch.finfo(torch.bfloat16).min])
@pytest.mark.parametrize("V", [1000, 32768, 49152])
def test_cross_entropy_of_large_logits(V, shift):
    """Loss and gradient depend on differences of logits, which bf16 values have exactly or with one rounding in fp32."""
    from torchft_b200.ops.functional import cross_entropy

    torch.manual_seed(V)
    logits = torch.full((4, V), shift, device=DEV).to(torch.bfloat16) if abs(shift) > 1e6 else (torch.randn(4, V, device=DEV) * 4 + shift).to(torch.bfloat16)
    targets = torch.tensor([0, 3, V // 2, V - 1], device=DEV)
    x = logits.double().requires_grad_()
    ref = torch.nn.functional.cross_entropy(x, targets)
    ref.backward()
    work = logits.clone().requires_grad_()
    loss = cross_entropy(work, targets)
    loss.backward()
    # fp32 sums of exponentials good to 2e-6 each, and one rounding to bf16 of every gradient
    assert abs(loss.item() - ref.item()) < 2e-5 * max(1.0, abs(ref.item()))
    assert ((work.grad.double() - x.grad).abs() <= 2.0**-8 * x.grad.abs() + 1e-6).all()


def test_adamw_of_many_tensors_equals_one_at_a_time():
    """Sizes around a vector and a block's chunk, an empty tensor, more tensors than one table holds: bit for bit the same."""
    from torchft_b200.ops.functional import adamw_multi_, adamw_step_

    torch.manual_seed(0)
    sizes = [1, 7, 8, 9, 4095, 4096, 4097, 4104, 3 * 4096 + 5, 0] + [5 + i for i in range(90)]
    kw = dict(lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3, grad_scale=0.5)
    ps, gs = [bf16(n) for n in sizes], [bf16(n) for n in sizes]
    ms, vs = [torch.randn(n, device=DEV) for n in sizes], [torch.rand(n, device=DEV) for n in sizes]
    single = [[t.clone() for t in ts] for ts in (ps, ms, vs)]
    adamw_multi_(ps, gs, ms, vs, **kw)
    for p, g, m, v in zip(single[0], gs, *single[1:]):
        adamw_step_(p, g, m, v, **kw)
    for got, want in zip((ps, ms, vs), single):
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    # and against the formula in 64 bits: fp32 moments to a few roundings, the parameter to one rounding of bf16
    n = 8 * 1000 + 5
    p, g, m, v = bf16(n), bf16(n), torch.randn(n, device=DEV), torch.rand(n, device=DEV)
    gd = g.double() * 0.5
    md, vd = 0.9 * m.double() + 0.1 * gd, 0.95 * v.double() + 0.05 * gd * gd
    want = p.double() * (1 - 3e-4 * 0.1) - 3e-4 * (md / (1 - 0.9**3)) / ((vd / (1 - 0.95**3)).sqrt() + 1e-8)
    m_old = m.clone()
    adamw_multi_([p], [g], [m], [v], **kw)
    # (1 - beta in fp32 is good to 2.4e-7)
    assert ((m - md).abs() <= 2.0**-21 * (m_old.abs() + gd.abs())).all() and ((v - vd).abs() <= 2.0**-21 * vd).all()
    assert ((p - want).abs() <= 2.0**-8 * want.abs() + 1e-6).all()


def test_adamw_of_parameters_that_share_memory():
    """One parameter listed twice, two that are the same memory, two that overlap: the updates follow one another, as one call
    for each would have them."""
    from torchft_b200.ops.functional import adamw_multi_, adamw_step_

    torch.manual_seed(0)
    kw = dict(lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3)
    base = bf16(200_000)
    before = base.clone()
    spans = [(0, 100_000), (100_000, 150_000), (0, 100_000), (0, 100_000), (99_992, 100_008), (150_000, 200_000)]
    gs = [bf16(b - a) for a, b in spans]
    ms, vs = [torch.randn(b - a, device=DEV) for a, b in spans], [torch.rand(b - a, device=DEV) for a, b in spans]
    ms[2], vs[2] = ms[0], vs[0]  # the first one again
    want_m, want_v = [m.clone() for m in ms], [v.clone() for v in vs]
    want_m[2], want_v[2] = want_m[0], want_v[0]
    adamw_multi_([base[a:b] for a, b in spans], gs, ms, vs, **kw)
    for (a, b), g, m, v in zip(spans, gs, want_m, want_v):
        adamw_step_(before[a:b], g, m, v, **kw)
    assert torch.equal(base, before)
    assert all(torch.equal(x, y) for x, y in zip(ms + vs, want_m + want_v))


@pytest.mark.parametrize("a_k,b_k", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("shape", [(1, 8, 2048), (256, 256, 2045 * 8), (257, 264, 2112), (1013, 2048, 5464), (300, 4600, 4104), (9471, 8, 2056)])
def test_gemm_with_a_divided_contraction(shape, a_k, b_k):
    """One tile in sixteen parts, ragged tiles, a last part shorter than the others, a contraction that ends inside a k-block,
    and 36 and 37 tiles, the most that are divided (on 74 CTA pairs)."""
    from torchft_b200.ops import _lib
    from torchft_b200.ops.gemm import gemm

    M, N, K = shape
    if not a_k:
        M += -M % 8  # the row stride of the transposed operand
    torch.manual_seed(K)
    a = bf16(M, K) if a_k else bf16(K, M)
    b = bf16(N, K) if b_k else bf16(K, N)
    ref = (a.double() if a_k else a.double().t()) @ (b.double().t() if b_k else b.double())
    kw = dict(a_kmajor=a_k, b_kmajor=b_k)
    assert _lib.lib().tft_gemm2_workspace(M, N, K) > 0
    out32 = gemm(a, b, out_dtype=torch.float32, **kw)
    whole = gemm(a, b, out_dtype=torch.float32, impl="single", **kw)
    # The tensor core drops what falls below the last bit of the running fp32 sum, up to 2^-23 of it in each of K / 16 steps,
    # so shorter parts can only come closer to the exact sum (a tenth allowed for the draw).
    assert norm_err(out32.double(), ref) < 1.1 * norm_err(whole.double(), ref) + 1e-8 < K / 16 * 2.0**-23
    out = gemm(a, b, **kw)
    assert torch.equal(out, out32.to(torch.bfloat16))
    acc = bf16(M, N)
    want = (out32 + acc.float()).to(torch.bfloat16)
    gemm(a, b, acc, accumulate=True, **kw)
    assert torch.equal(acc, want)
    wide = torch.zeros(M, N + 8, device=DEV, dtype=torch.bfloat16)
    gemm(a, b, wide[:, :N], **kw)
    assert torch.equal(wide[:, :N], out) and (wide[:, N:] == 0).all()
    _lib.check_status("gemm")
