"""Bandwidth-bound fused kernels vs plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def test_rms_norm_fwd_bwd():
    from paddle_b200.ops import native
    torch.manual_seed(0)
    x = torch.randn(37, 4096, device="cuda").to(BF)
    res = torch.randn(37, 4096, device="cuda").to(BF)
    w = (1 + 0.1 * torch.randn(4096, device="cuda")).to(BF)
    y, inv, res_out = native.rms_norm_fwd(x, w, 1e-5, residual=res, want_residual_out=True)
    s = (x.float() + res.float()).to(BF).float()
    r = torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-5)
    ref = s * r * w.float()
    assert torch.allclose(res_out.float(), s)
    assert torch.allclose(y.float(), ref, rtol=2e-2, atol=2e-2)
    assert torch.allclose(inv, r.squeeze(-1), rtol=1e-4, atol=1e-5)
    # backward against autograd
    xs = s.clone().requires_grad_(True)
    wf = w.float().clone().requires_grad_(True)
    dy = torch.randn(37, 4096, device="cuda").to(BF)
    (xs * torch.rsqrt(xs.pow(2).mean(-1, keepdim=True) + 1e-5) * wf).backward(dy.float())
    dx, dw = native.rms_norm_bwd(dy, res_out, w, inv)
    assert torch.allclose(dx.float(), xs.grad, rtol=3e-2, atol=3e-2)
    assert torch.allclose(dw, wf.grad, rtol=2e-2, atol=5e-2)


def test_layer_norm_fwd_bwd():
    from paddle_b200.ops import native
    torch.manual_seed(1)
    x = torch.randn(65, 1024, device="cuda").to(BF)
    w = (1 + 0.1 * torch.randn(1024, device="cuda"))
    b = 0.1 * torch.randn(1024, device="cuda")
    y, mean, rstd = native.layer_norm_fwd(x, w, b, 1e-5)
    xf = x.float().requires_grad_(True)
    wf, bf = w.clone().requires_grad_(True), b.clone().requires_grad_(True)
    ref = torch.nn.functional.layer_norm(xf, (1024,), wf, bf, 1e-5)
    assert torch.allclose(y.float(), ref, rtol=2e-2, atol=2e-2)
    dy = torch.randn(65, 1024, device="cuda").to(BF)
    ref.backward(dy.float())
    dx, dw, db = native.layer_norm_bwd(dy, x, w, mean, rstd)
    assert torch.allclose(dx.float(), xf.grad, rtol=3e-2, atol=3e-2)
    assert torch.allclose(dw, wf.grad, rtol=2e-2, atol=5e-2)
    assert torch.allclose(db, bf.grad, rtol=2e-2, atol=5e-2)


@pytest.mark.parametrize("half_style", [True, False])
def test_rope(half_style):
    from paddle_b200.ops import native
    torch.manual_seed(2)
    B, S, H, D = 2, 48, 4, 128
    x = torch.randn(B, S, H, D, device="cuda").to(BF)
    inv_freq = 1.0 / (10000 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    ang = torch.arange(S, device="cuda").float()[:, None] * inv_freq[None]
    if half_style:
        cos, sin = torch.cat([ang.cos(), ang.cos()], -1), torch.cat([ang.sin(), ang.sin()], -1)
    else:
        cos, sin = ang.cos().repeat_interleave(2, -1), ang.sin().repeat_interleave(2, -1)
    out = native.rope(x, cos.contiguous(), sin.contiguous(), half_style=half_style)
    xf = x.float()
    if half_style:
        rot = torch.cat([-xf[..., D // 2:], xf[..., :D // 2]], -1)
    else:
        rot = torch.stack([-xf[..., 1::2], xf[..., 0::2]], -1).reshape(xf.shape)
    ref = xf * cos[None, :, None, :] + rot * sin[None, :, None, :]
    assert torch.allclose(out.float(), ref, rtol=2e-2, atol=2e-2)
    back = native.rope(out, cos.contiguous(), sin.contiguous(), half_style=half_style, backward=True)
    assert torch.allclose(back.float(), xf, rtol=3e-2, atol=3e-2)


def test_swiglu():
    from paddle_b200.ops import native
    torch.manual_seed(3)
    x = torch.randn(33, 2 * 1376, device="cuda").to(BF)
    out = native.swiglu_fwd(x)
    a, b = x.float().chunk(2, -1)
    a.requires_grad_(True); b.requires_grad_(True)
    ref = torch.nn.functional.silu(a) * b
    assert torch.allclose(out.float(), ref, rtol=2e-2, atol=2e-2)
    do = torch.randn_like(out)
    ref.backward(do.float())
    dx, _ = native.swiglu_bwd(x, None, do)
    assert torch.allclose(dx.float(), torch.cat([a.grad, b.grad], -1), rtol=3e-2, atol=3e-2)
    o2 = native.swiglu_fwd(x[:, :1376].contiguous(), x[:, 1376:].contiguous())
    assert torch.equal(o2, out)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_softmax_ce(dtype):
    from paddle_b200.ops import native
    torch.manual_seed(4)
    T, V = 77, 32000
    logits = (torch.randn(T, V, device="cuda") * 3).to(dtype)
    labels = torch.randint(0, V, (T,), device="cuda")
    labels[5] = -100
    mx, sm, tg, loss = native.ce_stats(logits, labels)
    lf = logits.float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lf, labels, reduction="none", ignore_index=-100)
    assert torch.allclose(loss, ref, rtol=1e-3, atol=1e-3)
    dl = torch.rand(T, device="cuda")
    ref.backward(dl)
    lse = mx + sm.log()
    dlog = native.ce_bwd(logits, labels, lse, dl)
    tol = 2e-2 if dtype == torch.bfloat16 else 1e-4
    assert torch.allclose(dlog.float(), lf.grad, rtol=tol, atol=tol * 0.1)
    # vocab-parallel partial statistics combine to the same loss
    half = V // 2
    parts = [native.ce_stats(logits[:, i * half:(i + 1) * half].contiguous(), labels, vocab_start=i * half,
                             want_loss=False) for i in range(2)]
    gm = torch.maximum(parts[0][0], parts[1][0])
    gs = sum(p[1] * torch.exp(p[0] - gm) for p in parts)
    tgt = parts[0][2] + parts[1][2]
    l2 = torch.where(labels == -100, torch.zeros_like(gm), gs.log() + gm - tgt)
    assert torch.allclose(l2, ref.detach(), rtol=1e-3, atol=1e-3)


def test_embedding():
    from paddle_b200.ops import native
    torch.manual_seed(5)
    V, H = 1000, 256
    table = torch.randn(V, H, device="cuda").to(BF)
    ids = torch.randint(0, V, (4, 37), device="cuda")
    out = native.embedding_fwd(ids, table)
    assert torch.equal(out, table[ids])
    # sharded: rows outside the shard give zeros
    out2 = native.embedding_fwd(ids, table[500:], vocab_start=500)
    ref2 = torch.where((ids >= 500)[..., None], table[ids], torch.zeros_like(out))
    assert torch.equal(out2, ref2)
    dout = torch.randn(4, 37, H, device="cuda").to(BF)
    dt = torch.zeros(V, H, device="cuda")
    native.embedding_bwd(ids, dout, dt)
    ref = torch.zeros(V, H, device="cuda").index_add_(0, ids.reshape(-1), dout.reshape(-1, H).float())
    assert torch.allclose(dt, ref, rtol=1e-4, atol=1e-4)


def test_accumulate_and_add():
    from paddle_b200.ops import native
    a = torch.randn(100003, device="cuda").to(BF)[:100000]
    acc = torch.ones(100000, device="cuda")
    native.accumulate_into_f32(a, acc)
    assert torch.allclose(acc, 1 + a.float())
    b = torch.randn(100000, device="cuda").to(BF)
    assert torch.allclose(native.add_bf16(a.contiguous(), b).float(), (a.float() + b.float()).to(BF).float())


@pytest.mark.parametrize("act", [None, "relu", "gelu", "silu"])
def test_gemm_bias_activation_epilogue(act):
    """act(x @ W + b) from the GEMM epilogue against fp32."""
    import paddle_b200 as paddle
    from paddle_b200.ops import _lib
    torch.manual_seed(3)
    x = (torch.randn(3, 100, 256, device="cuda") * 0.5).bfloat16()
    w = (torch.randn(256, 520, device="cuda") * 0.1).bfloat16()
    b = torch.randn(520, device="cuda").bfloat16()
    with torch.no_grad():
        y = paddle.incubate.nn.functional.fused_linear_activation(x, w, b, activation=act)
    _lib.check_status()
    ref = x.float() @ w.float() + b.float()
    ref = {None: lambda t: t, "relu": torch.relu, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu}[act](ref)
    assert (y.float() - ref).abs().max().item() < 3e-2 * ref.abs().max().item() + 2e-2
    # training path: bias in the epilogue, gradients through autograd
    xg, wg, bg = x.clone().requires_grad_(True), w.clone().requires_grad_(True), b.clone().requires_grad_(True)
    out = paddle.nn.functional.linear(xg, wg, bg)
    out.float().pow(2).sum().backward()
    xf, wf, bf = (t.detach().float().requires_grad_(True) for t in (x, w, b))
    (xf @ wf + bf).bfloat16().float().pow(2).sum().backward()
    for a, r in ((xg.grad, xf.grad), (wg.grad, wf.grad), (bg.grad, bf.grad)):
        assert (a.float() - r).abs().max().item() < 3e-2 * r.abs().max().item() + 1e-1


def test_gemm_swiglu_epilogue():
    import paddle_b200 as paddle
    from paddle_b200.ops import _lib
    IF = paddle.incubate.nn.functional
    torch.manual_seed(4)
    x = (torch.randn(300, 512, device="cuda") * 0.5).bfloat16()
    gate = (torch.randn(512, 1376, device="cuda") * 0.05).bfloat16()
    up = (torch.randn(512, 1376, device="cuda") * 0.05).bfloat16()
    y = IF.fused_linear_swiglu_interleaved(x, IF.interleave_gate_up(gate, up))
    _lib.check_status()
    ref = torch.nn.functional.silu(x.float() @ gate.float()) * (x.float() @ up.float())
    assert list(y.shape) == [300, 1376]
    assert (y.float() - ref).abs().max().item() < 3e-2 * ref.abs().max().item() + 1e-2


@pytest.mark.parametrize("act", ["gelu", "relu", "silu", "swiglu", "geglu"])
def test_bias_act_kernel(act):
    import paddle_b200 as paddle
    torch.manual_seed(5)
    x = torch.randn(7, 33, 512, device="cuda").bfloat16()
    b = torch.randn(512, device="cuda").bfloat16()
    with torch.no_grad():
        y = paddle.incubate.nn.functional.fused_bias_act(x, b, act_method=act)
    h = x.float() + b.float()
    if act in ("swiglu", "geglu"):
        g, u = h.chunk(2, -1)
        ref = (torch.nn.functional.silu(g) if act == "swiglu" else torch.nn.functional.gelu(g)) * u
    else:
        ref = getattr(torch.nn.functional, act)(h)
    assert list(y.shape) == list(ref.shape)
    assert (y.float() - ref).abs().max().item() < 2e-2 * ref.abs().max().item() + 1e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_dropout_add_philox(dtype):
    """Keep rate, scaling, reproducibility from (seed, offset), backward mask = forward mask, generator advance."""
    import paddle_b200 as paddle
    from paddle_b200.ops import functional as K
    n, p = 1 << 20, 0.3
    x = torch.ones(n + 5, device="cuda", dtype=dtype).requires_grad_(True)
    y = torch.full((n + 5,), 2.0, device="cuda", dtype=dtype).requires_grad_(True)
    out, (seed, off) = K.dropout_add(x, y, p)
    kept = (out.float() - 2.0) > 0
    assert abs(kept.float().mean().item() - (1 - p)) < 5e-3
    assert torch.allclose(out.float()[kept], torch.tensor(2.0 + 1 / (1 - p), device="cuda"), atol=2e-2)
    out.sum().backward()
    assert torch.equal(x.grad.float() > 0, kept) and torch.all(y.grad.float() == 1)
    out2, _ = K.dropout_add(x.detach(), y.detach(), p, seed_offset=(seed, off))
    assert torch.equal(out2, out.detach())
    out3 = paddle.incubate.nn.functional.fused_dropout_add(x.detach(), y.detach(), p)      # generator moved on
    assert not torch.equal(out3, out.detach())
    paddle.seed(123)
    a = paddle.nn.functional.dropout(x.detach(), p)
    paddle.seed(123)
    b = paddle.nn.functional.dropout(x.detach(), p)
    assert torch.equal(a, b)


@pytest.mark.parametrize("rows,N", [(1, 8), (33, 72), (63, 64), (1000, 11008), (8191, 520), (300, 4096)])
def test_row_sum(rows, N):
    from paddle_b200.ops import native
    torch.manual_seed(rows)
    x = torch.randn(rows, N + 8, device="cuda").bfloat16()[:, :N]
    got, ref = native.row_sum(x), x.double().sum(0)
    # fp32 sums of `rows` values of size 4, one rounding to bf16
    assert (got.double() - ref).abs().le(ref.abs() * 2 ** -8 + rows * 4 * 2 ** -22).all()


@pytest.mark.parametrize("rows,H", [(1, 8), (5, 2048), (297, 2056), (300, 4096), (77, 6144), (650, 8192), (1000, 520)])
@pytest.mark.parametrize("add", [False, True])
def test_rms_norm_bwd_vectors_per_thread(rows, H, add):
    """Every number of vectors per thread with its edges, fewer and more rows than blocks, accumulation into dw."""
    from paddle_b200.ops import native
    torch.manual_seed(H + rows)
    x, dy, extra = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    inv = torch.rsqrt(x.float().pow(2).mean(-1) + 1e-5)
    acc = torch.randn(H, device="cuda")
    dx, dw = native.rms_norm_bwd(dy, x, w, inv, dx_add=extra if add else None, dw_out=acc.clone())
    xd, g, r = x.double(), dy.double() * w.double(), inv.double()[:, None]
    ref = r * (g - xd * (g * xd).sum(-1, keepdim=True) * r * r / H) + (extra.double() if add else 0)
    refw = acc.double() + (dy.double() * xd * r).sum(0)
    assert (dx.double() - ref).abs().le(ref.abs() * 2 ** -8 + 1e-4).all()
    assert (dw.double() - refw).abs().max() <= 1e-5 * rows ** 0.5 * 10


@pytest.mark.parametrize("D,heads", [(32, 3), (64, 33), (96, 5), (128, 64), (256, 7)])
def test_rope_head_dims(D, heads):
    """Head dims of the per-token kernel and one (96) of the general kernel, both directions, positions given and not."""
    from paddle_b200.ops import functional as K
    from paddle_b200.ops import native
    torch.manual_seed(D)
    x = torch.randn(2, 37, heads + 2, D, device="cuda").bfloat16()[:, :, :heads]
    cos, sin = K.rope_tables(64, D, 10000.0, torch.device("cuda"), True)
    pid = torch.randint(0, 64, (2, 37), device="cuda")
    for p in (None, pid):
        for back in (False, True):
            got = native.rope(x, cos, sin, p, half_style=True, backward=back)
            ref = K._rope_torch(x, cos, -sin if back else sin, p, True)
            assert (got.float() - ref.float()).abs().max() <= ref.float().abs().max() * 2 ** -7


def test_shape_keeping_operators_keep_the_distribution():
    """Norms and dropout of a distributed tensor are distributed as their input is."""
    import paddle_b200 as paddle
    import paddle_b200.distributed as dist
    from paddle_b200.ops import functional as K
    paddle.set_device("gpu:0")
    mesh = dist.ProcessMesh([0], dim_names=["x"])

    def make(*shape):
        t = dist.shard_tensor(paddle.to_tensor(torch.randn(shape, device="cuda").bfloat16()), mesh, [dist.Replicate()])
        t.stop_gradient = False
        return t
    x, w = make(2, 8, 256), make(256)
    outs = [K.rms_norm(x, w), *K.rms_norm(x, w, residual=x), K.layer_norm(x, 256, w, w), K.dropout_add(x, x, 0.1)[0]]
    for o in outs:
        assert o.is_dist() and o.process_mesh == mesh and o.placements == [dist.Replicate()] and o.shape == [2, 8, 256]
    sum(o.sum() for o in outs).backward()
    assert x.grad is not None and torch.isfinite(x.grad.float()).all()
    assert not K.rms_norm(paddle.to_tensor(torch.randn(4, 256, device="cuda").bfloat16()), w).is_dist()


@pytest.mark.parametrize("M,N,K,act", [(100, 256, 128, None), (129, 264, 200, None), (300, 520, 256, "silu"), (2331, 640, 512, None)])
def test_gemm_residual_epilogue(M, N, K, act):
    """act(x W + b) + residual from the GEMM epilogue, edges of rows and columns, a residual with its own row stride."""
    from paddle_b200.ops import _lib, native
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, b, wide = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (K, N), (N,), (M, N + 16)))
    res = wide[:, 8:N + 8]
    for bias in (None, b):
        y = native.gemm_epilogue(x, w, bias, act, residual=res)
        _lib.check_status()
        h = x.float() @ w.float() + (0 if bias is None else bias.float())
        ref = (torch.nn.functional.silu(h) if act else h) + res.float()
        # one rounding to bf16; sums of K products in fp32 (both sides), 2^-6 for the fast exponential of the activation
        assert ((y.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-3 + (2 ** -6 if act else 0)).all()


@pytest.mark.parametrize("M,N,K,width", [(2331, 5120, 512, 256), (2048, 2600, 8200, 512), (2048, 2840, 8200, 512)])
@pytest.mark.parametrize("with_bias", [False, True])
@pytest.mark.parametrize("round_product", [False, True])
def test_gemm_residual_epilogue_of_wide_tiles(M, N, K, width, with_bias, round_product):
    """Tiles of 256 columns, and of 512 whose last one has no second half or a partly filled one; a residual with its own row stride."""
    from paddle_b200.ops import _lib, native
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _lib.kernels().pd_gemm_2cta_tile_n_at(M, N, K, 1, 0) == width
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, b, wide = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (K, N), (N,), (M, N + 16)))
    res = wide[:, 8:N + 8]
    y = native.gemm_epilogue(x, w, b if with_bias else None, residual=res, round_product=round_product)
    _lib.check_status()
    h = x.double() @ w.double() + (b.double() if with_bias else 0)
    # the tensor cores cut off when they add: K / 16 steps lose up to 2^-23 of a running sum below 5 sqrt(K); bias and residual are added
    # in fp32; one rounding to bf16, with round_product one of the product before it
    tol = K / 16 * 5 * K ** 0.5 * 2 ** -23 + 2 ** -22 * h.abs() + (2 ** -8 * h.abs() if round_product else 0)
    ref = h + res.double()
    assert ((y.double() - ref).abs() <= 2 ** -8 * (ref.abs() + tol) + tol).all()


@pytest.mark.parametrize("tokens", [1, 295, 296, 1203])
@pytest.mark.parametrize("heads,D", [(1, 128), (5, 128), (33, 128), (9, 64), (3, 2048)])
def test_rope_whole_blocks_and_teams(tokens, heads, D):
    """Few tokens (a block each) and many (teams of threads), heads that do not divide among them, in place on a strided view, both
    directions."""
    from paddle_b200.ops import _lib, native
    g = torch.Generator(device="cuda").manual_seed(tokens + heads)
    buf = torch.randn(tokens, heads + 2, D, device="cuda", generator=g).bfloat16()
    x = buf[:, :heads]
    cos, sin = (torch.randn(tokens, D, device="cuda", generator=g) for _ in range(2))
    xf, h, kept = x.float().clone(), D // 2, buf[:, heads:].clone()
    for backward in (False, True):
        sg = -sin if backward else sin
        ref = torch.cat([xf[..., :h] * cos[:, None, :h] - xf[..., h:] * sg[:, None, :h],
                         xf[..., h:] * cos[:, None, h:] + xf[..., :h] * sg[:, None, h:]], -1)
        y = native.rope(x.unsqueeze(0), cos, sin, backward=backward)[0]
        assert ((y.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5).all()       # fp32 products, one rounding to bf16
    native.rope(x.unsqueeze(0), cos, sin, out=x.unsqueeze(0), backward=True)
    _lib.check_status()
    assert torch.equal(x, y) and torch.equal(buf[:, heads:], kept)


@pytest.mark.parametrize("rows,H", [(297, 2048), (298, 2048), (297, 4096), (301, 5120), (297, 256 * 16)])
@pytest.mark.parametrize("with_residual", [False, True])
@pytest.mark.parametrize("wdtype", [torch.bfloat16, torch.float32])
def test_rms_norm_rows_of_few_warps(rows, H, with_residual, wdtype):
    """Row lengths that two or four warps share, just above the rows from which they are taken, the last block half empty."""
    from paddle_b200.ops import _lib, native
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    x, r = (torch.randn(rows, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).to(wdtype)
    y, inv, out = native.rms_norm_fwd(x, w, 1e-5, r if with_residual else None, with_residual)
    _lib.check_status()
    s = (x.float() + r.float()).bfloat16() if with_residual else x
    if with_residual:
        assert torch.equal(out, s)
    d = s.double()
    ri = torch.rsqrt(d.pow(2).mean(-1) + 1e-5)
    assert ((inv.double() - ri).abs() <= 1e-5 * ri).all()            # fp32 sums of H squares
    ref = d * ri[:, None] * w.double()
    assert ((y.double() - ref).abs() <= (2 ** -8 + 2e-5) * ref.abs()).all()


@pytest.mark.parametrize("M,N,K,width", [(129, 264, 200, 128), (2331, 5120, 512, 256), (2048, 2600, 8200, 512), (2048, 2840, 8200, 512)])
def test_projection_adds_the_residual_to_a_bf16_product(M, N, K, width):
    """The projections of prompt processing: the product in bf16, then the residual, in one kernel with every width of its tiles."""
    from types import SimpleNamespace
    from paddle_b200.incubate.nn import FusedMultiTransformer
    from paddle_b200.ops import _lib, native
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _lib.kernels().pd_gemm_2cta_tile_n_at(M, N, K, 1, 0) == width
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, res = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (K, N), (M, N)))
    got = FusedMultiTransformer._gemm(SimpleNamespace(_ws={"out": (1, None)}), "out", x, w, residual=res)
    _lib.check_status()
    assert torch.equal(got, native.add_bf16(native.gemm(x, w), res))


@pytest.mark.parametrize("rows,H", [(297, 2048), (300, 4096), (299, 5120)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_rms_norm_rows_are_added_up_lane_by_lane(rows, H, with_residual):
    """However many warps share a row, lane l adds up the vectors l, l + 32, ... one after the other and the lanes come last.  Rows in
    which that order shows: a large first element of a lane, which the small ones behind it cannot change."""
    from paddle_b200.ops import _lib, native
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(rows, H // 8, 8, device="cuda", generator=g)
    x[1::2] = 0
    x[1::2, :, 0::2] = 1.0                    # squares of 1, one in a pair
    x[1::2, :32, 0] = 2.0 ** 12               # 2^24 + 1 is 2^24 in fp32
    x = x.reshape(rows, H).bfloat16()
    inv = native.rms_norm_fwd(x, torch.ones(H, device="cuda"), 1e-5, torch.zeros_like(x) if with_residual else None)[1]
    _lib.check_status()
    pairs = x.float().square().reshape(rows, H // 256, 32, 4, 2).sum(-1)       # squares of bf16 are exact, a pair rounds once
    lanes = torch.zeros(rows, 32, device="cuda")
    for k in range(H // 256):
        for j in range(4):
            lanes = lanes + pairs[:, k, :, j]
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, torch.arange(32, device="cuda") ^ o]
    ref = torch.rsqrt(lanes[:, 0].double() / H + 1e-5)
    # quotient and root in fp32; sums of warps that start from zero keep their H / 512 or more vectors of four ones: 2^-22 or more of the root
    off = ((inv.double() - ref) / ref).abs()
    assert off.max() <= 2.5 * 2 ** -23, off.max().item() * 2 ** 23
