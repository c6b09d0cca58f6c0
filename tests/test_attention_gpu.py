"""Flash attention kernels vs an fp32 PyTorch reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, causal, scale):
    qf, kf, vf = (t.float().transpose(1, 2) for t in (q, k, v))
    if kf.shape[1] != qf.shape[1]:
        rep = qf.shape[1] // kf.shape[1]
        kf, vf = kf.repeat_interleave(rep, 1), vf.repeat_interleave(rep, 1)
    s = qf @ kf.transpose(-1, -2) * scale
    if causal:
        Sq, Sk = s.shape[-2:]
        mask = torch.ones(Sq, Sk, dtype=torch.bool, device=s.device).tril(Sk - Sq)
        s = s.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(s, -1)
    return (torch.softmax(s, -1) @ vf).transpose(1, 2), lse


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 1, 1), (2, 256, 2, 2), (1, 384, 4, 2), (1, 200, 2, 1), (1, 1024, 2, 2)])
def test_flash_fwd(causal, B, S, Hq, Hkv):
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(S + Hq)
    q = torch.randn(B, S, Hq, 128, device="cuda").to(torch.bfloat16)
    k = torch.randn(B, S, Hkv, 128, device="cuda").to(torch.bfloat16)
    v = torch.randn(B, S, Hkv, 128, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)
    o, lse = attention.fwd(q, k, v, causal, scale)
    _lib.check_status()
    ro, rl = _ref(q, k, v, causal, scale)
    assert torch.allclose(lse, rl, rtol=1e-3, atol=2e-3), (lse - rl).abs().max()
    assert torch.allclose(o.float(), ro, rtol=2e-2, atol=2e-2), (o.float() - ro).abs().max()


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv", [(1, 1, 1, 1, 1), (1, 64, 65, 2, 1), (1, 129, 192, 2, 2), (1, 300, 100, 2, 2),
                                            (3, 257, 511, 32, 8), (7, 640, 640, 32, 32)])
def test_flash_fwd_steps_and_rescaling(causal, B, Sq, Sk, Hq, Hkv):
    """Edges of the 64-key steps and of the one- and two-tile forms (few / many blocks), with scores that grow along the keys
    so that the running maximum moves by more than 2^8 in many steps, the last one among them."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(Sq + Sk)
    ramp = torch.linspace(0, 1, Sk, device="cuda")[None, :, None, None]
    q = (torch.randn(B, Sq, Hq, 128, device="cuda") * 0.5 + 1.0).to(torch.bfloat16)
    k = (torch.randn(B, Sk, Hkv, 128, device="cuda") * 0.1 + ramp * 6.0).to(torch.bfloat16)
    v = torch.randn(B, Sk, Hkv, 128, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)
    o, lse = attention.fwd(q, k, v, causal, scale)
    _lib.check_status()
    ro, rl = _ref(q, k, v, causal, scale)
    ro = torch.nan_to_num(ro)                      # rows that see no key: zero output, log-sum-exp -inf
    live = torch.isfinite(rl)
    assert torch.equal(torch.isfinite(lse), live)
    assert torch.allclose(lse[live], rl[live], rtol=1e-3, atol=2e-3)
    # P and O are rounded to bf16 (2^-9 relative each); |v| stays below 6
    assert (o.float() - ro).abs().max() <= 6 * 2 ** -8 + 1e-3


def test_flash_fwd_packed_qkv_view():
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(0)
    B, S, H = 1, 512, 4
    qkv = torch.randn(B, S, 3 * H, 128, device="cuda").to(torch.bfloat16)
    q, k, v = qkv[:, :, :H], qkv[:, :, H:2 * H], qkv[:, :, 2 * H:]
    o, lse = attention.fwd(q, k, v, True, 0.088)
    _lib.check_status()
    ro, _ = _ref(q, k, v, True, 0.088)
    assert torch.allclose(o.float(), ro, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 128, 1, 1), (1, 256, 2, 2), (2, 384, 2, 1), (1, 200, 1, 1), (1, 1024, 2, 2)])
def test_flash_bwd(causal, B, S, Hq, Hkv):
    from paddle_b200.ops import _lib, attention
    if not hasattr(_lib.kernels(), "pd_flash_attn_bwd"):
        pytest.skip("backward kernel not built")
    torch.manual_seed(S * 3 + Hq)
    q = torch.randn(B, S, Hq, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    k = torch.randn(B, S, Hkv, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    v = torch.randn(B, S, Hkv, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    do = torch.randn(B, S, Hq, 128, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)
    o = attention.flash_attn_func(q, k, v, causal, scale)
    o.backward(do)
    _lib.check_status()
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ro, _ = _ref(qf, kf, vf, causal, scale)
    ro.backward(do.float())
    for name, a, b in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        err = (a.float() - b).abs().max().item()
        assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{name}: {err}"


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv", [(1, 1, 1, 1, 1), (1, 65, 64, 4, 2), (1, 64, 193, 2, 2), (2, 321, 257, 4, 1), (7, 640, 640, 32, 8)])
def test_flash_bwd_subtile_edges_and_head_chunks(causal, B, Sq, Sk, Hq, Hkv):
    """Edges of the 64-row query sub-tiles and 128-row key tiles, keys seen by no query, more queries than keys, and enough
    heads for several chunks of the block order."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(Sq + 3 * Sk)
    q, do = (torch.randn(B, Sq, Hq, 128, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, Sk, Hkv, 128, device="cuda").to(torch.bfloat16) for _ in range(2))
    scale = 1 / math.sqrt(128)
    qn, kn, vn = (t.clone().requires_grad_(True) for t in (q, k, v))
    attention.flash_attn_func(qn, kn, vn, causal, scale).backward(do)
    _lib.check_status()
    for b in range(B):
        qf, kf, vf = (t[b:b + 1].float().requires_grad_(True) for t in (q, k, v))
        blind = max(0, Sq - Sk) if causal else 0          # the first rows see no key: no gradient through them
        ro, _ = _ref(qf[:, blind:], kf, vf, causal, scale)
        ro.backward(do[b:b + 1, blind:].float())
        for name, got, want in (("dq", qn.grad, qf.grad), ("dk", kn.grad, kf.grad), ("dv", vn.grad, vf.grad)):
            # P and dS enter the products in bf16: 2^-8 of the largest value, and the result is rounded once more
            err = (got[b:b + 1].float() - want).abs().max().item()
            assert err <= 2 ** -6 * want.abs().max().item() + 1e-2, f"{name}: {err}"


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,S,Hq,Hkv,parts", [(1, 200, 4, 1, 4), (2, 321, 6, 1, 3), (1, 384, 8, 2, 2), (2, 640, 8, 8, 1)])
def test_flash_bwd_shared_key_tiles(causal, B, S, Hq, Hkv, parts, monkeypatch):
    """Several CTAs adding to the fp32 dK / dV of one key tile give what one CTA gives, for every split of the group; dk / dv go
    into views of a packed buffer.  The size rule itself splits when there are few kv heads and leaves full grids alone."""
    from paddle_b200.ops import _lib, attention
    k_ = _lib.kernels()
    assert k_.pd_flash_attn_bwd_parts(1, 1024, 1024, 8, 2, 0) == 4
    assert k_.pd_flash_attn_bwd_parts(1, 4096, 4096, 32, 32, 0) == 1 and k_.pd_flash_attn_bwd_parts(8, 4096, 4096, 32, 8, 1) == 1
    torch.manual_seed(S + Hq)
    qkv = torch.randn(B, S, Hq + 2 * Hkv, 128, device="cuda").to(torch.bfloat16)
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    do = torch.randn(B, S, Hq, 128, device="cuda").to(torch.bfloat16)
    o, lse = attention.fwd(q, k, v, causal, 0.088)
    got = []

    class Forced:
        def __init__(self, n):
            self.n = n

        def __getattr__(self, name):
            return (lambda *a: self.n) if name == "pd_flash_attn_bwd_parts" else getattr(k_, name)
    for n in (1, parts):
        monkeypatch.setattr(_lib, "kernels", lambda n=n: Forced(n))
        d = torch.full_like(qkv, float("nan"))
        attention.bwd(do, q, k, v, o, lse, causal, 0.088, dq=d[:, :, :Hq], dk=d[:, :, Hq:Hq + Hkv], dv=d[:, :, Hq + Hkv:])
        got.append(d.float())
    monkeypatch.undo()
    _lib.check_status()
    # the same fp32 terms in another order: one rounding to bf16 apart
    assert (got[0] - got[1]).abs().le(got[0].abs() * 2 ** -7 + 1e-3).all()


@pytest.mark.parametrize("S,Hq,Hkv", [(64, 1, 1), (200, 4, 4), (333, 8, 2)])
def test_flash_bwd_rounds_the_scaled_score_gradient(S, Hq, Hkv):
    """dS enters the products with K and Q as bf16 after the softmax scale: with everything else in 64 bits, dQ and dK come out as the
    same bf16 values but for the few whose exact value lies within fp32 rounding of a tie (of dS or of the result)."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(S)
    q, k, v, do = (torch.randn(1, S, h, 128, device="cuda").to(torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    scale = 1 / math.sqrt(128)
    o, lse = attention.fwd(q, k, v, True, scale)
    dq, dk, _ = attention.bwd(do, q, k, v, o, lse, True, scale)
    _lib.check_status()
    qd, dod, od = (t[0].double().transpose(0, 1) for t in (q, do, o))
    kd, vd = (t[0].double().transpose(0, 1).repeat_interleave(Hq // Hkv, 0) for t in (k, v))
    s = (qd @ kd.mT * scale).masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    ds = torch.softmax(s, -1) * (dod @ vd.mT - (dod * od).sum(-1, keepdim=True)) * scale
    ds = ds.to(torch.bfloat16).double()
    want_q = (ds @ kd).transpose(0, 1).to(torch.bfloat16)
    want_k = (ds.mT @ qd).view(Hkv, Hq // Hkv, S, 128).sum(1).transpose(0, 1).to(torch.bfloat16)
    for name, got, want in (("dq", dq[0], want_q), ("dk", dk[0], want_k)):
        # a tie in dS (2^-14 of them) moves up to 128 results of S terms by 2^-9 of one term: below 1 % of the results change
        assert (got == want).float().mean().item() > 0.97, (name, (got == want).float().mean().item())


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1024, 8, 2), (2, 1999, 32, 8), (1, 777, 40, 5)])
def test_flash_bwd_dk_dv_repeat_bit_for_bit(causal, B, S, Hq, Hkv):
    """dK / dV come out the same on every run, also where several CTAs share a key tile."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(S)
    q, k, v, do = (torch.randn(B, S, h, 128, device="cuda").to(torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    o, lse = attention.fwd(q, k, v, causal, 0.088)
    _, dk, dv = attention.bwd(do, q, k, v, o, lse, causal, 0.088)
    for _ in range(8):
        _, dk2, dv2 = attention.bwd(do, q, k, v, o, lse, causal, 0.088)
        assert torch.equal(dk, dk2) and torch.equal(dv, dv2)
    _lib.check_status()


@pytest.mark.parametrize("parts", [1, 2, 4])
def test_flash_bwd_shared_key_tile_that_no_query_sees(parts, monkeypatch):
    """Keys hidden from all queries by a column-sparse mask: their CTAs have nothing to walk over and leave zeros, whatever their
    scratch held."""
    from paddle_b200.ops import _lib, attention
    B, S, Hq, Hkv = 1, 300, 4, 1
    torch.manual_seed(parts)
    q, k, v, do = (torch.randn(B, S, h, 128, device="cuda").to(torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    idx = torch.full((B, 1, S, 1), S, dtype=torch.int32, device="cuda")
    idx[:, :, 128:256] = 0                             # the second key tile
    mask = attention.normalize_flashmask(idx, True, S)
    o, lse = attention.fwd(q, k, v, True, 0.088, mask)
    k_ = _lib.kernels()

    class Forced:
        def __getattr__(self, name):
            return (lambda *a: parts) if name == "pd_flash_attn_bwd_parts" else getattr(k_, name)
    monkeypatch.setattr(_lib, "kernels", lambda: Forced())
    junk = torch.full((8 * B * S * Hkv * 128,), float("nan"), device="cuda")
    del junk
    dq, dk, dv = attention.bwd(do, q, k, v, o, lse, True, 0.088, mask=mask)
    monkeypatch.undo()
    _lib.check_status()
    assert all(torch.isfinite(t.float()).all() for t in (dq, dk, dv))
    assert dk[:, 128:256].abs().max().item() == 0 and dv[:, 128:256].abs().max().item() == 0
    assert dk[:, :128].abs().max().item() > 0 and dv[:, 256:].abs().max().item() > 0


@pytest.mark.parametrize("Sq,Sk", [(200, 200), (64, 1), (300, 129)])
def test_flash_bwd_padded_keys_and_low_scores(Sq, Sk):
    """Scores far below zero against a key tile that is not full: the tile's padded rows must not reach dQ through an overflow."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(Sq + Sk)
    q = (torch.randn(1, Sq, 4, 128, device="cuda") * 0.02 + 3.0).to(torch.bfloat16).requires_grad_(True)
    k = (torch.randn(1, Sk, 2, 128, device="cuda") * 0.02 - 3.0).to(torch.bfloat16).requires_grad_(True)
    v = torch.randn(1, Sk, 2, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    do = torch.randn(1, Sq, 4, 128, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)                      # every score is near -9 * 128 * scale = -102
    attention.flash_attn_func(q, k, v, False, scale).backward(do)
    _lib.check_status()
    qf, kf, vf = (t.detach().double().requires_grad_(True) for t in (q, k, v))
    rep = [t.repeat_interleave(2, 2).transpose(1, 2) for t in (kf, vf)]
    (torch.softmax(qf.transpose(1, 2) @ rep[0].mT * scale, -1) @ rep[1]).transpose(1, 2).backward(do.double())
    for name, got, want in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        # P and dS enter the products in bf16 (2^-9 each) and the sums are of terms of one sign or cancel: |dS| sums to about 2 |dP|,
        # |k|, |q| = 3, so the rounding of dS alone gives up to 2^-8 * 2 * 12 * 3 * scale for dq and Sq / Sk times that for dk
        bound = {"dq": 0.03, "dk": 0.03 * max(1, 2 * Sq / Sk), "dv": 2 ** -6 * want.abs().max().item()}[name]
        assert torch.isfinite(got.float()).all(), name
        assert (got.double() - want).abs().max().item() <= bound + 1e-2, name


@pytest.mark.parametrize("S", [200, 100])
def test_flashmask_rows_that_see_no_key(S):
    """Query rows for which every key is masked, without a causal mask and with a key tile that is not full: zero output, zero
    gradient, nothing passed on to the other rows."""
    import paddle_b200 as paddle
    from paddle_b200.ops import _lib
    torch.manual_seed(S)
    q, k, v = (torch.randn(2, S, h, 128, device="cuda").to(torch.bfloat16).requires_grad_(True) for h in (4, 2, 2))
    do = torch.randn(2, S, 4, 128, device="cuda").to(torch.bfloat16)
    # rows [30, 45) and [S - 20, S) see nothing
    cols = torch.tensor([30, 45, S - 20, S], dtype=torch.int32, device="cuda")
    idx = torch.stack([cols[2], cols[3], cols[0], cols[1]]).view(1, 1, 1, 4).expand(2, 1, S, 4).contiguous()
    o = paddle.nn.functional.flashmask_attention(q, k, v, idx, causal=False)
    o.backward(do)
    _lib.check_status()
    masked = _dense_from_flashmask(idx, S, S, False)
    dead = masked.all(-1)[0, 0]
    assert int(dead.sum()) == 35
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ro = _masked_ref(qf, kf, vf, masked, 1 / math.sqrt(128))
    ro.backward(do.float())
    assert (o.float() - ro).abs().max().item() < 3e-2
    assert q.grad[:, dead].float().abs().max().item() == 0
    for nm, a, b in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        err = (a.float() - b).abs().max().item()
        assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{nm}: {err}"


def _dense_from_flashmask(idx, sq, sk, causal):
    from paddle_b200.nn.functional.flash_attention import _flashmask_dense
    return _flashmask_dense(idx, sq, sk, causal, idx.device)


def _masked_ref(q, k, v, masked, scale):
    """fp32 attention with a boolean [B, Hm, Sq, Sk] mask (True = hidden); rows with nothing visible give zeros."""
    qf, kf, vf = (t.float().transpose(1, 2) for t in (q, k, v))
    if kf.shape[1] != qf.shape[1]:
        rep = qf.shape[1] // kf.shape[1]
        kf, vf = kf.repeat_interleave(rep, 1), vf.repeat_interleave(rep, 1)
    s = (qf @ kf.transpose(-1, -2) * scale).masked_fill(masked, float("-inf"))
    dead = masked.all(-1, keepdim=True)
    p = torch.softmax(s.masked_fill(dead, 0.0), -1).masked_fill(dead, 0.0)
    return (p @ vf).transpose(1, 2)


def _flashmask_cases(S, device):
    g = torch.Generator(device="cpu").manual_seed(S)
    # causal document mask: three documents of uneven length
    cuts = sorted(torch.randint(1, S, (2,), generator=g).tolist())
    ends = torch.zeros(S, dtype=torch.int32)
    lo = 0
    for hi in cuts + [S]:
        ends[lo:hi] = hi
        lo = hi
    starts = torch.zeros(S, dtype=torch.int32)
    lo = 0
    for hi in cuts + [S]:
        starts[lo:hi] = lo
        lo = hi
    cols = torch.arange(S, dtype=torch.int32)
    yield "causal_document", True, ends.view(1, 1, S, 1)
    yield "causal_blockwise", True, torch.stack([(cols + S // 4).clamp(max=S), (cols + S // 2).clamp(max=S)], -1).view(1, 1, S, 2)
    yield "document", False, torch.stack([ends, starts], -1).view(1, 1, S, 2)
    yield "global_sliding", False, torch.stack([(cols + 40).clamp(max=S), torch.full((S,), S, dtype=torch.int32),
                                               torch.full((S,), 8, dtype=torch.int32), (cols - 40).clamp(min=8)], -1).view(1, 1, S, 4)


@pytest.mark.parametrize("S,Hq,Hkv", [(200, 2, 1), (1024, 4, 2)])
def test_flashmask_fwd_bwd(S, Hq, Hkv):
    """Column-sparse masks inside the flash kernels (forward, backward, whole-tile skipping) against a dense fp32 mask."""
    import paddle_b200 as paddle
    from paddle_b200.ops import _lib
    scale = 1 / math.sqrt(128)
    for name, causal, idx in _flashmask_cases(S, "cuda"):
        idx = idx.cuda()
        torch.manual_seed(S)
        q = torch.randn(2, S, Hq, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        k = torch.randn(2, S, Hkv, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        v = torch.randn(2, S, Hkv, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        do = torch.randn(2, S, Hq, 128, device="cuda").to(torch.bfloat16)
        idx2 = idx.expand(2, 1, S, idx.shape[-1]).contiguous()
        o = paddle.nn.functional.flashmask_attention(q, k, v, idx2, causal=causal)
        o.backward(do)
        _lib.check_status()
        masked = _dense_from_flashmask(idx2, S, S, causal)
        qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
        ro = _masked_ref(qf, kf, vf, masked, scale)
        ro.backward(do.float())
        assert (o.float() - ro).abs().max().item() < 3e-2, name
        for nm, a, b in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
            err = (a.float() - b).abs().max().item()
            assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{name} {nm}: {err}"


def test_varlen_packed_single_launch():
    """flash_attn_unpadded on a ragged packing runs as one masked launch and equals per-sequence attention."""
    import paddle_b200 as paddle
    from paddle_b200.ops import _lib, native
    lens = [37, 300, 128, 515]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    total, H = sum(lens), 2
    torch.manual_seed(1)
    scale = 1 / math.sqrt(128)
    for causal in (True, False):
        q = torch.randn(total, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        k = torch.randn(total, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        v = torch.randn(total, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
        do = torch.randn(total, H, 128, device="cuda").to(torch.bfloat16)
        before = native.LAUNCH_COUNT
        o, _ = paddle.nn.functional.flash_attn_unpadded(q, k, v, cu, cu, max(lens), max(lens), scale, causal=causal)
        assert native.LAUNCH_COUNT - before == 1
        o.backward(do)
        _lib.check_status()
        qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
        outs = []
        for i in range(len(lens)):
            sl = slice(int(cu[i]), int(cu[i + 1]))
            r, _ = _ref(qf[sl].unsqueeze(0), kf[sl].unsqueeze(0), vf[sl].unsqueeze(0), causal, scale)
            outs.append(r.squeeze(0))
        ro = torch.cat(outs, 0)
        ro.backward(do.float())
        assert (o.float() - ro).abs().max().item() < 3e-2
        for nm, a, b in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
            err = (a.float() - b).abs().max().item()
            assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{nm}: {err}"


def test_flash_long_sequence_bwd():
    """S = 4096, 8 heads, causal: forward and backward against the fp32 reference."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(11)
    B, S, H = 1, 4096, 8
    q = torch.randn(B, S, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    k = torch.randn(B, S, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    v = torch.randn(B, S, H, 128, device="cuda").to(torch.bfloat16).requires_grad_(True)
    do = torch.randn(B, S, H, 128, device="cuda").to(torch.bfloat16)
    scale = 1 / math.sqrt(128)
    o = attention.flash_attn_func(q, k, v, True, scale)
    o.backward(do)
    _lib.check_status()
    qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ro, _ = _ref(qf, kf, vf, True, scale)
    ro.backward(do.float())
    assert (o.float() - ro).abs().max().item() < 3e-2
    for nm, a, b in (("dq", q.grad, qf.grad), ("dk", k.grad, kf.grad), ("dv", v.grad, vf.grad)):
        err = (a.float() - b).abs().max().item()
        assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{nm}: {err}"


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,Sq,Sk", [(10, 300, 100), (10, 384, 200), (4, 520, 257), (10, 130, 400), (10, 256, 1)])
def test_flash_fwd_unequal_tiles(causal, B, Sq, Sk):
    """Enough blocks for two query tiles per CTA, whose tiles see different numbers of key tiles: one of them none (it lies
    behind the queries, or before the first visible key), one more than the other."""
    from paddle_b200.ops import _lib, attention
    torch.manual_seed(Sq + Sk)
    q, k, v = (torch.randn(B, s, h, 128, device="cuda").to(torch.bfloat16) for s, h in ((Sq, 40), (Sk, 8), (Sk, 8)))
    scale = 1 / math.sqrt(128)
    o, lse = attention.fwd(q, k, v, causal, scale)
    _lib.check_status()
    ro, rl = _ref(q, k, v, causal, scale)
    ro = torch.nan_to_num(ro)                      # rows that see no key: zero output, log-sum-exp -inf
    live = torch.isfinite(rl)
    assert torch.equal(torch.isfinite(lse), live)
    assert torch.allclose(lse[live], rl[live], rtol=1e-3, atol=2e-3)
    # P and O are rounded to bf16 (2^-9 relative each); |v| stays below 6
    assert (o.float() - ro).abs().max() <= 6 * 2 ** -8 + 1e-3


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("B,H,Sk", [(1, 2, 100), (1, 2, 128), (1, 2, 300), (10, 40, 300)])
def test_flash_fwd_largest_probability_is_exact(B, H, Sk, masked):
    """Each row's largest score lies in the second half of the first 128 keys, less than 2^8 above the first 64: its probability is
    the reference point of the row (1, exact in bf16), so that the output carries one rounding to bf16 and no second one.  One and
    two query tiles per CTA; with a column-sparse mask a larger score beside it is hidden and must not count."""
    from paddle_b200.ops import _lib, attention
    Sq = min(Sk, 257)
    a = torch.linspace(0.1, 7.4, Sq, device="cuda").to(torch.bfloat16)
    q, k, v = (torch.zeros(B, s, H, 128, device="cuda", dtype=torch.bfloat16) for s in (Sq, Sk, Sk))
    q[..., 0] = a[None, :, None]
    k[:, 64, :, 0] = 8.0                                # log2 of its probability to that of the others: 1.02 a
    v[:, 64] = 1.0
    scale, mask = 1 / math.sqrt(128), None
    if masked:
        k[:, 70, :, 0] = 8.5
        idx = torch.full((B, 1, Sk, 2), Sq, dtype=torch.int32, device="cuda")
        idx[..., 1] = 0
        idx[:, :, 70] = torch.tensor([0, Sq], dtype=torch.int32, device="cuda")
        mask = attention.normalize_flashmask(idx, False, Sq)
    o, _ = attention.fwd(q, k, v, False, scale, mask)
    _lib.check_status()
    want = 1 / (1 + (Sk - 1 - int(masked)) * torch.exp(-8 * a.double() * scale))
    err = ((o.double() - want[None, :, None, None]) / want[None, :, None, None]).abs().max().item()
    # one rounding to bf16 (8 significand bits: half a step is at most 2^-8 of the value); sums and exponentials are good to 1e-6
    assert err <= 2 ** -8 * 1.001, err


def _two_tile_masks(S, B, Hq):
    """Masks for grids that take two query tiles per CTA: (name, causal, startend_row_indices)."""
    for name, causal, idx in _flashmask_cases(S, "cpu"):
        yield name, causal, idx.expand(B, 1, S, idx.shape[-1])
    # a document mask of its own for every head and sequence
    g = torch.Generator().manual_seed(S)
    cut = torch.randint(1, S, (B, Hq, 1), generator=g)
    cols = torch.arange(S).view(1, 1, S)
    ends = torch.where(cols < cut, cut, torch.full_like(cut, S)).to(torch.int32)
    starts = torch.where(cols < cut, torch.zeros_like(cut), cut).to(torch.int32)
    yield "documents per head", True, ends.unsqueeze(-1)
    yield "documents per head", False, torch.stack([ends, starts], -1)
    # rows 128 .. 383 see nothing: the second tile of the first pair and the first tile of the second pair
    band = torch.tensor([128, 256, 256, 384], dtype=torch.int32)
    yield "one tile of a pair", False, band.expand(B, 1, S, 4)
    # the first 128 rows see the last keys only and the others the first keys only, so the tiles of a pair share no key tile
    half = torch.full((S, 4), S, dtype=torch.int32)
    half[:S // 2] = torch.tensor([0, 128, 0, 0], dtype=torch.int32)
    half[S // 2:] = torch.tensor([128, S, 0, 0], dtype=torch.int32)
    yield "tiles apart", False, half.view(1, 1, S, 4).expand(B, 1, S, 4)


@pytest.mark.parametrize("B,S", [(4, 520), (2, 1000)])
def test_flashmask_two_query_tiles(B, S):
    """The masked kernels with two query tiles per CTA (enough blocks that the size rule takes them): output, log-sum-exp and gradients
    against a dense mask, for tiles of a pair that see other keys than each other, or none."""
    from paddle_b200.ops import _lib, attention
    Hq, Hkv, scale = 40, 8, 1 / math.sqrt(128)
    for name, causal, idx in _two_tile_masks(S, B, Hq):
        idx = idx.cuda().contiguous()
        torch.manual_seed(S)
        q, k, v, do = (torch.randn(B, S, h, 128, device="cuda").to(torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
        mask = attention.normalize_flashmask(idx, causal, S)
        o, lse = attention.fwd(q, k, v, causal, scale, mask)
        dq, dk, dv = attention.bwd(do, q, k, v, o, lse, causal, scale, mask=mask)
        _lib.check_status()
        masked = _dense_from_flashmask(idx, S, S, causal)
        dead = masked.all(-1).expand(B, Hq, S)
        qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
        ro = _masked_ref(qf, kf, vf, masked, scale)
        ro.backward(do.float())
        with torch.no_grad():
            s = qf.transpose(1, 2) @ kf.transpose(1, 2).repeat_interleave(Hq // Hkv, 1).mT * scale
            rl = torch.logsumexp(s.masked_fill_(masked, float("-inf")), -1)
            del s
        assert torch.equal(torch.isfinite(lse), ~dead), (name, causal)
        assert torch.allclose(lse[~dead], rl[~dead], rtol=1e-3, atol=2e-3), (name, causal)
        assert (o.float() - ro).abs().max().item() < 3e-2, (name, causal)
        assert dq.transpose(1, 2)[dead].float().abs().sum().item() == 0, (name, causal)
        for nm, a, b in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
            err = (a.float() - b).abs().max().item()
            assert err <= 3e-2 * b.abs().max().item() + 2e-2, f"{name} {causal} {nm}: {err}"
