"""tcgen05 GEMM vs an fp32 PyTorch reference: every operand-layout combination, ragged edges,
bf16 / fp32 / fp32-accumulate epilogues, for both tile schemes (128 x 256 per SM; 256 x 256 per SM pair with
tcgen05 cta_group::2)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["1cta", "2cta"], autouse=True)
def gemm_impl(request):
    from paddle_b200.ops import native
    prev = native.set_gemm_impl(request.param)
    yield request.param
    native.set_gemm_impl(prev)


def _ref(a, b, ta, tb):
    A = a.float().t() if ta else a.float()
    B = b.float().t() if tb else b.float()
    return A @ B


def _mk(M, N, K, ta, tb, dev="cuda"):
    g = torch.Generator(device=dev).manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M) if ta else (M, K), device=dev, generator=g).to(torch.bfloat16)
    b = torch.randn((N, K) if tb else (K, N), device=dev, generator=g).to(torch.bfloat16)
    return a, b


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (384, 776, 200), (1000, 264, 1032), (136, 144, 72)])
def test_gemm_layouts(ta, tb, M, N, K):
    from paddle_b200.ops import _lib, native
    a, b = _mk(M, N, K, ta, tb)
    out = native.gemm(a, b, ta, tb)
    _lib.check_status()
    ref = _ref(a, b, ta, tb)
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 2e-2 * scale + 1e-2, f"max err {err} (scale {scale})"


def test_gemm_fp32_out_and_accumulate():
    from paddle_b200.ops import _lib, native
    M, N, K = 512, 768, 1024
    a, b = _mk(M, N, K, True, False)
    ref = _ref(a, b, True, False)
    out = native.gemm(a, b, True, False, out_dtype=torch.float32)
    _lib.check_status()
    assert torch.allclose(out, ref, rtol=1e-3, atol=1e-2)
    acc = torch.full((M, N), 2.0, device="cuda")
    native.gemm(a, b, True, False, out=acc, accumulate=True)
    native.gemm(a, b, True, False, out=acc, accumulate=True)
    _lib.check_status()
    assert torch.allclose(acc, 2.0 + 2 * ref, rtol=1e-3, atol=2e-2)


def test_gemm_large_and_deterministic():
    from paddle_b200.ops import _lib, native
    M, N, K = 4096, 11008, 4096
    a, b = _mk(M, N, K, False, False)
    o1 = native.gemm(a, b)
    o2 = native.gemm(a, b)
    _lib.check_status()
    assert torch.equal(o1, o2)
    ref = a[:256].float() @ b.float()
    assert torch.allclose(o1[:256].float(), ref, rtol=2e-2, atol=1.0)
    ref2 = a[-128:].float() @ b.float()
    assert torch.allclose(o1[-128:].float(), ref2, rtol=2e-2, atol=1.0)


def test_debug_bounds_build_runs_clean():
    """The -DPD_DEBUG_BOUNDS build of the kernels (every TMA / bulk copy checked before it is issued) computes the same
    results and records no violation for GEMM (all layouts, accumulate), attention forward / backward and RMSNorm."""
    import os
    import subprocess
    import sys
    code = r"""
import math, torch
from paddle_b200.ops import _lib, native, attention
assert hasattr(_lib.kernels(), "pd_debug_bounds_read")
torch.manual_seed(0)
a = torch.randn(300, 520, device="cuda").bfloat16(); b = torch.randn(520, 264, device="cuda").bfloat16()
for impl in ("2cta", "1cta"):
    native.set_gemm_impl(impl)
    y = native.gemm(a, b)
    assert (y.float() - a.float() @ b.float()).abs().max() < 0.5
    acc = torch.zeros(520, 264, device="cuda")
    x2 = torch.randn(300, 264, device="cuda").bfloat16()
    native.gemm(a, x2, trans_a=True, out=acc, accumulate=True)
    assert (acc - a.float().t() @ x2.float()).abs().max() < 0.5
q = torch.randn(1, 300, 2, 128, device="cuda").bfloat16().requires_grad_(True)
k = torch.randn(1, 300, 2, 128, device="cuda").bfloat16().requires_grad_(True)
v = torch.randn(1, 300, 2, 128, device="cuda").bfloat16().requires_grad_(True)
o = attention.flash_attn_func(q, k, v, True, 1 / math.sqrt(128))
o.backward(torch.randn_like(o))
w = torch.ones(512, device="cuda").bfloat16()
native.rms_norm_fwd(torch.randn(64, 512, device="cuda").bfloat16(), w, 1e-6)
torch.cuda.synchronize()
_lib.check_status()
assert _lib.debug_bounds_violation() is None
print("CLEAN")
"""
    env = dict(os.environ, PD_DEBUG_BOUNDS="1", PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=900)
    assert p.returncode == 0 and "CLEAN" in p.stdout, p.stdout[-2000:] + p.stderr[-3000:]


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K_", [(136, 8, 64), (264, 4680, 200), (264, 4744, 200), (1032, 2568, 72), (2304, 1160, 136)])
def test_narrow_and_wide_tiles(M, N, K_, ta, tb):
    """Both sides of the rule that picks 256 x 128 or 256 x 256 tiles (the most narrow tiles that run at once, and one column
    of tiles more), ragged in every extent, all layouts and epilogues."""
    from paddle_b200.ops import _lib, native
    torch.manual_seed(M + N)
    a = torch.randn((K_, M) if ta else (M, K_), device="cuda").bfloat16()
    b = torch.randn((N, K_) if tb else (K_, N), device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    # fp32 sums of K_ products of size 1, then one rounding to bf16
    tol, sums = ref.abs() * 2 ** -8 + 1e-3, 16 * K_ * 2 ** -22
    assert (native.gemm(a, b, ta, tb).double() - ref).abs().le(tol).all()
    acc = torch.randn(M, N, device="cuda")
    got = native.gemm(a, b, ta, tb, out=acc.clone(), accumulate=True)
    assert (got.double() - ref - acc.double()).abs().max() <= sums + 1e-5
    assert (native.gemm(a, b, ta, tb, out_dtype=torch.float32).double() - ref).abs().max() <= sums + 1e-5
    pre = ref + bias.double()
    assert (native.gemm_epilogue(a, b, bias, "relu", ta, tb).double() - pre.clamp(min=0)).abs().le(pre.abs() * 2 ** -8 + 1e-3).all()
    # a bias that does not start on 16 bytes
    odd = torch.randn(N + 1, device="cuda").bfloat16()[1:]
    pre = ref + odd.double()
    assert (native.gemm_epilogue(a, b, odd, None, ta, tb).double() - pre).abs().le(pre.abs() * 2 ** -8 + 1e-3).all()
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("max_ctas", [0, 1, 2, 16, 40])
def test_tile_width_follows_the_ctas_a_call_may_use(max_ctas):
    """Narrow tiles only where all of them run at once on the CTA pairs that the caller leaves to the product."""
    from paddle_b200.ops import _lib, native
    M, N, K_ = 1000, 1160, 264                       # 4 x 10 narrow tiles
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    pairs = max(1, min(pairs, max_ctas // 2)) if max_ctas else pairs
    assert _lib.kernels().pd_gemm_2cta_tile_n(M, N, 1, max_ctas) == (128 if 40 <= pairs else 256)
    torch.manual_seed(max_ctas)
    a, b = torch.randn(M, K_, device="cuda").bfloat16(), torch.randn(K_, N, device="cuda").bfloat16()
    ref = a.double() @ b.double()
    got = native.gemm(a, b, max_ctas=max_ctas)
    torch.cuda.synchronize()
    _lib.check_status()
    assert (got.double() - ref).abs().le(ref.abs() * 2 ** -8 + 1e-3).all()      # fp32 sums of products of size 1, one rounding


@pytest.mark.parametrize("M,N,counts", [(136, 144, [70, 0, 1, 64, 65]), (512, 264, [300, 129, 300]), (1024, 2048, [128] * 9 + [0, 500]), (256, 256, [0, 0])])
def test_gemm_grouped_weight_gradients(M, N, counts):
    """Uneven, equal, empty and more groups than one launch takes, on ragged sizes; rows past the counted ones are not read."""
    from paddle_b200.ops import _lib, native
    rows = sum(counts)
    a, b = _mk(M, N, max(rows, 1) + 40, True, False)
    a[rows:], b[rows:] = float("nan"), float("nan")
    acc = torch.randn(len(counts), M, N, device="cuda")
    start, plain = acc.clone(), torch.full((len(counts), M, N), 7.0, device="cuda", dtype=torch.bfloat16)
    native.gemm_grouped_tn(a, b, counts, acc, accumulate=True)
    native.gemm_grouped_tn(a, b, counts, plain)
    _lib.check_status()
    s = 0
    for g, n in enumerate(counts):
        ref = _ref(a[s:s + n], b[s:s + n], True, False)
        s += n
        # products of bf16 are exact in fp32, n of them are summed: errors of n * 2^-24 relative to the sum of magnitudes (< 6 n)
        tol = 6 * max(n, 1) * n * 2 ** -24 + 1e-5
        assert (acc[g] - start[g] - ref).abs().max() <= tol + 2 ** -22 * (start[g].abs().max() + ref.abs().max())
        if n:
            assert ((plain[g].float() - ref).abs() <= 2 ** -8 * ref.abs() + tol).all()
        else:
            assert torch.equal(plain[g], torch.full_like(plain[g], 7.0))


@pytest.mark.parametrize("M,N,K_,max_ctas,width", [(304, 776, 8200, 2, 512), (200, 1112, 8256, 8, 512), (304, 776, 8136, 2, 256), (304, 520, 8200, 2, 256),
                                                   (2048, 2600, 8200, 0, 512)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_deep_products_take_wide_tiles(M, N, K_, max_ctas, width, ta, tb):
    """256 x 512 tiles, the last one with its second half full, partly or wholly outside, all layouts and epilogues, and shapes just
    outside the rule; the same sums in the same order as the other tiles."""
    from paddle_b200.ops import _lib, native
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _lib.kernels().pd_gemm_2cta_tile_n_at(M, N, K_, 1, max_ctas) == width
    g = torch.Generator(device="cuda").manual_seed(M + N + K_)
    a = torch.randn((K_, M) if ta else (M, K_), device="cuda", generator=g).bfloat16()
    b = torch.randn((N, K_) if tb else (K_, N), device="cuda", generator=g).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    # The tensor cores cut off what does not fit when they add: each of K_ / 16 steps loses up to 2^-23 of a running sum, which for
    # products of size 1 stays below 5 sqrt(K_).  Then one rounding to bf16.
    sums = K_ / 16 * 5 * K_ ** 0.5 * 2 ** -23
    tol = ref.abs() * 2 ** -8 + sums
    assert (native.gemm(a, b, ta, tb, max_ctas=max_ctas).double() - ref).abs().le(tol).all()
    assert (native.gemm(a, b, ta, tb, out_dtype=torch.float32, max_ctas=max_ctas).double() - ref).abs().max() <= sums
    acc = torch.randn(M, N, device="cuda", generator=g)
    got = native.gemm(a, b, ta, tb, out=acc.clone(), accumulate=True, max_ctas=max_ctas)
    assert (got.double() - ref - acc.double()).abs().max() <= sums + 1e-4
    assert (native.gemm_epilogue(a, b, bias, None, ta, tb).double() - ref - bias.double()).abs().le(tol + bias.double().abs() * 2 ** -8).all()
    torch.cuda.synchronize()
    _lib.check_status()


@pytest.mark.parametrize("M,N,K_,width", [(4360, 264, 136, 128), (8200, 520, 136, 256), (4360, 776, 8200, 256), (3848, 776, 8200, 256),
                                          (3840, 776, 8200, 256), (4360, 1304, 8200, 512)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, True)])
def test_row_tiles_of_several_raster_groups(M, N, K_, width, ta, tb):
    """More row tiles than a raster group holds, the last group ragged: 18 and 33 in groups of 16, deep ones with 256 columns in groups
    of 8 from 16 row tiles on, in one group of 16 with 15."""
    from paddle_b200.ops import _lib, native
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _lib.kernels().pd_gemm_2cta_tile_n_at(M, N, K_, 1, 0) == width
    a, b = _mk(M, N, K_, ta, tb)
    ref = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    # as test_deep_products_take_wide_tiles: K_ / 16 steps lose up to 2^-23 of a running sum below 5 sqrt(K_); one rounding to bf16
    sums = K_ / 16 * 5 * K_ ** 0.5 * 2 ** -23 + 1e-5
    got = native.gemm(a, b, ta, tb)
    _lib.check_status()
    assert (got.double() - ref).abs().le(ref.abs() * 2 ** -8 + sums).all()
    acc = torch.ones(M, N, device="cuda")
    native.gemm(a, b, ta, tb, out=acc, accumulate=True)
    _lib.check_status()
    assert (acc.double() - 1 - ref).abs().max() <= sums + 1e-4
