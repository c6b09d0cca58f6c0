"""Saved-tensor hooks over the native operators: a pack hook gets a ``paddle.Tensor``, with the operator dispatch on.  On the CPU
the native kernels are replaced by plain torch."""
import pytest
import torch

import paddle_b200 as paddle
from paddle_b200.ops import attention, native
from paddle_b200.ops import functional as K


def _plain(*ts):
    return [t.as_subclass(torch.Tensor) for t in ts]


def _gemm(a, b, trans_a=False, trans_b=False, out=None, out_dtype=torch.bfloat16, accumulate=False, max_ctas=0):
    a, b = _plain(a, b)
    y = (a.t() if trans_a else a) @ (b.t() if trans_b else b)
    return out.add_(y) if accumulate else y


def _rms(x, w, eps):
    return x * torch.rsqrt(x.float().pow(2).mean(-1, keepdim=True) + eps).to(x.dtype) * w


def _swiglu(x):
    g, u = x.chunk(2, -1)
    return torch.nn.functional.silu(g) * u


def _attn(q, k, v):
    return torch.nn.functional.scaled_dot_product_attention(*(t.transpose(1, 2) for t in (q, k, v))).transpose(1, 2).contiguous()


def _vjp(fn, inputs, grad):
    with torch.enable_grad():
        xs = [t.detach().requires_grad_(True) for t in _plain(*inputs)]
        return torch.autograd.grad(fn(*xs), xs, *_plain(grad))


@pytest.fixture(params=["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def device(request, monkeypatch):
    if request.param == "cpu":
        def rms_fwd(x, w, eps, residual=None, want_residual_out=False):
            s = _plain(x)[0] if residual is None else _plain(x)[0] + _plain(residual)[0]
            return _rms(s, *_plain(w), eps), torch.zeros(s.shape[0]), (None if residual is None else s)

        def rms_bwd(dy, x, w, inv, dx_add=None, dw_out=None):
            dx, dw = _vjp(lambda a, b: _rms(a, b, 1e-6), (x, w), dy)
            return dx if dx_add is None else dx + _plain(dx_add)[0], dw.float()

        def attn_fwd(q, k, v, causal, scale, mask=None):
            return _attn(*_plain(q, k, v)), torch.zeros(q.shape[0], q.shape[2], q.shape[1])
        monkeypatch.setattr(K, "_native", lambda t: t.dtype == torch.bfloat16)
        monkeypatch.setattr(native, "gemm", _gemm)
        monkeypatch.setattr(native, "gemm_epilogue", lambda x, w, b: _gemm(x, w) + _plain(b)[0])
        monkeypatch.setattr(native, "row_sum", lambda d: _plain(d)[0].sum(0), raising=False)
        monkeypatch.setattr(native, "rms_norm_fwd", rms_fwd)
        monkeypatch.setattr(native, "rms_norm_bwd", rms_bwd)
        monkeypatch.setattr(native, "swiglu_fwd", lambda x, y=None: _swiglu(*_plain(x)))
        monkeypatch.setattr(native, "swiglu_bwd", lambda x, y, d: (_vjp(_swiglu, (x,), d)[0], None))
        monkeypatch.setattr(attention, "supported", lambda *a: True)
        monkeypatch.setattr(attention, "fwd", attn_fwd)
        monkeypatch.setattr(attention, "bwd", lambda do, q, k, v, *a, **kw: _vjp(_attn, (q, k, v), do))
    before = paddle.get_device()
    paddle.set_device("gpu:0" if request.param == "cuda" else "cpu")
    yield request.param
    paddle.set_device(before)


def _bf16(device, *shape, seed):
    g = torch.Generator().manual_seed(seed)
    t = paddle.to_tensor(torch.randn(shape, generator=g).to(torch.bfloat16).to(device))
    t.stop_gradient = False
    return t


def _ops(device):
    h, w, b, n = (_bf16(device, *s, seed=i) for i, s in enumerate([(2, 8, 256), (256, 512), (512,), (256,)]))
    r = _bf16(device, 2, 8, 256, seed=7)
    q, k, v = (_bf16(device, 1, 16, 2, 128, seed=i) for i in (8, 9, 10))
    # name, call, inputs, how many of the tensors it keeps are inputs or made from them by views and sums
    return [("linear", lambda: K.linear(h, w, b), (h, w, b), 2), ("rms_norm", lambda: K.rms_norm(h, n), (h, n), 2),
            ("rms_norm residual", lambda: sum(K.rms_norm(h, n, residual=r)), (h, n, r), 2),
            ("swiglu", lambda: K.swiglu(h), (h,), 1), ("swiglu of a view", lambda: K.swiglu(h.transpose([1, 0, 2])), (h,), 1),
            ("matmul", lambda: K.matmul(h.reshape([16, 256]), w), (h, w), 2),
            ("flash_attention", lambda: K.flash_attention(q, k, v), (q, k, v), 3)]


def _grads(f, inputs):
    f().astype("float32").sum().backward()
    got = [t.grad.astype("float32").numpy() for t in inputs]
    for t in inputs:
        t.clear_grad(set_to_zero=False)
    return got


@pytest.mark.parametrize("which", ["paddle", "torch"])
def test_saved_tensor_hooks_get_paddle_tensors(device, which):
    """Pack hooks that use the paddle surface (``astype``, ``numpy``) and dispatched arithmetic.  Through torch's own context manager
    the tensors that a node keeps of its inputs, reshaped or not, are paddle tensors too."""
    seen = []

    def pack(t):
        if which == "paddle":
            assert isinstance(t, paddle.Tensor)
        if isinstance(t, paddle.Tensor):
            assert isinstance(t + 0, paddle.Tensor)                     # the dispatch is on
            seen.append(1)
            return t.astype("float32").numpy(), t.dtype, t.device
        return t

    def unpack(s):
        if isinstance(s, torch.Tensor):
            return s
        seen.append(2)
        return paddle.to_tensor(s[0]).to(s[2]).to(s[1])
    hooks = paddle.autograd.saved_tensors_hooks if which == "paddle" else torch.autograd.graph.saved_tensors_hooks
    for name, f, inputs, kept in _ops(device):
        want = _grads(f, inputs)
        del seen[:]

        def hooked():
            with hooks(pack, unpack):
                return f()
        got = _grads(hooked, inputs)
        assert seen.count(1) >= kept and 2 in seen, name
        for a, b in zip(want, got):
            assert abs(a - b).max() <= 2 ** -7 * abs(a).max(), name         # dQ is summed in no fixed order
