"""The float32 products at the edges of their tiles, against float64 sums of the same operands."""
import ctypes

import pytest
import torch

from rai_b200 import _lib

pytestmark = pytest.mark.gpu
P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
DT = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}


def operands(m, n, k, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    return (r(m, k).to(dtype), (r(n, k) * 0.05).to(dtype), (r(n, k) * 0.05).to(dtype), r(n).to(dtype), r(m, n).to(dtype))


def bound(dtype, ref, k):
    # bf16: one rounding of the result, 2^-9 of it, and float32 sums; float32: k roundings of 2^-24 that do not all point one way
    return (2.0 ** -8 if dtype == torch.bfloat16 else 4 * k ** 0.5 * 2.0 ** -24) * float(ref.abs().max()) + 1e-6


def linear(cuda, x, w, b, r, act):
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), dtype=x.dtype, device="cuda")
    _lib.call("rb_linear", cuda.ctx, P(x), P(w), P(b), P(r), P(out), x.shape[0], w.shape[0], x.shape[1], act, DT[x.dtype])
    return out


def linear_ref(x, w, b, r, act):
    y = x.double() @ w.double().t()
    y = y + b.double() if b is not None else y
    y = torch.nn.functional.silu(y) if act == _lib.ACT_SILU else y
    return y + r.double() if r is not None else y


# rows: few (a dot product per row) and many (tiles of 16 to 128 rows); features around a tile; K cut in up to eight shares, not a
# multiple of a slice, not a multiple of four
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 16, 33, 77, 128, 145])
@pytest.mark.parametrize("n,k", [(64, 32), (65, 896), (130, 4864), (1000, 100), (7, 30), (896, 36)])
def test_float32_products(cuda, m, n, k):
    cuda.use_torch_stream()
    x, w, w2, b, r = operands(m, n, k, torch.float32, m * n + k)
    for bias, res, act in ((None, None, _lib.ACT_NONE), (b, r, _lib.ACT_SILU)):
        out = linear(cuda, x, w, bias, res, act)
        cuda.synchronize()
        ref = linear_ref(x, w, bias, res, act)
        assert float((out.double() - ref).abs().max()) <= bound(torch.float32, ref, k)
    out = torch.full((m, n), float("nan"), device="cuda")
    _lib.call("rb_gated_linear", cuda.ctx, P(x), P(w), P(w2), P(out), m, n, k, _lib.ACT_SILU, _lib.F32)
    cuda.synchronize()
    ref = torch.nn.functional.silu(x.double() @ w.double().t()) * (x.double() @ w2.double().t())
    assert float((out.double() - ref).abs().max()) <= 2 * bound(torch.float32, ref, k)
