"""Short prompts' products on single SMs (bf16, no residual), at the edges of their tiles and of the rule that sends them there, against
float64 sums and the paired-SM kernel's bits: both add the slices of K in their order, so a row's bits do not hang on which one ran."""
import ctypes

import pytest
import torch
from test_gpu_21_prompt_gemm import bound, linear, linear_ref, operands

from rai_b200 import _lib

pytestmark = pytest.mark.gpu
P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


def on_pairs(cuda, x, w, w2, b, act):
    out = torch.full((x.shape[0], w.shape[0]), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.call("rb_selftest_pair_linear", cuda.ctx, P(x), P(w), P(w2), P(b), None, P(out), *out.shape, x.shape[1], act, 256, 0)
    return out


# a row more than two tiles, a tile and a row less, part of a tile; a piece of columns, within a tile, a whole one; part of a slice of K, the
# last K that one round takes and the first it leaves; two and three rounds where pairs need one more; too many tiles, odd columns
@pytest.mark.parametrize("m,n,k", [(257, 8, 8), (257, 264, 72), (511, 256, 896), (383, 1000, 328), (300, 520, 3584), (300, 520, 3592), (1400, 10240, 256),
                                   (600, 7680, 640), (1400, 9000, 64), (600, 1003, 256)])
def test_linear(cuda, m, n, k):
    cuda.use_torch_stream()
    x, w, _, b, _ = operands(m, n, k, torch.bfloat16, m + n + k)
    for bias, act in ((None, _lib.ACT_NONE), (b, _lib.ACT_SILU)):
        got, ref = linear(cuda, x, w, bias, None, act), linear_ref(x, w, bias, None, act)
        cuda.synchronize()
        assert float((got.double() - ref).abs().max()) <= bound(torch.bfloat16, ref, k)
        assert torch.equal(got, on_pairs(cuda, x, w, None, bias, act))


@pytest.mark.parametrize("m,n,k", [(129, 8, 8), (200, 136, 72), (256, 4864, 896), (257, 128, 3584), (257, 128, 3592), (1400, 4864, 136), (600, 4096, 1024), (600, 4096, 1032),
                                   (2100, 4104, 64)])
def test_gated_linear(cuda, m, n, k):
    cuda.use_torch_stream()
    x, w, w2, _, _ = operands(m, n, k, torch.bfloat16, m + n + k)
    got = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.call("rb_gated_linear", cuda.ctx, P(x), P(w), P(w2), P(got), m, n, k, _lib.ACT_SILU, _lib.BF16)
    cuda.synchronize()
    ref = torch.nn.functional.silu(x.double() @ w.double().t()) * (x.double() @ w2.double().t())
    assert float((got.double() - ref).abs().max()) <= 2 * bound(torch.bfloat16, ref, k)   # (and a fast exponential)
    assert torch.equal(got, on_pairs(cuda, x, w, w2, None, _lib.ACT_SILU))


def test_infinities_and_nan_stay_in_their_rows(cuda):
    cuda.use_torch_stream()
    x, w, _, _, _ = operands(300, 520, 1000, torch.bfloat16, 4)
    clean = linear(cuda, x, w, None, None, _lib.ACT_NONE)
    x2 = x.clone()
    x2[299, 5], x2[130, 990] = float("nan"), float("inf")
    out = linear(cuda, x2, w, None, None, _lib.ACT_NONE)
    cuda.synchronize()
    assert torch.isnan(out[299]).all() and not torch.isfinite(out[130]).any()
    keep = [i for i in range(300) if i not in (130, 299)]
    assert torch.equal(out[keep], clean[keep])


# rb_linear by itself has no workspace to be cut in: one round of tiles at any K, two where pairs need three
@pytest.mark.parametrize("m,n,k", [(300, 520, 8200), (511, 3584, 4096), (513, 14336, 3592)])
def test_linear_of_many_slices(cuda, m, n, k):
    test_linear(cuda, m, n, k)


@pytest.mark.parametrize("m,n,k", [(257, 264, 8200), (129, 4096, 4096), (257, 10240, 1032)])
def test_gated_linear_of_many_slices(cuda, m, n, k):
    test_gated_linear(cuda, m, n, k)
