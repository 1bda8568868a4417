"""The products of prompts: the paired-SM bf16 kernel at the edges of its tiles and with tiles cut along K, and the float32
kernels at the edges of theirs, against float32 / float64 sums of the same operands."""
import ctypes

import pytest
import torch

from rai_b200 import _lib, configs, synth
from rai_b200.models import Model

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


# one row more or less than a tile of 256 or 512; columns that end in a tile, in a piece of eight and (250) within one; K of part
# of a slice; few tiles with many slices (cut among all clusters), and a little more than one tile for each cluster
SHAPES = [(257, 256, 64), (511, 264, 72), (512, 8, 8), (513, 250, 192), (300, 512, 8192), (1300, 4096, 2048), (770, 2816, 6400),
          (4096, 2560, 1024), (2600, 1000, 328)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_prompt_products(cuda, m, n, k):
    cuda.use_torch_stream()
    x, w, w2, b, r = operands(m, n, k, torch.bfloat16, m + n + k)
    for bias, res, act in ((None, None, _lib.ACT_NONE), (b, r, _lib.ACT_SILU)):
        out = linear(cuda, x, w, bias, res, act)
        cuda.synchronize()
        ref = linear_ref(x, w, bias, res, act)
        assert float((out.double() - ref).abs().max()) <= bound(torch.bfloat16, ref, k)
    # the residual may be the output itself, and a second pass over fresh sums gives the same bits
    again, once = r.clone(), linear(cuda, x, w, None, r, _lib.ACT_NONE)
    _lib.call("rb_linear", cuda.ctx, P(x), P(w), None, P(again), P(again), m, n, k, _lib.ACT_NONE, _lib.BF16)
    cuda.synchronize()
    assert torch.equal(again, once)
    if n % 8 == 0:
        out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        _lib.call("rb_gated_linear", cuda.ctx, P(x), P(w), P(w2), P(out), m, n, k, _lib.ACT_SILU, _lib.BF16)
        cuda.synchronize()
        ref = torch.nn.functional.silu(x.double() @ w.double().t()) * (x.double() @ w2.double().t())
        assert float((out.double() - ref).abs().max()) <= 2 * bound(torch.bfloat16, ref, k)  # (and a fast exponential)


def test_infinities_and_nan_stay_in_their_rows(cuda):
    cuda.use_torch_stream()
    x, w, _, _, _ = operands(600, 512, 4096, torch.bfloat16, 7)
    clean = linear(cuda, x, w, None, None, _lib.ACT_NONE)
    x2 = x.clone()
    x2[599, 5], x2[300, 4000] = float("nan"), float("inf")
    out = linear(cuda, x2, w, None, None, _lib.ACT_NONE)
    cuda.synchronize()
    assert torch.isnan(out[599]).all() and not torch.isfinite(out[300]).any()
    keep = [i for i in range(600) if i not in (300, 599)]
    assert torch.equal(out[keep], clean[keep])


def test_same_bits_on_every_stream_and_under_capture(cuda):
    """A product called by itself has no workspace that a stream or a graph could share with another."""
    x, w, _, _, _ = operands(300, 512, 8192, torch.bfloat16, 3)
    ref = linear_ref(x, w, None, None, _lib.ACT_NONE)
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    torch.cuda.synchronize()
    for s in streams * 3 + [torch.cuda.Stream() for _ in range(6)]:
        with torch.cuda.stream(s):
            cuda.use_torch_stream()
            outs.append(linear(cuda, x, w, None, None, _lib.ACT_NONE))
    torch.cuda.synchronize()
    graph, static = torch.cuda.CUDAGraph(), torch.zeros(300, 512, dtype=torch.bfloat16, device="cuda")
    with torch.cuda.graph(graph):
        cuda.use_torch_stream()
        _lib.call("rb_linear", cuda.ctx, P(x), P(w), None, None, P(static), 300, 512, 8192, _lib.ACT_NONE, _lib.BF16)
    graph.replay()
    torch.cuda.synchronize()
    cuda.use_torch_stream()
    cuda.synchronize()
    for out in outs + [static]:
        assert float((out.double() - ref).abs().max()) <= bound(torch.bfloat16, ref, 8192)
        assert torch.equal(out, outs[0])


def test_a_row_has_the_same_bits_in_any_batch(cuda):
    cuda.use_torch_stream()
    x, w, w2, _, _ = operands(1300, 512, 8192, torch.bfloat16, 5)
    whole = linear(cuda, x, w, None, None, _lib.ACT_NONE)
    for m in (257, 300, 700):
        assert torch.equal(linear(cuda, x[:m].contiguous(), w, None, None, _lib.ACT_NONE), whole[:m])
    cuda.synchronize()


def test_products_by_themselves_allocate_nothing(cuda):
    """Every stream's first product, too: a host that owns the GPU's memory does not see it shrink."""
    x, w, _, _, _ = operands(300, 512, 8192, torch.bfloat16, 6)
    out = torch.empty(300, 512, dtype=torch.bfloat16, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(3)]

    def product(s):
        with torch.cuda.stream(s):
            cuda.use_torch_stream()
            _lib.call("rb_linear", cuda.ctx, P(x), P(w), None, None, P(out), 300, 512, 8192, _lib.ACT_NONE, _lib.BF16)
        s.synchronize()

    product(torch.cuda.default_stream())     # (the kernel's code is loaded)
    free = torch.cuda.mem_get_info()[0]
    for s in streams:
        product(s)
    left = torch.cuda.mem_get_info()[0]
    cuda.use_torch_stream()
    assert free - left < 8 << 20


def test_a_model_on_any_stream_has_the_same_bits(cuda):
    """A model's products are cut along K in a workspace of its own, whichever stream its calls come on."""
    cfg = configs.get("qwen2-0.5b")
    cfg.update(num_hidden_layers=2, vocab_size=512)
    m = Model(cfg, _lib.BF16, cuda, 1, 320, 320)
    m.update_params(synth.weights(cfg, 8))
    ids = synth.prompt(cfg, 1, 300, 8)
    outs = []
    torch.cuda.synchronize()
    for s in [torch.cuda.Stream() for _ in range(7)]:
        with torch.cuda.stream(s):
            m.clear_kv_cache()
            outs.append(m.forward(ids, 0))
        s.synchronize()
    cuda.use_torch_stream()
    assert all(torch.equal(o, outs[0]) for o in outs)
    m.close()


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


# K too short to be cut: as many tiles as fit the GPU at once, then taller ones
@pytest.mark.parametrize("m,n,k", [(128, 64, 64), (300, 2048, 100), (513, 200, 220), (1000, 64, 8), (700, 6000, 36), (257, 64, 224)])
def test_float32_products_of_short_rows(cuda, m, n, k):
    test_float32_products(cuda, m, n, k)
