"""Prompt attention on tcgen05 at every head size it takes, on an empty and on a filled cache, against float64 sums over the
same bf16 operands."""
import ctypes
import math

import pytest
import torch

from rai_b200 import _lib
from test_gpu_30_attention import Cache

pytestmark = pytest.mark.gpu
P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


def append(cuda, cache, rows, batch, s_new, nq, d):
    """rows [batch * s_new, (nq + 2 kv) * d] into the cache as they are (a rotary width of 0); the query part comes back."""
    q, none = torch.empty(batch * s_new, nq * d, dtype=torch.bfloat16, device="cuda"), torch.zeros(64, device="cuda")
    _lib.call("rb_rope_kv_append", cuda.ctx, P(rows), None, 0, None, P(none), P(none), 0, batch, s_new, nq, cache.h, 0, P(q), _lib.BF16)
    return q


@pytest.mark.parametrize("nq,nkv,d", [(4, 2, 64), (3, 3, 80), (2, 2, 96), (4, 2, 128), (8, 1, 256), (3, 1, 256)])
@pytest.mark.parametrize("cached,s_new", [(0, 128), (0, 129), (0, 383), (70, 200), (64, 256)])
def test_prompt_attention(cuda, nq, nkv, d, cached, s_new):
    cuda.use_torch_stream()
    batch, total = 2, cached + s_new
    g = torch.Generator(device="cuda").manual_seed(d + total)
    rows = (torch.randn(batch, total, (nq + 2 * nkv) * d, generator=g, device="cuda") * 1.5).to(torch.bfloat16)
    cache = Cache(cuda, 1, nkv, d, batch, total + 3, torch.bfloat16)
    if cached:
        cache.set_len(batch, cached)
        append(cuda, cache, rows[:, :cached].reshape(batch * cached, -1).contiguous(), batch, cached, nq, d)
    cache.set_len(batch, total)
    q = append(cuda, cache, rows[:, cached:].reshape(batch * s_new, -1).contiguous(), batch, s_new, nq, d)
    out = torch.full((batch, s_new, nq, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    _lib.call("rb_attention", cuda.ctx, P(q), cache.h, 0, batch, s_new, nq, 1.0 / math.sqrt(d), P(out), _lib.BF16)
    cuda.synchronize()
    cache.close()
    parts = rows.double().split([nq * d, nkv * d, nkv * d], -1)
    qh, kh, vh = (t.reshape(batch, total, -1, d).transpose(1, 2) for t in parts)
    kh, vh = (t.repeat_interleave(nq // nkv, 1) for t in (kh, vh))
    z = qh[:, :, cached:] @ kh.transpose(2, 3) / math.sqrt(d)
    z = z.masked_fill(torch.arange(total, device="cuda") > torch.arange(cached, total, device="cuda")[:, None], -math.inf)
    ref = (torch.softmax(z, -1) @ vh).transpose(1, 2)
    # weights and result are each rounded to bf16 once (2^-9), weights of one row up to 2^8 apart from their reference point
    assert float((out.double() - ref).abs().max()) <= 3 * 2.0 ** -9 * float(vh.abs().max())
