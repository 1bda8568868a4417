"""Prompt attention on tcgen05 at every head size it takes, on an empty and on a filled cache, and ragged batches whose
padding is left out, against float64 sums over the same bf16 operands."""
import ctypes
import math

import numpy as np
import pytest
import torch

from rai_b200 import _lib, configs, synth
from rai_b200.models import Model
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


@pytest.mark.parametrize("name,dtype", [("tiny-qwen2-g7", _lib.BF16), ("tiny-phi2", _lib.BF16), ("tiny-phi3", _lib.BF16),
                                        ("tiny-gemma", _lib.BF16), ("tiny-qwen2", _lib.F32)])
@pytest.mark.parametrize("lens", [[150, 1, 33], [0, 140, 129], [2, 0, 1], [128, 127, 5]])
def test_a_ragged_call_is_its_sequences_alone(cuda, name, dtype, lens):
    """Logits of a ragged call, and of the single tokens after it, against each sequence in a call of its own; then a call that
    wants the logits of a padding row, which keeps its padding."""
    cfg = configs.get(name)
    w = synth.weights(cfg, 5)
    rng = np.random.default_rng(6)
    ids = rng.integers(0, cfg["vocab_size"], size=(len(lens), max(lens) + 3)).astype(np.int32)
    seq = ids.shape[1]
    m = Model(cfg, dtype, cuda, len(lens), 256, len(lens) * seq)
    m.update_params(w)
    real = [b for b, n in enumerate(lens) if n]
    got = m.forward_rows(ids, lens, [b * seq + lens[b] - 1 for b in real], 0)
    nxt = rng.integers(0, cfg["vocab_size"], size=(len(lens), 1)).astype(np.int32)
    then = m.forward_rows(nxt, None, range(len(lens)))
    m.clear_kv_cache()
    padded = m.forward_rows(ids, lens, [b * seq + lens[b] - 1 for b in real] + [seq - 1], 0)
    alone = Model(cfg, dtype, cuda, 1, 256, seq)
    alone.update_params(w)
    tol = 1e-4 if dtype == _lib.F32 else 2e-2
    for i, b in enumerate(real):
        alone.clear_kv_cache()
        want = alone.forward(ids[b:b + 1, :lens[b]], 0).float().reshape(-1)
        after = alone.forward(nxt[b:b + 1], lens[b]).float().reshape(-1)
        for have, ref in ((got[i], want), (padded[i], want), (then[b], after)):
            assert float((have.float() - ref).abs().max()) <= tol * float(ref.max() - ref.min()), (b, lens)
    assert torch.isfinite(padded[-1].float()).all()
    m.close()
    alone.close()
