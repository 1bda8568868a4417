"""Head split of prompts: the kernel for many rows, against the same rows in calls too small for it."""
import ctypes

import pytest
import torch

from rai_b200 import _lib
from test_gpu_30_attention import Cache

pytestmark = pytest.mark.gpu
P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


@pytest.mark.parametrize("nq,nkv,d,rot", [(4, 2, 64, 64), (3, 3, 80, 32), (2, 2, 96, 96), (7, 1, 128, 128), (8, 1, 256, 256), (5, 2, 64, 16),
                                          (2, 1, 128, 0),
                                          # rows as wide as the kernel for many of them wants, or wider
                                          (28, 6, 64, 64), (30, 5, 64, 16), (16, 8, 80, 32), (24, 2, 96, 96), (21, 3, 128, 128), (18, 1, 128, 0)])
def test_head_split_of_many_rows(cuda, nq, nkv, d, rot):
    """1200 rows at once, and in two calls of 600: the same bits in q and in the cache."""
    cuda.use_torch_stream()
    batch, s = 3, 400
    g = torch.Generator(device="cuda").manual_seed(d + rot)
    rows = torch.randn(batch, s, (nq + 2 * nkv) * d, generator=g, device="cuda").to(torch.bfloat16)
    cos, sin = (torch.randn(s, max(rot // 2, 8), generator=g, device="cuda") for _ in range(2))
    got = []
    for calls in (1, 2):
        cache, q, n = Cache(cuda, 1, nkv, d, batch, s, torch.bfloat16), [], s // calls
        for i in range(calls):
            cache.set_len(batch, (i + 1) * n)
            part = rows[:, i * n:(i + 1) * n].reshape(batch * n, -1).contiguous()
            out = torch.full((batch * n, nq * d), float("nan"), dtype=torch.bfloat16, device="cuda")
            _lib.call("rb_rope_kv_append", cuda.ctx, P(part), None, 0, None, P(cos), P(sin), rot, batch, n, nq, cache.h, 0, P(out), _lib.BF16)
            q.append(out.reshape(batch, n, -1))
        cuda.synchronize()
        kv = [cache.read(0, b, h, t, 3) for b in range(batch) for h in range(nkv) for t in (0, 62, s // 2 - 1, s - 3)]
        cache.close()
        got.append((torch.cat(q, 1), kv))
    assert torch.equal(got[0][0], got[1][0])
    for (k0, v0), (k1, v1) in zip(got[0][1], got[1][1]):
        assert torch.equal(k0, k1) and torch.equal(v0, v1)
