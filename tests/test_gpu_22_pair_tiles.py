"""The paired-SM product with tiles of 256 and of 512 rows, whole and cut along K, at the edges of its tiles, rings and shares, against
float64 sums.  rb_linear takes the height that its cost model finds cheaper and models lend the workspace that cutting needs; here
both are the caller's choice."""
import ctypes

import pytest
import torch
from test_gpu_21_prompt_gemm import bound, linear_ref, operands

from rai_b200 import _lib

pytestmark = pytest.mark.gpu
P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731


def product(cuda, rows, cut, x, w, w2=None, b=None, r=None, act=_lib.ACT_NONE, out=None):
    m, k, n = x.shape[0], x.shape[1], w.shape[0]
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda") if out is None else out
    _lib.call("rb_selftest_pair_linear", cuda.ctx, P(x), P(w), P(w2), P(b), P(r), P(out), m, n, k, act, rows, int(cut))
    return out


def check(cuda, rows, cut, m, n, k, gated):
    cuda.use_torch_stream()
    x, w, w2, b, r = operands(m, n, k, torch.bfloat16, m + n + k)
    if gated:
        got, ref = product(cuda, rows, cut, x, w, w2, act=_lib.ACT_SILU), x.double() @ w.double().t()
        ref = torch.nn.functional.silu(ref) * (x.double() @ w2.double().t())
        assert float((got.double() - ref).abs().max()) <= 2 * bound(torch.bfloat16, ref, k)   # (and a fast exponential)
    else:
        for bias, res, act in ((None, None, _lib.ACT_NONE), (b, r, _lib.ACT_SILU)):
            got, ref = product(cuda, rows, cut, x, w, None, bias, res, act), linear_ref(x, w, bias, res, act)
            assert float((got.double() - ref).abs().max()) <= bound(torch.bfloat16, ref, k)
        # the residual may be the output, and a second pass gives the same bits
        again = product(cuda, rows, cut, x, w, None, None, r)
        assert torch.equal(product(cuda, rows, cut, x, w, None, None, out := r.clone(), out=out), again)
        got = product(cuda, rows, cut, x, w)
    if cut and m * n > 500000:   # other sums, so among so many some rounding falls the other way: tiles were cut
        assert not torch.equal(got, product(cuda, rows, False, x, w, w2 if gated else None, act=_lib.ACT_SILU if gated else _lib.ACT_NONE))


# rows: one more than half a tile of 512, a tile and one row less or more; columns: a piece of eight, within one, a tile and a piece; K: part
# of a slice, as many slices as a ring has stages (four and six), one more, more than two rings
@pytest.mark.parametrize("rows", [256, 512])
@pytest.mark.parametrize("m,n,k", [(257, 8, 8), (257, 264, 64), (511, 250, 200), (512, 256, 256), (513, 520, 320), (770, 250, 392), (1281, 136, 1000)])
def test_whole_tiles(cuda, rows, m, n, k):
    check(cuda, rows, False, m, n, k, False)


@pytest.mark.parametrize("rows", [256, 512])
@pytest.mark.parametrize("m,n,k", [(129, 8, 8), (200, 136, 64), (257, 264, 256), (511, 128, 320), (513, 520, 392), (300, 18936, 1032)])
def test_whole_gated_tiles(cuda, rows, m, n, k):
    check(cuda, rows, False, m, n, k, True)


# few tiles, each cut among several clusters, the last slice of K a piece of eight; and tiles for one to three rounds and a rest that is cut
@pytest.mark.parametrize("rows", [256, 512])
@pytest.mark.parametrize("gated,m,n,k", [(False, 300, 264, 4104), (False, 257, 8, 5000), (False, 1281, 520, 5000), (False, 1281, 9720, 2056),
                                         (False, 1281, 9722, 2056), (True, 300, 136, 4104), (True, 1281, 264, 5000), (True, 1281, 4856, 2056)])
def test_cut_tiles(cuda, rows, gated, m, n, k):
    check(cuda, rows, True, m, n, k, gated)


@pytest.mark.parametrize("rows", [256, 512])
@pytest.mark.parametrize("cut", [False, True])
def test_infinities_and_nan_stay_in_their_rows(cuda, rows, cut):
    cuda.use_torch_stream()
    x, w, _, _, _ = operands(600, 520, 5000, torch.bfloat16, 9)
    clean = product(cuda, rows, cut, x, w)
    x2 = x.clone()
    x2[599, 5], x2[300, 4990] = float("nan"), float("inf")
    out = product(cuda, rows, cut, x2, w)
    assert torch.isnan(out[599]).all() and not torch.isfinite(out[300]).any()
    keep = [i for i in range(600) if i not in (300, 599)]
    assert torch.equal(out[keep], clean[keep])
