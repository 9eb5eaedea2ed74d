"""The strip kernel against a dense float64 / integer sum over the table, where it can go wrong: rows of widths that end
inside a 16-byte unit (pieces of 8, 4, 2 and 1 bytes), output widths around its tiles, row counts around a tile of 256, more
than one group of offsets, tables whose rows do not fit a buffer (operands from global memory), the end of a line of columns
inside a tile (two windows), entries that are no rows."""
import numpy as np
import pytest
import torch

from sphconv_b200 import _capi as C
from sphconv_b200 import check_status
from sphconv_b200 import sphconv_cuda as ops
from oracle import conv_np
from test_gpu_conv import TOL, _close, _setup

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _operands(rng, n_in, kv, K, N, dtype):
    if dtype == torch.int8:
        x, w = (torch.as_tensor(rng.integers(-127, 128, s), dtype=dtype, device=DEV) for s in ((n_in, K), (kv, K, N)))
    else:
        x = torch.as_tensor(rng.standard_normal((n_in, K)), device=DEV).to(dtype)
        w = torch.as_tensor(rng.uniform(-1, 1, (kv, K, N)) / np.sqrt(4 * K), device=DEV).to(dtype)
    return x, w


def _reference(x, w, nbr):
    out = torch.zeros((nbr.shape[1], w.shape[2]), dtype=torch.float64, device=DEV)
    for k in range(w.shape[0]):
        m = nbr[k] >= 0
        out[m] += x.double()[nbr[k][m].long()] @ w[k].double()
    return out.cpu().numpy()


def _check(x, w, nbr, flip=False):
    got = ops._gather(x, w, nbr.flip(0).contiguous() if flip else nbr, nbr.shape[1], flip, None, None, False, torch.float32)
    _close(got, _reference(x, w, nbr), 0.0 if x.dtype == torch.int8 else TOL[x.dtype])
    assert check_status() == 0


@pytest.mark.parametrize("K,N", [(16, 16), (16, 8), (20, 32), (37, 11), (40, 7), (12, 33), (64, 20), (32, 57), (1, 1), (24, 40)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.int8])
@pytest.mark.parametrize("n_out,spread", [(1, 1), (255, 40), (257, 40), (1500, 100000)])
def test_local_and_scattered_tables(K, N, dtype, n_out, spread):
    """Entries near the diagonal (one window) and spread over 100 k rows (no buffer holds them)."""
    rng = np.random.default_rng(K * 100 + N)
    n_in = n_out + spread
    nbr = np.arange(n_out)[None, :] + rng.integers(0, spread + 1, (27, n_out))
    nbr[rng.random((27, n_out)) < 0.5] = -1
    x, w = _operands(rng, n_in, 27, K, N, dtype)
    _check(x, w, torch.as_tensor(nbr.astype(np.int32), device=DEV), flip=n_out == 257)


@pytest.mark.parametrize("kv", [1, 9, 10, 45])
@pytest.mark.parametrize("jump", [5000, 100000])
def test_two_windows_and_groups(kv, jump):
    """A jump of the input rows inside the first tile and behind it."""
    rng = np.random.default_rng(kv)
    n_out = 700
    at = np.arange(n_out) + np.where(np.arange(n_out) >= 100, jump, 0) + np.where(np.arange(n_out) >= 640, jump, 0)
    nbr = at[None, :] + rng.integers(0, 60, (kv, n_out))
    nbr[rng.random((kv, n_out)) < 0.6] = -1
    x, w = _operands(rng, n_out + 2 * jump + 60, kv, 24, 24, torch.float16)
    _check(x, w, torch.as_tensor(nbr.astype(np.int32), device=DEV))


@pytest.mark.parametrize("K,N", [(16, 16), (4, 16), (37, 11), (64, 24), (45, 51), (33, 64), (32, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("n_out,spread,kv", [(1, 1, 27), (257, 40, 27), (1500, 100000, 10), (3000, 30, 45)])
def test_weight_gradient_tables(K, N, dtype, n_out, spread, kv):
    """The pairs' weight gradient on the same kinds of table; one offset has every row, as the centre of a layer does."""
    rng = np.random.default_rng(K + N)
    n_in = n_out + spread
    nbr = np.arange(n_out)[None, :] + rng.integers(0, spread + 1, (kv, n_out))
    nbr[rng.random((kv, n_out)) < 0.8] = -1
    nbr[kv // 2] = np.arange(n_out)
    t = torch.as_tensor(nbr.astype(np.int32), device=DEV)
    x, _ = _operands(rng, n_in, 1, K, N, dtype)
    g, _ = _operands(rng, n_out, 1, N, K, dtype)
    dw = C.host().conv_wgrad(x, g, t, None, False)
    want = torch.stack([x.double()[t[k][t[k] >= 0].long()].T @ g.double()[t[k] >= 0] for k in range(kv)])
    assert float((dw.double() - want).abs().max()) <= 1e-4 * max(1.0, float(want.abs().max()))
    assert check_status() == 0


def test_entries_that_are_no_rows():
    rng = np.random.default_rng(3)
    x, w = _operands(rng, 300, 27, 16, 16, torch.float16)
    nbr = torch.as_tensor(rng.integers(-1, 300, (27, 300)).astype(np.int32), device=DEV)
    want = ops._gather(x, w, nbr, 300, False, None, None, False, None)
    spoiled = nbr.clone()
    spoiled[nbr < 0] = 300
    spoiled[5][nbr[5] < 0] = -7
    got = ops._gather(x, w, spoiled, 300, False, None, None, False, None)
    assert torch.equal(got, want)
    with pytest.raises(RuntimeError):
        check_status()
    assert check_status() == 0 and C.lib() is not None


@pytest.mark.parametrize("flip", [False, True])
def test_tables_of_more_than_2_to_the_32_entries(flip):
    """Entries at both ends of the planes on either side of the 2^32nd; every other row has no neighbour."""
    kv, n_out = 27, (1 << 32) // 27 + 300
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of device memory")
    rng = np.random.default_rng(5)
    x, w = _operands(rng, 100, kv, 16, 4, torch.float16)
    at = torch.cat([torch.arange(300), torch.arange(n_out - 600, n_out)]).to(DEV)
    some = torch.as_tensor(rng.integers(-1, 100, (kv, at.numel())).astype(np.int32), device=DEV)
    nbr = torch.full((kv, n_out), -1, dtype=torch.int32, device=DEV)
    nbr[:, at] = some
    got = ops._gather(x, w, nbr, n_out, flip, None, None, False, torch.float32)
    _close(got[at], _reference(x, w, some.flip(0) if flip else some), TOL[torch.float16])
    assert int(torch.count_nonzero(got)) == int(torch.count_nonzero(got[at]))
    assert check_status() == 0


@pytest.mark.parametrize("iC,oC", [(16, 16), (4, 16), (24, 40), (5, 7), (32, 64)])
@pytest.mark.parametrize("ks,subm", [((3, 3, 1), True), ((3, 1, 3), True), ((3, 1, 1), True), ((3, 3, 3), False)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_filters_whose_groups_span_lines_of_columns(iC, oC, ks, subm, dtype):
    """Nine consecutive offsets in three lines of 1500 rows, and input gradients of strided layers, in both directions."""
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(1, [5, 300, 16], subm, 0.3, 17, iC, oC, dtype, ks)
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    _close(ops.rule_conv(feat, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[dtype])
    g = torch.as_tensor(rng.standard_normal((n_out, oC)), dtype=torch.float32).to(dtype).to(DEV)
    g64 = g.double().cpu().numpy()
    dx = ops.rule_conv_d_feature(g, w.permute(0, 2, 1).contiguous(), rules, rule_size, [3, 150], n_in)
    _close(dx, conv_np.conv_dgrad(g64, w64, pairs, n_in), TOL[dtype])
    dw = ops.rule_conv_d_weight(feat, g, rules, rule_size)
    want = conv_np.conv_wgrad(f64, g64, pairs, int(np.prod(ks)))
    assert np.abs(dw.double().cpu().numpy() - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
    assert check_status() == 0
