"""The fp32-arithmetic kernels (float32 layers of any width, 16-bit layers of odd widths) at the edges of their tiles:
channel counts around the column groups of 8 / 16 / 32 / 64 and the steps of 32 input channels, output channels beyond one
tile of 64, kernel volumes beyond one batch of lists, full tiles (more than 64 pairs per offset) and nearly empty ones."""
import numpy as np
import pytest
import torch

from oracle import conv_np
from sphconv_b200 import check_status
from sphconv_b200 import sphconv_cuda as ops
from test_gpu_conv import TOL, _close, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iC,oC", [(1, 1), (33, 9), (36, 17), (31, 33), (40, 64), (64, 32), (65, 68), (20, 130)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dens,ks", [(1.0, (3, 3, 3)), (0.01, (3, 3, 3)), (0.4, (5, 3, 3))])
def test_forward_and_gradients(iC, oC, dtype, dens, ks):
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(1, [9, 13, 12], True, dens, 11, iC, oC, dtype, ks)
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    _close(ops.rule_conv(feat, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[dtype])
    g = torch.as_tensor(rng.standard_normal((n_out, oC)), dtype=torch.float32).to(dtype).cuda()
    g64 = g.double().cpu().numpy()
    dx = ops.rule_conv_d_feature(g, w.permute(0, 2, 1).contiguous(), rules, rule_size, [5, 7], n_in)
    _close(dx, conv_np.conv_dgrad(g64, w64, pairs, n_in), TOL[dtype])
    if iC <= 64 and oC <= 64:
        dw = ops.rule_conv_d_weight(feat, g, rules, rule_size)
        ref = conv_np.conv_wgrad(f64, g64, pairs, int(np.prod(ks)))
        _close(dw, ref, 1e-4 if dtype == torch.float32 else 1e-3)


@pytest.mark.parametrize("iC,oC", [(5, 5), (8, 8), (4, 64), (7, 64), (9, 16), (16, 8), (12, 40), (16, 17), (24, 24)])
@pytest.mark.parametrize("dens", [1.0, 0.02])
def test_narrow_float32_rows(iC, oC, dens):
    """Rows of up to 8 and 16 channels take steps of that width with more of them in flight; small products have up to 256
    copies whose sum is folded within the warps."""
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(2, [9, 17, 12], True, dens, 3, iC, oC, torch.float32, (3, 3, 3))
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    _close(ops.rule_conv(feat, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[torch.float32])
    g = torch.as_tensor(rng.standard_normal((n_out, oC)), dtype=torch.float32).cuda()
    dw = ops.rule_conv_d_weight(feat, g, rules, rule_size)
    _close(dw, conv_np.conv_wgrad(f64, g.double().cpu().numpy(), pairs, 27), 1e-4)


@pytest.mark.parametrize("iC,oC", [(17, 9), (20, 12), (32, 32), (33, 10), (37, 64), (40, 66)])
@pytest.mark.parametrize("dens,ks", [(0.02, (3, 3, 3)), (0.07, (3, 3, 3)), (0.1, (3, 3, 3)), (0.15, (1, 3, 3)), (0.05, (5, 5, 5))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_sparse_and_dense_tiles(iC, oC, dens, ks, dtype):
    """Around two pairs a row, tiles of one layer go to either kernel; each must take exactly what the other leaves."""
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(2, [17, 23, 16], True, dens, 5, iC, oC, dtype, ks)
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    _close(ops.rule_conv(feat, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[dtype])


@pytest.mark.parametrize("iC,oC,dtype", [(9, 16, torch.float32), (3, 16, torch.float32), (12, 40, torch.float32), (24, 40, torch.float32),
                                         (33, 64, torch.float16), (48, 40, torch.bfloat16), (40, 130, torch.float16)])
@pytest.mark.parametrize("dens,ks", [(0.03, (3, 3, 3)), (1.0, (3, 3, 3)), (0.3, (5, 5, 3)), (0.3, (1, 1, 1)), (0.1, (7, 7, 7))])
def test_layers_walked_whole(iC, oC, dtype, dens, ks):
    """Layers whose padding makes staging dear are walked whatever their tiles hold: kernel volumes of one to many words of
    offsets, and an entry that is no row."""
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(1, [11, 13, 9], True, dens, 5, iC, oC, dtype, ks)
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    x = torch.cat([feat.new_zeros(1), feat.flatten()])[1:].view_as(feat)         # off a 16-byte boundary: no other kernel
    _close(ops.rule_conv(x, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[dtype])
    nbr = rules._sph.nbr.clone()
    nbr[0][nbr[0] < 0] = n_in
    got = ops._gather(x, w, nbr, n_out, False, None, None, False, None)
    assert torch.equal(got, ops._gather(x, w, rules._sph.nbr, n_out, False, None, None, False, None))
    if bool((rules._sph.nbr[0] < 0).any()):
        with pytest.raises(RuntimeError):
            check_status()


@pytest.mark.parametrize("iC,oC", [(64, 64), (62, 61), (31, 30), (48, 60)])
@pytest.mark.parametrize("dens,ks", [(0.02, (3, 3, 3)), (0.07, (3, 3, 3)), (0.15, (5, 3, 3))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_tiles_shared_at_widths_that_fill_their_tiles(iC, oC, dens, ks, dtype):
    """Widths with little padding, whose tiles do go to either kernel (padded ones of this size are walked whole)."""
    rng, feat, w, rules, rule_size, pairs, n_in, n_out = _setup(2, [17, 23, 16], True, dens, 5, iC, oC, dtype, ks)
    f64, w64 = feat.double().cpu().numpy(), w.double().cpu().numpy()
    _close(ops.rule_conv(feat, w, rules, rule_size, n_out), conv_np.conv_forward(f64, w64, pairs, n_out), TOL[dtype])


@pytest.mark.parametrize("iC,oC,dtype", [(32, 32, torch.float32), (24, 40, torch.float32), (9, 16, torch.float32), (64, 64, torch.float16),
                                         (48, 40, torch.float16), (64, 33, torch.bfloat16)])
@pytest.mark.parametrize("kv", [27, 45])
def test_layers_larger_than_the_machine(iC, oC, dtype, kv):
    """80 k rows (the rules for large layers), tiles of half a pair to eight pairs a row side by side."""
    g = torch.Generator(device="cuda").manual_seed(iC + kv)
    n = 80123
    share = torch.rand(kv, n // 128 + 1, generator=g, device="cuda").pow(3).repeat_interleave(128, 1)[:, :n] * 0.5
    nbr = torch.randint(0, n, (kv, n), generator=g, device="cuda", dtype=torch.int32)
    nbr[torch.rand(kv, n, generator=g, device="cuda") > share] = -1
    x = torch.randn(n, iC, generator=g, device="cuda").to(dtype)
    w = (torch.randn(kv, iC, oC, generator=g, device="cuda") / (4 * iC) ** 0.5).to(dtype)
    want = torch.zeros(n, oC, dtype=torch.float64, device="cuda")
    for k in range(kv):
        m = nbr[k] >= 0
        want[m] += x.double()[nbr[k][m].long()] @ w[k].double()
    _close(ops._gather(x, w, nbr, n, False, None, None, False, torch.float32), want.cpu().numpy(), TOL[dtype])
    assert check_status() == 0
