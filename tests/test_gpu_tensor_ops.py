"""COO -> range-voxel and range-voxel <-> dense on the GPU (through the C ABI) against the CPU restatement, for every
dtype and for row widths that exercise the 16- / 4- / 2- / 1-byte copy paths."""
import numpy as np
import pytest
import torch

from oracle import tensor_np
from sphconv_b200 import check_status
from sphconv_b200 import sphconv_cuda as ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _coo(rng, B, shape, dens):
    occ = rng.random((B, *shape)) < dens
    idx = np.stack(np.nonzero(occ), axis=1).astype(np.int32)
    rng.shuffle(idx)
    return idx


@pytest.mark.parametrize("dtype,C", [(torch.float32, 4), (torch.float32, 5), (torch.float16, 8), (torch.float16, 3),
                                     (torch.bfloat16, 64), (torch.int8, 7), (torch.int8, 32), (torch.float64, 2)])
def test_ops_match_oracle(dtype, C):
    rng = np.random.default_rng(C + 1)
    B, shape = 3, [6, 9, 70]
    idx = _coo(rng, B, shape, 0.2)
    if dtype == torch.int8:
        feat = torch.as_tensor(rng.integers(-100, 100, (idx.shape[0], C)), dtype=dtype)
    else:
        feat = torch.as_tensor(rng.standard_normal((idx.shape[0], C))).to(dtype)
    want_f, want_zi, want_zp, want_perm = tensor_np.init_tensor(feat.view(torch.uint8).numpy().reshape(idx.shape[0], -1),
                                                                idx, B, shape)
    f2, z_idx, z_ptr, perm = ops.init_tensor(feat.to(DEV), torch.as_tensor(idx, device=DEV), B, shape)
    assert (z_idx.cpu().numpy() == want_zi).all() and (z_ptr.cpu().numpy() == want_zp).all()
    assert (perm.cpu().numpy() == want_perm).all()
    assert (f2.cpu().view(torch.uint8).numpy().reshape(idx.shape[0], -1) == want_f).all()
    dense = torch.zeros((B, *shape, C), dtype=dtype, device=DEV)
    ops.to_dense(f2, z_idx, z_ptr, shape[2], dense)
    want_dense = tensor_np.to_dense(want_f, want_zi, want_zp, B, shape)
    assert (dense.cpu().view(torch.uint8).numpy().reshape(want_dense.shape) == want_dense).all()
    # backwards (pure row moves: bit-exact for every dtype)
    g = dense * 0 + torch.as_tensor(rng.integers(-3, 4, tuple(dense.shape)), device=DEV).to(dtype)
    rows_g = ops.to_dense_backward(g, z_idx, z_ptr)
    want_rows_g = tensor_np.to_dense_backward(g.cpu().view(torch.uint8).numpy().reshape(want_dense.shape), want_zi, want_zp)
    assert (rows_g.cpu().view(torch.uint8).numpy().reshape(want_rows_g.shape) == want_rows_g).all()
    back = ops.init_tensor_backward(rows_g, perm)
    want_back = tensor_np.init_tensor_backward(want_rows_g, want_perm)
    assert (back.cpu().view(torch.uint8).numpy().reshape(want_back.shape) == want_back).all()
    assert check_status() == 0


def test_empty_and_bad_coordinates():
    f2, z_idx, z_ptr, perm = ops.init_tensor(torch.zeros((0, 4), device=DEV), torch.zeros((0, 4), dtype=torch.int32, device=DEV),
                                             2, [3, 4, 5])
    assert f2.shape == (0, 4) and (z_ptr.cpu().numpy() == 0).all()
    idx = torch.tensor([[0, 1, 2, 3], [0, 1, 2, 9], [5, 0, 0, 0]], dtype=torch.int32, device=DEV)   # two rows out of range
    f2, z_idx, z_ptr, perm = ops.init_tensor(torch.ones((3, 2), device=DEV), idx, 2, [3, 4, 5])
    assert perm.cpu().tolist() == [0, -1, -1] and int(z_ptr.reshape(-1)[-1]) == 1
    with pytest.raises(RuntimeError):      # SPH_STATUS_BAD_INDEX is reported (and cleared) by the status read
        check_status()
    assert check_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("C,n", [(16, 1000), (64, 12345), (32, 7), (128, 300)])
def test_epilogue_backward(dtype, C, n):
    """Gradient mask of relu(acc + bias) and the bias gradient in one pass, against the torch expressions."""
    g = torch.Generator(device=DEV).manual_seed(C + n)
    out = torch.relu(torch.randn((n, C), generator=g, device=DEV)).to(dtype)
    d_out = torch.randn((n, C), generator=g, device=DEV).to(dtype)
    for relu in (True, False):
        d_pre, d_bias = ops.epilogue_backward(d_out, out, relu, True)
        want = torch.where(out > 0, d_out, torch.zeros((), dtype=dtype, device=DEV)) if relu else d_out
        assert torch.equal(d_pre, want)
        ref = want.double().sum(0)
        assert torch.allclose(d_bias.double(), ref, rtol=1e-4, atol=1e-3 * max(1.0, float(ref.abs().max())))
    d_pre, d_bias = ops.epilogue_backward(d_out, out, True, False)
    assert d_bias is None and torch.equal(d_pre, torch.where(out > 0, d_out, torch.zeros((), dtype=dtype, device=DEV)))


@pytest.mark.parametrize("dtype,C", [(torch.float16, 64), (torch.float16, 3), (torch.float32, 5), (torch.int8, 6), (torch.float64, 2),
                                     (torch.bfloat16, 130)])
@pytest.mark.parametrize("shape,dens", [([5, 7, 16], 0.3), ([3, 9, 13], 1.0), ([2, 3, 300], 0.1), ([1, 2, 2048], 0.5), ([4, 4, 1], 0.5)])
def test_dense_channels_first_matches_two_step(dtype, C, shape, dens):
    """The one-pass channels-first dense tensor and its gradient against the channels-last operator and torch's permute, at
    depths on either side of the block size, odd volumes (no 16-byte vectors) and rows wider than one chunk."""
    rng = np.random.default_rng(C)
    idx = torch.as_tensor(_coo(rng, 2, shape, dens), device=DEV)
    feat = torch.as_tensor(rng.integers(-100, 100, (idx.shape[0], C)), device=DEV).to(dtype)
    f, z_idx, z_ptr, _ = ops.init_tensor(feat, idx, 2, shape)
    want = torch.zeros((2, *shape, C), dtype=dtype, device=DEV)
    ops.to_dense(f, z_idx, z_ptr, shape[2], want)
    got = ops.dense_channels_first(f, z_idx, z_ptr, [2, C, *shape])
    assert torch.equal(got, want.permute(0, 4, 1, 2, 3))
    assert torch.equal(ops.dense_channels_first_backward(got, z_idx, z_ptr), f)
    assert check_status() == 0


@pytest.mark.parametrize("dtype,C", [(torch.float16, 64), (torch.float16, 3), (torch.float32, 5), (torch.int8, 6), (torch.bfloat16, 130)])
@pytest.mark.parametrize("shape,per_column", [([5, 7, 16], 9), ([3, 9, 13], 40), ([2, 3, 300], 700), ([1, 2, 2048], 2500)])
def test_dense_channels_first_rows_without_a_cell_of_their_own(dtype, C, shape, per_column):
    """Repeated depths - some blocks with more rows than cells - against the oracle (the last row of a depth is the cell's value,
    each of them gets its gradient), then with depths outside the grid (status bit, gradient zero) and with rows behind the
    last column's (gradient zero)."""
    rng = np.random.default_rng(C + per_column)
    B, (H, W, D) = 2, shape
    counts = rng.integers(0, per_column + 1, (B, H, W))
    counts[0, 0, 0] = per_column
    z_ptr = counts.reshape(-1).cumsum().astype(np.int32).reshape(B, H, W)
    n = int(z_ptr[-1, -1, -1])
    z_idx = rng.integers(0, D, n).astype(np.int32)
    feat = torch.as_tensor(rng.integers(-100, 100, (n, C))).to(dtype)
    grad = torch.as_tensor(rng.integers(-100, 100, (B, C, *shape))).to(dtype)
    zi, zp = torch.as_tensor(z_idx, device=DEV), torch.as_tensor(z_ptr, device=DEV)

    def dense(rows, depths, ptr):
        return torch.as_tensor(tensor_np.to_dense(rows.double().numpy(), depths, ptr, B, shape)).permute(0, 4, 1, 2, 3)

    def back(depths, ptr):
        d = grad.double().permute(0, 2, 3, 4, 1).numpy()
        return torch.as_tensor(tensor_np.to_dense_backward(d, depths, ptr))

    got = ops.dense_channels_first(feat.to(DEV), zi, zp, [B, C, *shape])
    assert torch.equal(got.cpu().double(), dense(feat, z_idx, z_ptr))
    got = ops.dense_channels_first_backward(grad.to(DEV), zi, zp)
    assert torch.equal(got.cpu().double(), back(z_idx, z_ptr))
    longer = torch.cat([zi, torch.zeros(3, dtype=torch.int32, device=DEV)])
    got = ops.dense_channels_first_backward(grad.to(DEV), longer, zp)
    assert torch.equal(got[:n].cpu().double(), back(z_idx, z_ptr)) and not got[n:].any()
    assert check_status() == 0

    out = rng.random(n) < 0.1
    out[0] = True
    column = np.repeat(np.arange(B * H * W), counts.reshape(-1))[~out]
    ptr = np.bincount(column, minlength=B * H * W).cumsum().astype(np.int32).reshape(B, H, W)
    bad = torch.as_tensor(np.where(out, np.where(rng.random(n) < 0.5, D, -1), z_idx).astype(np.int32), device=DEV)
    got = ops.dense_channels_first(feat.to(DEV), bad, zp, [B, C, *shape])
    assert torch.equal(got.cpu().double(), dense(feat[torch.as_tensor(~out)], z_idx[~out], ptr))
    got = ops.dense_channels_first_backward(grad.to(DEV), bad, zp)
    assert torch.equal(got[~out].cpu().double(), back(z_idx[~out], ptr)) and not got[out].any()
    with pytest.raises(RuntimeError):
        check_status()


def test_one_kernel_with_two_sizes_from_two_threads():
    """Launches of one kernel that take 8 and 70 KB of shared memory, through the C ABI from two threads at once: neither
    lowers the bound the other one needs."""
    import threading

    from sphconv_b200 import _capi as C
    lib, errors = C.lib(), []
    gate = threading.Barrier(2)

    def work(C_, D):
        torch.cuda.set_device(0)
        H, W = 2, 4
        zi = torch.zeros(H * W, dtype=torch.int32, device=DEV)
        zp = torch.arange(1, H * W + 1, dtype=torch.int32, device=DEV)
        rows = torch.ones(H * W, C_, dtype=torch.float16, device=DEV)
        dense = torch.empty(1, C_, H, W, D, dtype=torch.float16, device=DEV)
        torch.cuda.synchronize()
        shape = ops._shape3([H, W, D])
        gate.wait()
        for _ in range(3000):
            rc = lib.sph_dense_channels_first(C.ptr(rows), 2, C_, H * W, C.ptr(zi), C.ptr(zp), 1, shape, C.ptr(dense), 0, None,
                                              C.stream_ptr(zi.device))
            if rc != 0:
                errors.append(lib.sph_last_error().decode())
                return
        torch.cuda.synchronize()
        if float(dense.sum()) != H * W * C_:
            errors.append("wrong values")

    threads = [threading.Thread(target=work, args=a) for a in ((4, 512), (64, 512))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("dtype,C", [(torch.float16, 2), (torch.float16, 33), (torch.float16, 64), (torch.float32, 1), (torch.int8, 12),
                                     (torch.float16, 400)])
@pytest.mark.parametrize("shift", [0, 1])
def test_dense_rows_copied_ahead(dtype, C, shift):
    """Rows that are whole 4-byte words (copied while the map of the cells is made) and rows that are not, or do not start on
    one; more channels than a block stages at a time."""
    g = torch.Generator(device="cuda").manual_seed(C)
    B, H, W, D = 2, 5, 9, 48
    m = torch.rand(B, H, W, D, device="cuda", generator=g) < 0.3
    at = m.nonzero()
    z_idx, z_ptr = at[:, 3].int().contiguous(), m.sum(-1).view(-1).cumsum(0).int().view(B, H, W)
    n = at.shape[0]
    memory = torch.randint(-100, 100, (n * C + 1,), device="cuda", generator=g).to(dtype)
    rows = memory[shift:shift + n * C].view(n, C)
    dense = ops.dense_channels_first(rows, z_idx, z_ptr, [B, C, H, W, D])
    want = torch.zeros(B, C, H, W, D, dtype=dtype, device="cuda")
    want.permute(0, 2, 3, 4, 1)[m] = rows
    assert torch.equal(dense, want)
    assert torch.equal(ops.dense_channels_first_backward(dense, z_idx, z_ptr), rows)


@pytest.mark.parametrize("dtype,C", [(torch.float32, 1), (torch.int8, 12), (torch.float16, 3), (torch.float32, 4), (torch.int8, 1)])
@pytest.mark.parametrize("B,H,W,D", [(2, 40, 1001, 64), (1, 50, 1003, 100), (3, 7, 300, 900), (1, 3, 1100, 2000)])
def test_dense_of_narrow_rows_on_large_grids(dtype, C, B, H, W, D):
    """Blocks of up to 2048 cells: several columns, a last block with fewer, columns of more than half a block."""
    g = torch.Generator(device="cuda").manual_seed(D)
    at = torch.rand(B, H, W, D, device="cuda", generator=g)
    m = (at < 0.03) & (torch.rand(B, H, W, 1, device="cuda", generator=g) < 0.7)
    z_idx, z_ptr = m.nonzero()[:, 3].int().contiguous(), m.sum(-1).view(-1).cumsum(0).int().view(B, H, W)
    rows = torch.randint(-100, 100, (z_idx.numel(), C), device="cuda", generator=g).to(dtype)
    dense = ops.dense_channels_first(rows, z_idx, z_ptr, [B, C, H, W, D])
    want = torch.zeros(B, C, H, W, D, dtype=dtype, device="cuda")
    want.permute(0, 2, 3, 4, 1)[m] = rows
    assert torch.equal(dense, want)
    grad = torch.randint(-100, 100, (B, C, H, W, D), device="cuda", generator=g).to(dtype)
    assert torch.equal(ops.dense_channels_first_backward(grad, z_idx, z_ptr), grad.permute(0, 2, 3, 4, 1)[m])
