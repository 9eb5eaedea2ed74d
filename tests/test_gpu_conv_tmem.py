"""The tcgen05 kernel with the gathered rows in tensor memory (9 and 27 offsets), against a plain PyTorch fp32 reference and,
bit for bit, against the kernels that gather into shared memory: those run the same layer when an offset without pairs is
added to its table (10 and 28 offsets), and sum in the same order."""
import numpy as np
import pytest
import torch

from sphconv_b200 import _capi as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CODE = {torch.float16: C.SPH_F16, torch.bfloat16: C.SPH_BF16, torch.int8: C.SPH_I8, torch.float32: C.SPH_F32}


def _gather(rows, weight, nbr, flip=False, bias=None, relu=False, out_dtype=None):
    lib, st = C.lib(), C.stream_ptr(torch.device(DEV))
    kv, K, N = weight.shape
    code = CODE[rows.dtype]
    packed = torch.empty(lib.sph_packed_weight_bytes(code, kv, K, N), dtype=torch.uint8, device=DEV)
    assert lib.sph_pack_weight(C.ptr(weight), code, kv, K, N, C.ptr(packed), st) == 0
    out = torch.empty(nbr.shape[1], N, dtype=out_dtype or (torch.float32 if rows.dtype == torch.int8 else rows.dtype), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    rc = lib.sph_conv_gather(C.ptr(rows), code, rows.shape[0], C.ptr(weight), C.ptr(packed), C.ptr(nbr), nbr.shape[1], kv, K, N,
                             int(flip), None, C.ptr(bias) if bias is not None else None, int(relu), C.ptr(out), CODE[out.dtype],
                             C.ptr(status), st)
    assert rc == 0, lib.sph_last_error()
    torch.cuda.synchronize()
    return out, int(status.item())


def _operands(K, N, dtype, n_rows, kv, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if dtype == torch.int8:
        return (torch.randint(-127, 128, (n_rows, K), device=DEV, dtype=dtype, generator=g),
                torch.randint(-127, 128, (kv, K, N), device=DEV, dtype=dtype, generator=g))
    return (torch.randn(n_rows, K, device=DEV, generator=g).to(dtype), (torch.randn(kv, K, N, device=DEV, generator=g) * 0.1).to(dtype))


def _table(kv, n_out, n_rows, spread, share, seed):
    """Entries within `spread` rows of where the output row's own position falls, `share` of them present."""
    g = np.random.default_rng(seed)
    at = np.arange(n_out) * n_rows // max(n_out, 1)
    t = np.clip(at[None] + g.integers(-spread, spread + 1, (kv, n_out)), 0, n_rows - 1)
    t[g.random((kv, n_out)) >= share] = -1
    return torch.as_tensor(t, dtype=torch.int32, device=DEV)


def _check(rows, weight, nbr, flip=False, **more):
    kv, K, N = weight.shape
    code = CODE[rows.dtype]
    assert C.lib().sph_conv_uses_tmem(code, kv, K, N) and not C.lib().sph_conv_uses_tmem(code, kv + 1, K, N)
    out, status = _gather(rows, weight, nbr, flip, **more)
    assert status == 0
    none = torch.full((1, nbr.shape[1]), -1, dtype=torch.int32, device=DEV)
    wider = torch.cat([weight, torch.zeros_like(weight[:1])])
    other, status = _gather(rows, wider, torch.cat([none, nbr] if flip else [nbr, none]).contiguous(), flip, **more)
    assert status == 0
    assert torch.equal(out, other)
    ref = torch.zeros(nbr.shape[1], N, dtype=torch.float64, device=DEV)
    for k in range(kv):
        idx = nbr[kv - 1 - k if flip else k].long()
        m = idx >= 0
        ref[m] += rows[idx[m]].double() @ weight[k].double()
    if more.get("bias") is not None:
        ref += more["bias"].double()
    if more.get("relu"):
        ref.clamp_(min=0)
    # sums of at most 27 * 64 products in 32 bits (int8: exact), then one rounding to the output's type
    eps = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}[out.dtype]
    scale = ref.abs().max().clamp_min(1)
    assert ((out.double() - ref).abs() <= eps * ref.abs() * 1.01 + (0 if rows.dtype == torch.int8 else 2.0 ** -17 * scale)).all()


@pytest.mark.parametrize("K,N,dtype", [(16, 32, torch.float16), (32, 16, torch.bfloat16), (32, 32, torch.float16), (32, 64, torch.bfloat16),
                                       (64, 64, torch.float16), (64, 48, torch.bfloat16), (32, 32, torch.int8), (64, 64, torch.int8),
                                       (128, 32, torch.int8)])
@pytest.mark.parametrize("n_out,n_rows,kv", [(1, 1, 27), (127, 40, 27), (129, 300, 9), (257, 257, 27), (19000, 30000, 27), (40000, 25000, 9),
                                             (150000, 150000, 27)])
def test_local_tables(K, N, dtype, n_out, n_rows, kv):
    rows, weight = _operands(K, N, dtype, n_rows, kv, n_out)
    _check(rows, weight, _table(kv, n_out, n_rows, 60, 0.4, kv), flip=n_out % 2 == 1)


@pytest.mark.parametrize("K,N,dtype", [(16, 32, torch.float16), (32, 32, torch.bfloat16), (64, 64, torch.float16), (128, 64, torch.int8)])
@pytest.mark.parametrize("spread", [400, 1200, 40000])
def test_runs_longer_than_their_buffer(K, N, dtype, spread):
    rows, weight = _operands(K, N, dtype, 40000, 27, 1)
    _check(rows, weight, _table(27, 30000, 40000, spread, 0.5, 2))


@pytest.mark.parametrize("K,N,dtype", [(16, 32, torch.float16), (32, 64, torch.bfloat16), (64, 64, torch.float16), (32, 32, torch.int8)])
@pytest.mark.parametrize("n_out,kv", [(5000, 27), (20001, 27), (20001, 9)])
@pytest.mark.parametrize("shift", [0, 16])
def test_tables_without_locality(K, N, dtype, n_out, kv, shift):
    """Runs that are not brought to shared memory at all; rows that start on a multiple of 16 bytes, but not of 32; more input rows
    than output rows and fewer; entries that are no rows among those that the gather reads itself."""
    for n_rows in (200000, n_out // 2):
        rows, weight = _operands(K, N, dtype, n_rows, kv, 11)
        memory = torch.empty(rows.numel() + 16, dtype=dtype, device=DEV)
        off = shift // rows.element_size()
        rows = memory[off:off + rows.numel()].view_as(rows).copy_(rows)
        assert rows.data_ptr() % 32 == shift
        nbr = _table(kv, n_out, n_rows, n_rows, 0.5, 12)
        nbr[:, n_out // 2:] = _table(kv, n_out - n_out // 2, n_rows, 700, 0.5, 13)      # every second row's runs a little too long
        _check(rows, weight, nbr, flip=kv == 9)
        bad = nbr.clone()
        bad[1, ::7], bad[kv - 1, 5::9], bad[kv // 2, 3::8] = n_rows, n_rows + 100, -5
        nbr[1, ::7], nbr[kv - 1, 5::9], nbr[kv // 2, 3::8] = -1, -1, -1
        out, status = _gather(rows, weight, bad)
        assert status & C.STATUS_BAD_INDEX
        assert torch.equal(out, _gather(rows, weight, nbr)[0])


@pytest.mark.parametrize("K,N,dtype", [(16, 32, torch.float16), (32, 32, torch.float16), (64, 64, torch.float16), (64, 64, torch.int8)])
def test_offsets_and_tiles_without_pairs(K, N, dtype):
    """Offsets that tiles, or halves of tiles, do not have; tiles and whole tables without any pair."""
    rows, weight = _operands(K, N, dtype, 60000, 27, 3)
    nbr = _table(27, 60000, 60000, 50, 0.3, 4)
    tile = torch.arange(60000, device=DEV) // 128
    for k in range(27):
        nbr[k][(tile * 7 + k) % 5 < 3] = -1
    nbr[:, (tile > 100) & (tile < 140)] = -1
    nbr[:9, tile % 9 == 4] = -1
    _check(rows, weight, nbr)
    _check(rows, weight, torch.full_like(nbr, -1))


def test_bias_relu_and_output_types():
    bias = torch.randn(32, device=DEV)
    for dtype, outs in ((torch.float16, (torch.float16, torch.float32, torch.bfloat16)), (torch.int8, (torch.float32, torch.bfloat16))):
        rows, weight = _operands(32, 32, dtype, 5000, 27, 5)
        for out in outs:
            _check(rows, weight, _table(27, 5000, 5000, 40, 0.4, 6), bias=bias, relu=True, out_dtype=out)


def test_entries_that_are_no_rows():
    rows, weight = _operands(32, 32, torch.float16, 1000, 27, 7)
    nbr = _table(27, 1000, 1000, 40, 0.4, 8)
    bad = nbr.clone()
    bad[3, 17], bad[20, 999], bad[0, 0] = 1000, 2 ** 31 - 1, -7
    for k, o in ((3, 17), (20, 999), (0, 0)):
        nbr[k, o] = -1
    out, status = _gather(rows, weight, bad)
    assert status & C.STATUS_BAD_INDEX
    assert torch.equal(out, _gather(rows, weight, nbr)[0])
