"""Module-level API (SparseConvTensor, SubMConv3d, Conv3d, Sequential, autograd) against dense torch conv3d,
the ground truth of the reference's test/test_module.py, test/test_grad.py and test/test_util.py."""
import numpy as np
import pytest
import torch

import sphconv_b200 as sphconv
from oracle import dense_ref, rules_np
from sphconv_b200 import synthetic

from gpu_util import DEV

pytestmark = pytest.mark.gpu


def _coo(rng, B, shape, dens):
    occ = rng.random((B, *shape)) < dens
    idx = np.stack(np.nonzero(occ), axis=1).astype(np.int32)
    rng.shuffle(idx)                       # COO rows in arbitrary order
    return idx


def test_init_tensor_and_dense_roundtrip():
    rng = np.random.default_rng(0)
    B, shape, C = 3, [6, 7, 9], 5
    idx = _coo(rng, B, shape, 0.3)
    feat = rng.standard_normal((idx.shape[0], C)).astype(np.float32)
    t = sphconv.SparseConvTensor(torch.as_tensor(feat, device=DEV), shape, B, indices=torch.as_tensor(idx, device=DEV))
    # the reference's shape property is [B, C, D, H, W] with (D, W, H) = (s0, s1, s2) (sphconv/tensor.py:104-106)
    assert t.shape == [B, C, shape[0], shape[2], shape[1]]
    dense = t.dense().cpu()
    want = torch.zeros((B, C, *shape))
    want[idx[:, 0], :, idx[:, 1], idx[:, 2], idx[:, 3]] = torch.as_tensor(feat)
    assert torch.equal(dense, want)
    zp = t.z_ptr.cpu().numpy().reshape(-1)
    assert zp[-1] == idx.shape[0] and (np.diff(zp) >= 0).all()
    # gradient flows through dense() and the COO reorder back to the raw rows
    raw = torch.as_tensor(feat, device=DEV).requires_grad_(True)
    t2 = sphconv.SparseConvTensor(raw, shape, B, indices=torch.as_tensor(idx, device=DEV))
    g = torch.as_tensor(rng.standard_normal((B, C, *shape)).astype(np.float32), device=DEV)
    (t2.dense() * g).sum().backward()
    want_g = g.cpu()[idx[:, 0], :, idx[:, 1], idx[:, 2], idx[:, 3]]
    assert torch.allclose(raw.grad.cpu(), want_g)


@pytest.mark.parametrize("subm", [True, False])
@pytest.mark.parametrize("iC,oC", [(4, 16), (16, 16), (32, 64)])
def test_module_forward_backward_vs_dense(subm, iC, oC):
    rng = np.random.default_rng(1)
    B, shape = 2, [8, 10, 12]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3)
    feat = rng.standard_normal((z_idx.shape[0], iC)).astype(np.float32)
    if subm:
        layer = sphconv.SubMConv3d(iC, oC, 3, bias=False).to(DEV)
        st, pd = [1, 1, 1], [1, 1, 1]
    else:
        layer = sphconv.Conv3d(iC, oC, 3, stride=2, padding=1, bias=False).to(DEV)
        st, pd = [2, 2, 2], [1, 1, 1]
    f = torch.as_tensor(feat, device=DEV).requires_grad_(True)
    x = sphconv.SparseConvTensor(f, shape, B, z_idx=torch.as_tensor(z_idx, device=DEV), z_ptr=torch.as_tensor(z_ptr, device=DEV))
    y = layer(x)
    yd = y.dense()
    w5 = layer.weight.detach().cpu().numpy()
    up = rng.standard_normal(tuple(yd.shape)).astype(np.float32)
    if subm:   # gradient only at active sites
        mask = (dense_ref.densify(np.ones((z_idx.shape[0], 1), np.float32), z_idx, z_ptr, B, shape) != 0).numpy()
        up = up * mask
    (yd * torch.as_tensor(up, device=DEV)).sum().backward()
    ref_y, ref_dx, ref_dw = dense_ref.dense_conv_grads(feat, w5, lambda t: torch.as_tensor(up).double(), z_idx, z_ptr,
                                                       B, shape, st, pd)
    if subm:
        ref_y = ref_y * torch.as_tensor(mask)
    assert torch.allclose(yd.cpu().double(), ref_y, atol=1e-4)
    assert torch.allclose(f.grad.cpu().double(), ref_dx, atol=1e-4)
    assert torch.allclose(layer.weight.grad.cpu().double(), ref_dw, atol=1e-3)


def test_sequential_rule_cache_and_dense_modules():
    rng = np.random.default_rng(2)
    B, shape = 2, [8, 10, 12]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3)
    feat = torch.as_tensor(rng.standard_normal((z_idx.shape[0], 4)).astype(np.float32), device=DEV)
    net = sphconv.Sequential(
        sphconv.SubMConv3d(4, 16, 3, indice_key="subm0"), torch.nn.ReLU(),
        sphconv.SubMConv3d(16, 16, 3, indice_key="subm0"), torch.nn.ReLU(),
        sphconv.SparseConv3d(16, 32, 3, stride=2, padding=1),
    ).to(DEV)
    x = sphconv.SparseConvTensor(feat, shape, B, z_idx=torch.as_tensor(z_idx, device=DEV), z_ptr=torch.as_tensor(z_ptr, device=DEV))
    with torch.no_grad():
        y = net(x)
    assert "subm0" in y.rule_cache and len(y.rule_cache) == 1
    assert y.feature.shape[1] == 32 and [y.D, y.W, y.H] == [4, 5, 6]
    # dense reference of the same stack
    d = dense_ref.densify(feat.cpu().numpy(), z_idx, z_ptr, B, shape)
    mask = dense_ref.densify(np.ones((z_idx.shape[0], 1), np.float32), z_idx, z_ptr, B, shape) != 0
    convs = [m for m in net._modules.values() if isinstance(m, sphconv.Conv3d)]
    for i, m in enumerate(convs):
        w = m.weight.detach().cpu().permute(4, 3, 0, 1, 2).contiguous()
        if m.subm:
            d = torch.relu(torch.nn.functional.conv3d(d, w, None, 1, 1)) * mask
        else:
            d = torch.nn.functional.conv3d(d, w, None, 2, 1)
    assert torch.allclose(y.dense().cpu(), d, atol=1e-4)


def test_fused_bias_relu_extension_matches_unfused():
    rng = np.random.default_rng(3)
    B, shape = 1, [8, 10, 12]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3)
    feat = torch.as_tensor(rng.standard_normal((z_idx.shape[0], 16)).astype(np.float32), device=DEV).half()
    layer = sphconv.SubMConv3d(16, 32, 3, bias=True, apply_bias=True, activation='relu').to(DEV).half()
    plain = sphconv.SubMConv3d(16, 32, 3, bias=True).to(DEV).half()
    plain.load_state_dict(layer.state_dict())
    mk = lambda: sphconv.SparseConvTensor(feat, shape, B, z_idx=torch.as_tensor(z_idx, device=DEV), z_ptr=torch.as_tensor(z_ptr, device=DEV))
    with torch.no_grad():
        fused = layer(mk()).feature
        ref = torch.relu(plain(mk()).feature.float() + plain.bias.float())
    assert torch.allclose(fused.float(), ref, atol=2e-2, rtol=1e-2)
    # the reference applies no bias by default (sphconv/conv.py:182-185)
    with torch.no_grad():
        assert not torch.allclose(plain(mk()).feature.float(), ref)


def test_sequential_starts_strided_rules_ahead():
    """Sequential enqueues the first step of a strided layer's rule generation before the submanifold layer in front
    of it runs; outputs and rules are those of the layers called one by one."""
    from sphconv_b200 import sphconv_cuda as ops
    rng = np.random.default_rng(31)
    B, shape = 2, [12, 20, 16]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.25)
    feat = torch.as_tensor(rng.standard_normal((z_idx.shape[0], 16)), dtype=torch.float16, device=DEV)
    zi, zp = torch.as_tensor(z_idx, device=DEV), torch.as_tensor(z_ptr, device=DEV)
    torch.manual_seed(3)
    net = sphconv.Sequential(
        sphconv.SubMConv3d(16, 16, 3, indice_key="a", name="s0"),
        torch.nn.ReLU(),
        sphconv.SparseConv3d(16, 32, 3, stride=2, padding=1, name="d0"),
        sphconv.SubMConv3d(32, 32, 3, indice_key="b", name="s1"),
        sphconv.SparseConv3d(32, 32, 3, stride=2, padding=1, name="d1"),
    ).to(DEV).half().eval()
    calls = []
    real_begin = ops.get_rules_begin

    def spy(*a, **k):
        calls.append(a[0])
        return real_begin(*a, **k)

    ops.get_rules_begin = spy
    try:
        with torch.no_grad():
            x = sphconv.SparseConvTensor(feat, shape, B, z_idx=zi, z_ptr=zp)
            y = net(x)
            assert len(calls) == 2                      # one per strided layer, none repeated by get_rules
            assert not any(isinstance(k, tuple) for k in y.rule_cache)     # the handles were consumed
            t = sphconv.SparseConvTensor(feat, shape, B, z_idx=zi, z_ptr=zp)
            for m in net:
                if isinstance(m, torch.nn.ReLU):
                    t.feature = m(t.feature)
                else:
                    t = m(t)
            assert len(calls) == 4                      # called one by one: get_rules runs both steps itself
    finally:
        ops.get_rules_begin = real_begin
    assert torch.equal(y.z_idx, t.z_idx) and torch.equal(y.z_ptr, t.z_ptr) and torch.equal(y.feature, t.feature)
    sphconv.check_status()
    # the handle API itself: a mismatching handle is ignored, a matching one is used
    geom = (zi, zp, B, shape, [6, 10, 8], [3, 3, 3], [2, 2, 2], [1, 1, 1], [1, 1, 1], [2, 2])
    want = ops.get_rules(*geom)
    pend = ops.get_rules_begin(*geom)
    got = ops.get_rules(*geom, pending=pend)
    other = ops.get_rules(zi.clone(), zp, *geom[2:], pending=ops.get_rules_begin(*geom))
    for a, b, c in zip(want, got, other):
        assert torch.equal(a, b) and torch.equal(a, c)


def test_module_rules_written_beside_the_convolution():
    """The module path writes the reference-format pair lists on a side stream while the convolution runs; once the
    layer has returned they are complete on the caller's stream and equal those of the plain ops."""
    from sphconv_b200 import sphconv_cuda as ops
    rng = np.random.default_rng(17)
    B, shape = 3, [10, 14, 12]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3, False)        # unsorted columns too
    feat = torch.as_tensor(rng.standard_normal((z_idx.shape[0], 16)), dtype=torch.float16, device=DEV)
    zi, zp = torch.as_tensor(z_idx, device=DEV), torch.as_tensor(z_ptr, device=DEV)
    sub = sphconv.SubMConv3d(16, 16, 3, indice_key="k").to(DEV).half().eval()
    down = sphconv.SparseConv3d(16, 32, 3, stride=2, padding=1, indice_key="d").to(DEV).half().eval()

    def canon(rules, rule_size):
        r, n = rules.cpu().numpy(), rule_size.cpu().numpy()
        out = {}
        for t in range(r.shape[0]):
            for k in range(r.shape[1]):
                m = min(int(n[t, k]), r.shape[3])
                out[(t, k)] = sorted(zip(r[t, k, 0, :m].tolist(), r[t, k, 1, :m].tolist()))
        return n, out

    for flag in (True, False):
        ops.config.overlap_rule_lists = flag
        try:
            with torch.no_grad():
                x = sphconv.SparseConvTensor(feat, shape, B, z_idx=zi, z_ptr=zp)
                y = down(sub(x))
                # a kernel of the caller's on the current stream, right behind the layers, already sees the lists
                _, _, rules_s, size_s, _ = x.rule_cache["k"]
                _, _, rules_d, size_d, _ = y.rule_cache["d"]
                snap = (rules_s.clone(), size_s.clone(), rules_d.clone(), size_d.clone())
            assert getattr(rules_s, "_sph_ready", None) is None and getattr(rules_d, "_sph_ready", None) is None
        finally:
            ops.config.overlap_rule_lists = True
        want_s = ops.get_rules_subm(zi, zp, B, shape, shape, [3] * 3, [1] * 3, [1] * 3, [1] * 3, [2, 2])
        want_d = ops.get_rules(zi, zp, B, shape, [5, 7, 6], [3] * 3, [2] * 3, [1] * 3, [1] * 3, [2, 2])
        for (r, n), (wr, wn) in (((snap[0], snap[1]), (want_s[2], want_s[3])), ((snap[2], snap[3]), (want_d[2], want_d[3]))):
            n_got, got = canon(r, n)
            n_want, want = canon(wr, wn)
            assert (n_got == n_want).all() and got == want
    sphconv.check_status()


@pytest.mark.parametrize("fill", [True, False])
def test_module_rules_of_large_sets_written_beside_the_convolution(fill):
    """The same with rule sets that are large enough for the side stream (100 k rows), submanifold and strided: the plain ops hand
    out lists that are still to be joined, and behind a layer, on whichever stream it runs, they are complete."""
    from sphconv_b200 import sphconv_cuda as ops
    rng = np.random.default_rng(18)
    B, shape, small = 3, [64, 100, 64], [32, 50, 32]
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3, False)
    zi, zp = torch.as_tensor(z_idx, device=DEV), torch.as_tensor(z_ptr, device=DEV)
    feat = torch.as_tensor(rng.standard_normal((z_idx.shape[0], 16)), dtype=torch.float32, device=DEV)
    sub = sphconv.SubMConv3d(16, 32, 3, indice_key="k").to(DEV).eval()
    down = sphconv.SparseConv3d(32, 32, 3, stride=2, padding=1, indice_key="d").to(DEV).eval()
    geom_s = (zi, zp, B, shape, shape, [3] * 3, [1] * 3, [1] * 3, [1] * 3, [2, 2])
    geom_d = (zi, zp, B, shape, small, [3] * 3, [2] * 3, [1] * 3, [1] * 3, [2, 2])
    ops.config.fill_unused_rules = fill

    def used(rules, size):
        return torch.arange(rules.shape[3], device=DEV) < size[:, :, None, None]

    def same(got, want):
        (rules, size), (want_rules, want_size) = got, want
        assert torch.equal(size, want_size)
        mask = torch.ones_like(rules, dtype=torch.bool) if fill else used(rules, size).expand_as(rules)
        assert torch.equal(rules[mask], want_rules[mask])

    try:
        want_s, want_d = ops.get_rules_subm(*geom_s)[2:], ops.get_rules(*geom_d)[2:]
        res = rules_np.get_rules_subm(z_idx, z_ptr, B, shape, shape, [3] * 3, [1] * 3, [1] * 3, [1] * 3, [2, 2])
        assert (want_s[1].cpu().numpy() == res["rule_size"]).all()
        assert (rules_np.canonical_pairs(want_s[0].cpu().numpy(), res["rule_size"]) == rules_np.canonical_from_table(res)).all()
        torch.cuda.synchronize()
        for fn, geom, want, n_out in ((ops.get_rules_subm, geom_s, want_s, zi.numel()), (ops.get_rules, geom_d, want_d, None)):
            oz_idx, _, rules, size = fn(*geom, defer_lists=True)
            assert oz_idx.numel() >= 100000 and rules._sph_ready is not None
            assert getattr(fn(*geom, defer_lists=True, lists_beside=False)[2], "_sph_ready", None) is None
            ops.rule_conv(feat, torch.zeros(27, 16, 16, device=DEV), rules, size, oz_idx.numel())
            snap = rules.clone(), size.clone()
            assert rules._sph_ready is None
            same(snap, want)
        for i in range(6):
            ops.config.overlap_rule_lists = i < 5
            stream = torch.cuda.Stream() if i % 2 else torch.cuda.current_stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream), torch.no_grad():
                x = sphconv.SparseConvTensor(feat, shape, B, z_idx=zi, z_ptr=zp)
                y = down(sub(x))
                _, _, rules_s, size_s, _ = x.rule_cache["k"]
                _, _, rules_d, size_d, _ = y.rule_cache["d"]
                snap = rules_s.clone(), size_s.clone(), rules_d.clone(), size_d.clone()
            del x, y, rules_s, rules_d         # their memory is taken again by the next pass
            torch.cuda.current_stream().wait_stream(stream)
            same(snap[:2], want_s)
            same(snap[2:], want_d)
    finally:
        ops.config.overlap_rule_lists, ops.config.fill_unused_rules = True, True
    sphconv.check_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.int8])
def test_weights_that_are_not_contiguous_are_refused(dtype):
    """An expanded or transposed weight is refused before anything reads its memory as [KV, iC, oC]."""
    from sphconv_b200 import sphconv_cuda as ops
    x = torch.zeros(8, 16, device=DEV, dtype=dtype)
    nbr = torch.full((27, 8), -1, dtype=torch.int32, device=DEV)
    for w in (torch.zeros(1, 1, 16, device=DEV, dtype=dtype).expand(27, 16, 16),
              torch.zeros(27, 16, 16, device=DEV, dtype=dtype).transpose(1, 2)):
        with pytest.raises(RuntimeError, match="contiguous"):
            ops._gather(x, w, nbr, 8, False, None, None, False, None)


def test_layers_whose_lists_are_written_beside_them():
    from sphconv_b200 import sphconv_cuda as ops
    f32, f16, i8 = torch.float32, torch.float16, torch.int8
    for dtype, iC, oC, padded, want in ((f32, 16, 32, False, True), (f32, 64, 64, True, True), (f32, 16, 16, True, False), (f16, 32, 32, True, False),
                                        (f16, 48, 40, False, True), (f16, 16, 16, True, True), (f16, 16, 16, False, False), (i8, 64, 64, True, False),
                                        (torch.float64, 64, 64, True, False)):
        assert ops.lists_beside(dtype, 27, iC, oC, padded) is want


FIRST_USE = """
import sys, threading
import torch
sys.path[:0] = sys.argv[1:]
import sphconv_b200 as sphconv
from sphconv_b200 import sphconv_cuda as ops
x = torch.ones(300, 16, device="cuda", dtype=torch.float16)
nbr = torch.arange(300, device="cuda", dtype=torch.int32).repeat(27, 1)
nbr[3, 5] = 300                                   # no row: every call sets the status bit
w = torch.ones(27, 16, 16, device="cuda", dtype=torch.float16)
torch.cuda.synchronize()
gate, out = threading.Barrier(8), [None] * 8
def work(i):
    with torch.cuda.stream(torch.cuda.Stream()):
        gate.wait()
        out[i] = (ops.C.host().conv_wgrad(x, x, nbr, None, False), ops.C.host().status_tensor(0).data_ptr())
        torch.cuda.current_stream().synchronize()
threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
[t.start() for t in threads]; [t.join() for t in threads]
assert all(torch.equal(o[0], out[0][0]) and o[1] == out[0][1] for o in out)
try:
    sphconv.check_status()
except RuntimeError:
    print("status seen")
"""


def test_first_use_from_many_threads():
    """The first operators of a process, issued by eight threads on eight streams: one status word, and none of its bits lost."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    got = subprocess.run([sys.executable, "-c", FIRST_USE, root], capture_output=True, text=True, timeout=300)
    assert got.returncode == 0 and "status seen" in got.stdout, got.stderr[-2000:]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_bias_written_in_place_is_seen_at_inference(dtype):
    """The bias is read in every call, also after a write that leaves the parameter's version as it was."""
    rng = np.random.default_rng(4)
    zi, zp = (torch.as_tensor(a, device=DEV) for a in synthetic.make_random_occupancy(rng, 1, [5, 6, 7], 0.4))
    layer = sphconv.SubMConv3d(16, 32, 3, bias=True, apply_bias=True).to(DEV).to(dtype).eval()
    x = torch.zeros(zi.numel(), 16, device=DEV, dtype=dtype)
    with torch.no_grad():
        for value in (0.25, -3.0):
            layer.bias.data.fill_(value)
            y = layer(sphconv.SparseConvTensor(x, [5, 6, 7], 1, z_idx=zi, z_ptr=zp))
            assert torch.equal(y.feature, torch.full_like(y.feature, value))


@pytest.mark.parametrize("K,N", [(4, 16), (16, 16), (32, 64), (64, 64), (128, 128), (24, 40), (5, 7), (48, 48), (100, 9), (33, 130)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_bias_in_the_type_of_the_rows(K, N, dtype):
    """A 16-bit bias gives what its float32 values give, bit for bit, in each kernel that has an epilogue; other types of bias
    are refused."""
    from sphconv_b200 import sphconv_cuda as ops
    g = torch.Generator(device=DEV).manual_seed(K * N)
    n = 1000
    nbr = torch.randint(0, n, (27, n), generator=g, device=DEV, dtype=torch.int32)
    nbr[torch.rand(27, n, generator=g, device=DEV) < 0.9] = -1
    w = torch.randn(27, K, N, generator=g, device=DEV).to(dtype)
    x = torch.randn(n, K, generator=g, device=DEV).to(dtype)
    bias = torch.randn(N, generator=g, device=DEV).to(dtype)
    plain = ops._gather(x, w, nbr, n, False, None, None, False, None)
    for relu in (False, True):
        a, b = (ops._gather(x, w, nbr, n, False, None, v, relu, None) for v in (bias, bias.float()))
        assert torch.equal(a, b) and not torch.equal(a, plain)
    for other in (bias.double(), bias.to(torch.bfloat16 if dtype == torch.float16 else torch.float16)):
        with pytest.raises(RuntimeError):
            ops._gather(x, w, nbr, n, False, None, other, False, None)
    with pytest.raises(RuntimeError):
        ops._gather(x.float(), w.float(), nbr, n, False, None, bias, False, None)
