"""Kernels are launched before the ones in front of them have ended and wait inside: chains that follow one another without a
synchronisation, on two streams, and chains captured in a graph give what single steps with a synchronisation in between give."""
import numpy as np
import pytest
import torch

import sphconv_b200 as sphconv
from sphconv_b200 import sphconv_cuda as ops
from sphconv_b200.encoder import build_encoder8

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scan(seed, shape, B):
    rng = np.random.default_rng(seed)
    cells = rng.random((B, *shape)) < 0.06 + 0.02 * seed
    z_idx, per = np.nonzero(cells)[3], cells.sum(-1).reshape(-1)
    return (torch.as_tensor(z_idx, dtype=torch.int32, device=DEV), torch.as_tensor(per.cumsum(), dtype=torch.int32, device=DEV).view(B, *shape[:2]),
            torch.as_tensor(rng.standard_normal((z_idx.size, 4)), device=DEV).half())


@pytest.mark.parametrize("shape,B,dtype", [([16, 48, 32], 2, torch.float16), ([64, 128, 64], 4, torch.float16),
                                           ([64, 128, 64], 4, torch.float32)])       # the last one's lists: on the side stream
def test_passes_without_synchronisation_on_two_streams(shape, B, dtype):
    scans = [_scan(s, shape, B) for s in range(4)]
    scans = [(z_idx, z_ptr, feature.to(dtype)) for z_idx, z_ptr, feature in scans]
    net = build_encoder8(dtype=dtype, device=DEV).eval()

    def run(scan):
        z_idx, z_ptr, feature = scan
        with torch.no_grad():
            y = net(sphconv.SparseConvTensor(feature, shape, B, z_idx=z_idx, z_ptr=z_ptr))
        rules = [r[2:4] for r in y.rule_cache.values()]
        assert len(rules) == 3                 # of the submanifold levels
        return [y.feature, y.z_idx, y.z_ptr] + [t.clone() for pair in rules for t in pair]

    want = []
    for scan in scans:
        want.append(run(scan))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for i in range(24):
        with torch.cuda.stream(streams[i % 2]):
            got.append(run(scans[i % 4]))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i % 4]))


@pytest.mark.parametrize("K,N", [(4, 16), (16, 16), (32, 32), (64, 64)])
def test_rules_and_layers_in_a_graph(K, N):
    """A submanifold rule set with its lists and two layers, captured once and replayed on other inputs."""
    shape, B = [24, 40, 32], 2
    z_idx, z_ptr, _ = _scan(2, shape, B)
    n = z_idx.numel()
    feature = torch.randn(n, K, device=DEV).half()
    w1, w2 = (torch.randn(27, K, N, device=DEV) * 0.1).half(), (torch.randn(27, N, N, device=DEV) * 0.1).half()

    def chain():
        _, _, rules, size = ops.get_rules_subm(z_idx, z_ptr, B, shape, shape, [3] * 3, [1] * 3, [1] * 3, [1] * 3, [2, 2])
        y = ops.rule_conv(feature, w1, rules, size, n)
        return ops.rule_conv(y, w2, rules, size, n), size

    chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, size = chain()
    for _ in range(3):
        feature.copy_(torch.randn(n, K, device=DEV))
        want, want_size = (t.clone() for t in chain())
        torch.cuda.synchronize()
        for _ in range(5):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(size, want_size)


@pytest.mark.parametrize("K,N,kv,dtype", [(16, 16, 27, torch.float32), (64, 64, 27, torch.float32), (20, 12, 27, torch.int8),
                                          (4, 16, 27, torch.float16), (16, 16, 27, torch.float16), (24, 40, 27, torch.bfloat16),
                                          (16, 32, 27, torch.float16), (32, 32, 9, torch.bfloat16), (64, 64, 27, torch.float16),
                                          (32, 64, 27, torch.int8), (32, 32, 28, torch.float16), (128, 64, 27, torch.float16)])
def test_rows_written_by_the_kernel_in_front(K, N, kv, dtype):
    """Convolutions and weight gradients whose input rows the kernel in front of them in the stream, a small one that lets them in at
    once, writes over the rows of the pass before."""
    from sphconv_b200 import _capi as C
    g = torch.Generator(device=DEV).manual_seed(K * N)
    n = 4001
    table = torch.arange(n, device=DEV) + torch.randint(-60, 61, (kv, n), device=DEV, generator=g)
    table = torch.where((table < 0) | (table >= n) | (torch.rand(kv, n, device=DEV, generator=g) < 0.5), -1, table).int().contiguous()
    rules = ops._Tables(table, None, n, n, 0, False)

    def values(*shape):
        if dtype == torch.int8:
            return torch.randint(-100, 101, shape, device=DEV, generator=g, dtype=dtype)
        return torch.randn(*shape, device=DEV, generator=g).to(dtype)

    sources, weight, d_out = [values(n, K), values(n, K)], values(kv, K, N), None if dtype == torch.int8 else values(n, N)
    order = torch.randperm(n, device=DEV, generator=g).int()

    def step(i, wait=lambda: None):
        x = C.host().gather_rows(sources[i % 2], order)
        wait()
        y = ops.rule_conv(x, weight, rules, None, n)
        if d_out is None:
            return y, None
        x = C.host().gather_rows(sources[(i + 1) % 2], order)
        wait()
        return y, ops.rule_conv_d_weight(x, d_out, rules, None)

    want = [step(i, torch.cuda.synchronize) for i in range(2)]
    got = [step(i) for i in range(40)]
    torch.cuda.synchronize()
    for i, (y, dw) in enumerate(got):
        assert torch.equal(y, want[i % 2][0])
        if dw is not None:                 # sums of up to 4001 products in another order: 2^-24 sqrt(4001) of about 45, and 16 bits of result
            w = want[i % 2][1].double()
            assert (dw.double() - w).norm() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * w.norm()
