"""Rule generation on the GPU against the CPU oracle: bit-exact rule_size, pair multisets per (tile,k),
oz_idx and oz_ptr.  Shapes follow the reference's test/test_rules.py (small literal cases, kernels 1-3,
strides 1-2, paddings 0-1, batch 1-8, non-cubic shapes) with seeded random occupancies."""
import itertools

import numpy as np
import pytest
import torch

from oracle import rules_np
from sphconv_b200 import check_status, synthetic
from sphconv_b200 import sphconv_cuda as ops

from gpu_util import DEV, assert_rules_equal, assert_tables_match, gpu_rules, oracle_rules, to_dev
from test_oracle import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("i", range(len(CASES)))
@pytest.mark.parametrize("sort_columns", [True, False])
def test_strided_small(i, sort_columns):
    B, shape, ks, st, pd, tile, dens = CASES[i]
    rng = np.random.default_rng(100 + i)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, dens, sort_columns)
    with torch.enable_grad():
        zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, False)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, False)
    assert_rules_equal(res, oz_idx, oz_ptr, rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])
    assert rules._sph.nbr_t is not None
    assert check_status() & 1 == 0


@pytest.mark.parametrize("ks", [[3, 3, 3], [1, 1, 1], [3, 3, 1], [2, 2, 2], [3, 1, 3], [5, 5, 5]])
@pytest.mark.parametrize("sort_columns", [True, False])
def test_subm_small(ks, sort_columns):
    B, shape, tile = 3, [7, 9, 6], [2, 2]
    rng = np.random.default_rng(7)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.3, sort_columns)
    pd = [k // 2 for k in ks]
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, [1, 1, 1], pd, tile, True)
    assert oz_idx is zi and oz_ptr is zp           # same objects, as the reference returns them
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, [1, 1, 1], pd, tile, True)
    assert_rules_equal(res, oz_idx, oz_ptr.reshape(B, *shape[:2]), rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], z_idx.shape[0])


def test_exhaustive_2x2x2():
    """Every occupancy of a 2x2x2 grid, batch 2 (second scan = complement), subm 3x3x3 and strided k2 s2 / k3 s2 p1."""
    shape = [2, 2, 2]
    for code in range(256):
        occ = np.array([(code >> b) & 1 for b in range(8)], dtype=bool).reshape(1, 2, 2, 2)
        occ = np.concatenate([occ, ~occ], axis=0)
        counts = occ.sum(axis=3).reshape(-1)
        z_ptr = np.cumsum(counts).astype(np.int32).reshape(2, 2, 2)
        z_idx = np.nonzero(occ)[3].astype(np.int32)
        for subm, ks, st, pd in [(True, [3, 3, 3], [1, 1, 1], [1, 1, 1]), (False, [2, 2, 2], [2, 2, 2], [0, 0, 0]),
                                 (False, [3, 3, 3], [2, 2, 2], [1, 1, 1])]:
            _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, 2, shape, ks, st, pd, [2, 2], subm)
            res = oracle_rules(z_idx, z_ptr, 2, shape, ks, st, pd, [2, 2], subm)
            assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size, check_padding=False)


def test_empty_and_single():
    shape, ks = [4, 4, 4], [3, 3, 3]
    z_ptr = np.zeros((1, 4, 4), np.int32)
    z_idx = np.zeros((0,), np.int32)
    for subm, st, pd in [(True, [1, 1, 1], [1, 1, 1]), (False, [2, 2, 2], [1, 1, 1])]:
        _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, 1, shape, ks, st, pd, [2, 2], subm)
        assert int(rule_size.sum()) == 0 and oz_idx.shape[0] == 0
    occ = np.zeros((1, 4, 4, 4), bool)
    occ[0, 3, 3, 3] = True
    z_ptr = np.cumsum(occ.sum(axis=3).reshape(-1)).astype(np.int32).reshape(1, 4, 4)
    z_idx = np.array([3], np.int32)
    for subm, st, pd in [(True, [1, 1, 1], [1, 1, 1]), (False, [2, 2, 2], [1, 1, 1]), (False, [1, 1, 1], [0, 0, 0])]:
        _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, 1, shape, ks, st, pd, [2, 2], subm)
        res = oracle_rules(z_idx, z_ptr, 1, shape, ks, st, pd, [2, 2], subm)
        assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size)


def test_full_columns_and_big_tiles():
    """Dense grid (every depth bin active: maximum column length) and tiles larger than the grid."""
    B, shape = 2, [5, 6, 40]
    occ = np.ones((B, *shape), bool)
    z_ptr = np.cumsum(occ.sum(axis=3).reshape(-1)).astype(np.int32).reshape(B, 5, 6)
    z_idx = np.nonzero(occ)[3].astype(np.int32)
    for subm, ks, st, pd, tile in [(True, [3, 3, 3], [1, 1, 1], [1, 1, 1], [8, 8]),
                                   (False, [3, 3, 3], [2, 2, 2], [1, 1, 1], [2, 2]),
                                   (False, [3, 3, 3], [1, 1, 1], [0, 0, 0], [4, 3])]:
        _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
        res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
        assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size, check_padding=False)


def test_overflow_is_flagged_and_tables_stay_exact():
    """A tile_n_max overflow drops pairs from `rules` exactly like the reference (src/sphconv/rules.cu:217-224:
    rule_size keeps counting) and raises the status bit; the neighbour tables are not limited."""
    B, shape = 1, [16, 16, 64]
    occ = np.zeros((B, *shape), bool)
    occ[0, :2, :2, :] = True      # one dense tile in an otherwise empty grid: the sparsity heuristic underestimates
    z_ptr = np.cumsum(occ.sum(axis=3).reshape(-1)).astype(np.int32).reshape(B, 16, 16)
    z_idx = np.nonzero(occ)[3].astype(np.int32)
    check_status()
    _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, [3, 3, 3], [1, 1, 1], [1, 1, 1], [2, 2], True)
    res = oracle_rules(z_idx, z_ptr, B, shape, [3, 3, 3], [1, 1, 1], [1, 1, 1], [2, 2], True)
    assert res["rule_size"].max() > rules.shape[3]
    assert check_status() & 1
    assert (rule_size.cpu().numpy() == res["rule_size"]).all()
    assert_tables_match(res, rules, z_idx.shape[0], z_idx.shape[0])


@pytest.mark.parametrize("subm", [True, False])
def test_exact_rule_capacity_never_overflows(subm):
    """config.exact_rule_capacity: tile_n_max is the longest list (counted first), so the input that overflows the
    reference's heuristic capacity keeps every pair and raises no status bit."""
    from sphconv_b200 import sphconv_cuda as ops
    B, shape = 2, [16, 16, 64]
    occ = np.zeros((B, *shape), bool)
    occ[:, :2, :2, :] = True
    occ[1, 7, 9, 3] = True
    z_ptr = np.cumsum(occ.sum(axis=3).reshape(-1)).astype(np.int32).reshape(B, 16, 16)
    z_idx = np.nonzero(occ)[3].astype(np.int32)
    ks, st, pd = ([3, 3, 3], [1, 1, 1], [1, 1, 1]) if subm else ([3, 3, 3], [2, 2, 2], [1, 1, 1])
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, [2, 2], subm)
    check_status()
    ops.config.exact_rule_capacity = True
    try:
        _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, [2, 2], subm)
    finally:
        ops.config.exact_rule_capacity = False
    assert check_status() == 0
    if subm:
        assert res["rule_size"].max() > res["tile_n_max"], "the case must overflow the heuristic capacity"
    assert rules.shape[3] == res["rule_size"].max()
    rs, r = rule_size.cpu().numpy(), rules.cpu().numpy()
    assert (rs == res["rule_size"]).all()
    got = set()
    for t, k in zip(*np.nonzero(rs)):
        n = rs[t, k]
        got.update((int(k), int(i), int(o)) for i, o in zip(r[t, k, 0, :n], r[t, k, 1, :n]))
    want = set(zip(res["k"].tolist(), res["in"].tolist(), res["out"].tolist()))
    assert got == want and len(want) == int(rs.sum())
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])


@pytest.mark.parametrize("name,batch", [("cfg1", 1), ("cfg2", 4), ("cfg3", 2)])
def test_config_first_layer(name, batch):
    """BASELINE configs at full per-scan size: first layer's rule set (cfg1 SubM; cfg2 strided; cfg3 SubM)."""
    cfg = synthetic.CONFIGS[name]
    b = synthetic.make_batch(name, batch=batch)
    subm = name != "cfg2"
    ks = [3, 3, 3]
    st, pd = ([1, 1, 1], [1, 1, 1]) if subm else ([2, 2, 2], [1, 1, 1])
    _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(b["z_idx"], b["z_ptr"], batch, cfg["shape"], ks, st, pd, [2, 2], subm)
    res = oracle_rules(b["z_idx"], b["z_ptr"], batch, cfg["shape"], ks, st, pd, [2, 2], subm)
    assert (rule_size.cpu().numpy() == res["rule_size"]).all()
    assert (oz_idx.cpu().numpy() == res["oz_idx"]).all() and (oz_ptr.cpu().numpy() == res["oz_ptr"]).all()
    assert res["rule_size"].max() <= rules.shape[3], "heuristic tile_n_max overflowed on a BASELINE config"
    assert_tables_match(res, rules, b["z_idx"].shape[0], oz_idx.shape[0])
    # pair multisets via the attached tables (the padded tensor is GB-scale here); lists themselves on a sample of tiles
    r = rules[:64].cpu().numpy()
    rs = rule_size[:64].cpu().numpy()
    got = rules_np.canonical_pairs(r, rs)
    full = rules_np.canonical_from_table(res)
    assert (got == full[full[:, 0] < 64]).all()


def test_encoder_rule_chain_cfg3():
    """Rule sets of the whole 8-layer encoder on one cfg3 scan: each level's oz_idx/oz_ptr feed the next."""
    cfg = synthetic.CONFIGS["cfg3"]
    b = synthetic.make_batch("cfg3", batch=1)
    z_idx, z_ptr, shape = b["z_idx"], b["z_ptr"], list(cfg["shape"])
    seen = set()
    for subm, iC, oC, stride, key in synthetic.ENCODER8:
        if key is not None and key in seen:
            continue
        seen.add(key)
        st, pd = [stride] * 3, [1, 1, 1]
        _, _, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, 1, shape, [3, 3, 3], st, pd, [2, 2], subm)
        res = oracle_rules(z_idx, z_ptr, 1, shape, [3, 3, 3], st, pd, [2, 2], subm)
        assert (rule_size.cpu().numpy() == res["rule_size"]).all()
        assert (oz_idx.cpu().numpy() == res["oz_idx"]).all()
        assert (oz_ptr.cpu().numpy().reshape(-1) == res["oz_ptr"].reshape(-1)).all()
        assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])
        if not subm:
            z_idx, z_ptr, shape = res["oz_idx"], res["oz_ptr"], osh


def test_deterministic_and_foreign_rules():
    """Two runs give identical tensors (list order included); a cloned rules tensor (no attached tables)
    converts to the same tables."""
    B, shape = 4, [8, 12, 16]
    rng = np.random.default_rng(3)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.2)
    a = gpu_rules(z_idx, z_ptr, B, shape, [3, 3, 3], [2, 2, 2], [1, 1, 1], [2, 2], False)
    b = gpu_rules(z_idx, z_ptr, B, shape, [3, 3, 3], [2, 2, 2], [1, 1, 1], [2, 2], False)
    for x, y in zip(a[3:], b[3:]):
        assert torch.equal(x, y)
    rules, rule_size = a[5], a[6]
    clone = rules.clone()
    assert not hasattr(clone, "_sph")
    tb = ops._tables_for(clone, rule_size, z_idx.shape[0], a[3].shape[0], need_t=True)
    assert torch.equal(tb.nbr, rules._sph.nbr)
    res = oracle_rules(z_idx, z_ptr, B, shape, [3, 3, 3], [2, 2, 2], [1, 1, 1], [2, 2], False)
    assert_tables_match(res, clone, z_idx.shape[0], a[3].shape[0])
    assert check_status() == 0


def test_bad_arguments_raise():
    zi, zp = to_dev(np.zeros(0, np.int32), np.zeros((1, 4, 4), np.int32))
    with pytest.raises(RuntimeError):
        ops.get_rules(zi, zp, 1, [4, 4, 4], [2, 2, 2], [3, 3, 3], [2, 2, 2], [1, 1, 1], [0, 1, 1], [2, 2])   # dilation 0
    with pytest.raises(RuntimeError):
        ops.get_rules_subm(zi, zp, 1, [4, 4, 4], [2, 2, 2], [3, 3, 3], [1, 1, 1], [1, 1, 1], [1, 1, 1], [2, 2])  # shape
    with pytest.raises(RuntimeError):
        ops.get_rules(zi.cpu(), zp.cpu(), 1, [4, 4, 4], [2, 2, 2], [3, 3, 3], [2, 2, 2], [1, 1, 1], [1, 1, 1], [2, 2])


@pytest.mark.parametrize("dens", [0.002, 0.05, 0.6])
@pytest.mark.parametrize("subm", [True, False])
def test_index_and_scan_paths_agree(dens, subm):
    """Nearly empty grids take the per-column scan kernels (no column index is built), denser ones the row-parallel
    kernels on the index; both must give the oracle's rules."""
    B, shape, tile = 2, [12, 20, 96], [2, 2]
    rng = np.random.default_rng(int(dens * 1000) + (7 if subm else 0))
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, dens, True)
    ks, st, pd = ([3, 3, 3], [1, 1, 1], [1, 1, 1]) if subm else ([3, 3, 3], [2, 2, 2], [1, 1, 1])
    _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])


@pytest.mark.parametrize("ks,st,pd", [([7, 7, 7], [1, 1, 1], [3, 3, 3]), ([3, 3, 7], [2, 2, 6], [1, 1, 3]),
                                      ([2, 2, 2], [2, 2, 2], [0, 0, 0]), ([3, 3, 5], [1, 2, 4], [1, 1, 2])])
def test_large_kernels_and_strides(ks, st, pd):
    """Kernel extents up to 7 and depth strides beyond what the bit-parallel pattern kernel handles."""
    B, shape, tile = 2, [9, 11, 70], [2, 2]
    rng = np.random.default_rng(sum(ks) * 10 + sum(st))
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.15, True)
    subm = st == [1, 1, 1]
    _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])


@pytest.mark.parametrize("subm", [True, False])
def test_tables_without_rule_lists(subm):
    """config.materialize_rules = False: no rules / rule_size, the neighbour tables alone, still exact."""
    B, shape, tile = 3, [10, 14, 40], [2, 2]
    rng = np.random.default_rng(11)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.2, True)
    ks, st, pd = ([3, 3, 3], [1, 1, 1], [1, 1, 1]) if subm else ([3, 3, 3], [2, 2, 2], [1, 1, 1])
    ops.config.materialize_rules = False
    try:
        with torch.enable_grad():
            _, _, _, oz_idx, oz_ptr, tables, none = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    finally:
        ops.config.materialize_rules = True
    assert none is None
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    assert (oz_idx.cpu().numpy() == res["oz_idx"]).all()
    KV = res["rule_size"].shape[1]
    want = np.full((KV, oz_idx.shape[0]), -1, dtype=np.int64)
    want[res["k"], res["out"]] = res["in"]
    assert (tables.nbr.cpu().numpy() == want).all()
    if not subm:
        want_t = np.full((KV, z_idx.shape[0]), -1, dtype=np.int64)
        want_t[res["k"], res["in"]] = res["out"]
        assert (tables.nbr_t.cpu().numpy() == want_t).all()


@pytest.mark.parametrize("subm", [True, False])
def test_deep_grid(subm):
    """More than 256 depth bins: the column index is built by the kernel that works in global memory."""
    B, shape, tile = 2, [6, 10, 300], [2, 2]
    rng = np.random.default_rng(5)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.1, True)
    ks, st, pd = ([3, 3, 3], [1, 1, 1], [1, 1, 1]) if subm else ([3, 3, 3], [2, 2, 2], [1, 1, 1])
    _, _, _, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    assert_rules_equal(res, oz_idx, oz_ptr.reshape(res["oz_ptr"].shape), rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])


@pytest.mark.parametrize("depth", [3, 5, 31, 32, 33, 63, 64, 65, 66, 100, 129, 256])
@pytest.mark.parametrize("dens", [0.15, 1.0])
def test_stride2_depth_pattern_word_boundaries(depth, dens):
    """The usual stride-2, 3-deep, padding-1 layer at depths around the 32-bin word boundaries of the column index: the
    output pattern (oz_idx, oz_ptr), the pair lists and the tables against the oracle, sparse and completely full."""
    B, shape, tile = 2, [5, 6, depth], [2, 2]
    rng = np.random.default_rng(900 + depth)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, dens)
    ks, st, pd = [3, 3, 3], [2, 2, 2], [1, 1, 1]
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, False)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, False)
    assert_rules_equal(res, oz_idx, oz_ptr, rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])
    assert check_status() & 1 == 0


@pytest.mark.parametrize("subm", [True, False])
def test_more_runs_per_tile_than_one_staging_pass(subm):
    """150 scans in the batch: a tile of 2 x 2 columns then has 300 (batch, tile row) runs, more than the pair-list kernels
    stage at a time (128), so they go through a tile in several passes."""
    B, shape, tile = 150, [4, 6, 9], [2, 2]
    rng = np.random.default_rng(77)
    z_idx, z_ptr = synthetic.make_random_occupancy(rng, B, shape, 0.4)
    ks = [3, 3, 3]
    st, pd = ([1, 1, 1], [1, 1, 1]) if subm else ([2, 2, 2], [1, 1, 1])
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    res = oracle_rules(z_idx, z_ptr, B, shape, ks, st, pd, tile, subm)
    if subm:
        oz_ptr = oz_ptr.reshape(B, *shape[:2])
    assert_rules_equal(res, oz_idx, oz_ptr, rules, rule_size)
    assert_tables_match(res, rules, z_idx.shape[0], oz_idx.shape[0])
    assert check_status() & 1 == 0


def _small(n, seed):
    rng = np.random.default_rng(seed)
    zi, zp = synthetic.make_random_occupancy(rng, 1, [6, 8, 10], 0.1 + 0.8 * (n % 7) / 7)
    return to_dev(zi, zp)


GEOM = (1, [6, 8, 10], [3, 4, 5], [3, 3, 3], [2, 2, 2], [1, 1, 1], [1, 1, 1], [2, 2])


def test_many_rule_sets_begun_before_the_first_is_completed():
    """Handles outlive any number of further calls, whatever those write their counts to; dropped ones harm nobody."""
    from sphconv_b200.voxelize import VoxelGenerator
    inputs = [_small(n, n) for n in range(600)]
    begun = [ops.get_rules_begin(zi, zp, *GEOM) for zi, zp in inputs]
    gen = VoxelGenerator([0, -40, -3, 70.4, 40, 1], [0, -45, 87.5, 70.4, 45, 100], 2, 100, [10, 8, 6], "spherical")
    pts = torch.rand(200, 4, device=inputs[0][0].device) * 40
    for n in range(200):
        gen.generate(pts[: 100 + n % 50])
        ops.get_rules_begin(*inputs[n], *GEOM)          # dropped at once
    for n in list(range(0, 600, 37)) + [599]:
        got = ops.get_rules(*inputs[n], *GEOM, pending=begun[n])
        want = ops.get_rules(*inputs[n], *GEOM)
        assert all(torch.equal(a, b) for a, b in zip(got, want)), n


def test_counts_handed_to_the_caller_are_not_turned_by_calls_that_wait():
    """C ABI: a count word stays its caller's while waiting calls come and go."""
    import ctypes

    from sphconv_b200 import _capi as C
    lib = C.lib()
    zi, zp = _small(3, 3)
    g = C.make_geom(GEOM[0], GEOM[1], GEOM[2], GEOM[3], GEOM[4], GEOM[5], GEOM[7], GEOM[6])
    bytes_ = lib.sph_rules_strided_scratch_bytes(ctypes.byref(g), zi.numel())
    new = lambda *s: torch.empty(s, dtype=torch.int32, device=zi.device)  # noqa: E731
    scratch, oz_ptr, count = new(bytes_ // 4), new(1, 3, 4), new(1)
    word = ctypes.c_void_p(0)
    C.check(lib.sph_rules_strided_count_async(C.ptr(zi), C.ptr(zp), zi.numel(), ctypes.byref(g), C.ptr(scratch), C.ptr(oz_ptr),
                                              C.ptr(count), ctypes.byref(word), C.stream_ptr(zi.device)))
    torch.cuda.synchronize()
    want = int(count)
    empty = torch.zeros_like(zp)
    h = ctypes.c_int32(-1)
    for _ in range(300):
        C.check(lib.sph_rules_strided_count(C.ptr(zi), C.ptr(empty), zi.numel(), ctypes.byref(g), C.ptr(scratch), C.ptr(oz_ptr),
                                            C.ptr(count), ctypes.byref(h), C.stream_ptr(zi.device)))
        assert h.value == 0
    assert want > 0 and ctypes.c_int32.from_address(word.value).value == want


def test_rule_set_begun_on_another_stream():
    """What a handle holds is not reused on the stream it was begun on while the completing stream still reads it."""
    rng = np.random.default_rng(8)
    B, shape, out = 2, [64, 256, 64], [32, 128, 32]
    zi, zp = to_dev(*synthetic.make_random_occupancy(rng, B, shape, 0.05))
    args = (zi, zp, B, shape, out, [3, 3, 3], [2, 2, 2], [1, 1, 1], [1, 1, 1], [2, 2])
    want = ops.get_rules(*args)
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s1):
        handle = ops.get_rules_begin(*args)
    with torch.cuda.stream(s2):
        a = torch.randn(4096, 4096, device=zi.device)
        for _ in range(20):                     # the completing kernels wait behind these
            a = a @ a * 1e-3
        got = ops.get_rules(*args, pending=handle)
    del handle
    with torch.cuda.stream(s1):
        spoil = [torch.full((1 << 16,), -1, dtype=torch.int32, device=zi.device) for _ in range(400)]
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, want)) and len(spoil) == 400


def test_tables_of_other_sizes_are_refused():
    """A rule set without lists serves the row counts it was made for, and no others."""
    ops.config.materialize_rules = False
    try:
        zi, zp = _small(4, 4)
        n = zi.numel()
        tables = ops.get_rules_subm(zi, zp, 1, [6, 8, 10], [6, 8, 10], [3] * 3, [1] * 3, [1] * 3, [1] * 3, [2, 2])[2]
    finally:
        ops.config.materialize_rules = True
    w = torch.zeros(27, 16, 16, device=zi.device)
    assert ops.rule_conv(torch.zeros(n, 16, device=zi.device), w, tables, None, n).shape == (n, 16)
    for n_in, n_out in ((n - 1, n), (n, n + 1000)):
        with pytest.raises(RuntimeError, match="rows"):
            ops.rule_conv(torch.zeros(n_in, 16, device=zi.device), w, tables, None, n_out)
        with pytest.raises(RuntimeError, match="rows"):
            ops.rule_conv_d_weight(torch.zeros(n_in, 16, device=zi.device), torch.zeros(n_out, 16, device=zi.device), tables, None)


@pytest.mark.parametrize("B,H,W,D,occ,nmax,subm", [(1, 64, 66, 96, 1.0, 96, True),       # tiles of 290 rows, columns of up to 96
                                                   (6, 64, 64, 128, 0.95, 128, True),    # more than 2048 positions in a tile
                                                   (70, 64, 64, 16, 0.9, 3, True),       # more than 128 runs in a tile
                                                   (3, 130, 126, 64, 0.9, 12, False)])
def test_lists_of_large_tiles_in_order(B, H, W, D, occ, nmax, subm):
    """Lists that a CTA per tile writes (27 offsets, 1024 tiles of 256 rows and more): every pair of the table, by tile and
    offset, in the order (batch, tile row, row)."""
    rng = np.random.default_rng(B)
    want = np.where(rng.random((B, H, W)) < occ, rng.integers(nmax // 2 + 1, nmax + 1, (B, H, W)), 0)
    cells = rng.random((B, H, W, D)).argsort(-1).argsort(-1) < want[..., None]
    z_idx, z_ptr = np.nonzero(cells)[3].astype(np.int32), want.reshape(-1).cumsum().reshape(B, H, W).astype(np.int32)
    _check_lists_of_large_tiles(z_idx, z_ptr, B, (H, W, D), (1, 1, 1) if subm else (2, 2, 2), subm)


def _check_lists_of_large_tiles(z_idx, z_ptr, B, shape, stride, subm):
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, shape, (3, 3, 3), stride, (1, 1, 1), (2, 2), subm)
    n, tiles = oz_idx.numel(), rules.shape[0]
    assert tiles >= 1024 and n >= 256 * tiles
    column = torch.repeat_interleave(torch.arange(oz_ptr.numel(), device=DEV), torch.diff(oz_ptr.view(-1), prepend=oz_ptr.new_zeros(1)).long())
    oy, ox, b = column % osh[1], column // osh[1] % osh[0], column // (osh[0] * osh[1])
    tile = ox // 2 * ((osh[1] + 1) // 2) + oy // 2
    order = (((tile * B + b) * 2 + ox % 2) * n + torch.arange(n, device=DEV)).argsort()      # rows in list order
    nbr = rules._sph.nbr[:, order]
    for k in range(27):
        has = nbr[k] >= 0
        size = torch.bincount(tile[order][has], minlength=tiles)
        assert torch.equal(rule_size[:, k].long(), size)
        used = torch.arange(rules.shape[3], device=DEV) < size[:, None]
        assert torch.equal(rules[:, k, 0][used], nbr[k][has]) and torch.equal(rules[:, k, 1][used].long(), order[has])


@pytest.mark.parametrize("B,empty", [(70, (0, 64)), (140, (0, 64)), (200, (64, 128)), (200, (0, 128)), (140, (64, 140))])
def test_lists_of_large_tiles_with_groups_of_empty_runs(B, empty):
    """More than 128 runs in a tile (two a scan), of which whole groups of 128 have no row in a quarter of the tiles."""
    rng = np.random.default_rng(B)
    H, W, D = 64, 64, 16
    want = rng.integers(2, 7, (B, H, W))
    want[empty[0]:empty[1], :H // 2, W // 2:] = 0
    cells = rng.random((B, H, W, D)).argsort(-1).argsort(-1) < want[..., None]
    z_idx, z_ptr = np.nonzero(cells)[3].astype(np.int32), want.reshape(-1).cumsum().reshape(B, H, W).astype(np.int32)
    _check_lists_of_large_tiles(z_idx, z_ptr, B, (H, W, D), (1, 1, 1), True)


@pytest.mark.parametrize("D", [1, 2, 31, 32, 33, 64, 95])
@pytest.mark.parametrize("sD,pD", [(1, 0), (1, 1), (1, 4), (2, 1), (3, 2), (2, 31), (1, 33)])
def test_three_deep_filters_across_words_of_the_index(D, sD, pD):
    """Depths whose three neighbours lie in two words of the column index, in front of the first depth and behind the last."""
    if (D + 2 * pD - 3) // sD + 1 < 1:
        pytest.skip("no output")
    rng = np.random.default_rng(D * 100 + pD)
    B, H, W = 2, 3, 5
    cells = rng.random((B, H, W, D)) < 0.6
    z_idx, z_ptr = np.nonzero(cells)[3].astype(np.int32), cells.sum(-1).reshape(-1).cumsum().reshape(B, H, W).astype(np.int32)
    args = (z_idx, z_ptr, B, [H, W, D], [3, 3, 3], [1, 1, sD], [1, 1, pD], [2, 2], False)
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(*args)
    res = oracle_rules(*args)
    assert (oz_idx.cpu().numpy() == res["oz_idx"]).all() and (rule_size.cpu().numpy() == res["rule_size"]).all()
    assert_tables_match(res, rules, z_idx.size, oz_idx.numel())


def test_lists_of_large_tiles_beyond_their_capacity():
    """The kernel of large tiles with lists too short for some tiles: sizes in full, the status bit, no write behind a list; and
    sizes alone."""
    import ctypes
    from sphconv_b200 import _capi as C
    B, H, W, D = 2, 64, 64, 64
    rng = np.random.default_rng(5)
    cells = rng.random((B, H, W, D)) < 0.6
    z_idx, z_ptr = np.nonzero(cells)[3].astype(np.int32), cells.sum(-1).reshape(-1).cumsum().reshape(B, H, W).astype(np.int32)
    zi, zp, osh, oz_idx, oz_ptr, rules, rule_size = gpu_rules(z_idx, z_ptr, B, (H, W, D), (3, 3, 3), (1, 1, 1), (1, 1, 1), (2, 2), True)
    assert rules.shape[0] >= 1024 and oz_idx.numel() >= 256 * rules.shape[0]
    three, two = ctypes.c_int32 * 3, ctypes.c_int32 * 2
    g = C.Geom(B=B, in_shape=three(H, W, D), out_shape=three(H, W, D), ksize=three(3, 3, 3), stride=three(1, 1, 1), padding=three(1, 1, 1),
               tile=two(2, 2), dilation=three(1, 1, 1))
    lib, st, nbr = C.lib(), C.stream_ptr(torch.device(DEV)), rules._sph.nbr
    assert lib.sph_num_tiles(ctypes.byref(g)) == rules.shape[0]
    capacity = int(rule_size.max()) - 20
    short = torch.full((rules.shape[0], 27, 2, capacity), -7, dtype=torch.int32, device=DEV)
    size, status = torch.zeros_like(rule_size), torch.zeros(1, dtype=torch.int32, device=DEV)
    assert lib.sph_rule_lists(C.ptr(oz_ptr), ctypes.byref(g), nbr.shape[1], C.ptr(nbr), capacity, C.ptr(short), C.ptr(size), 0, C.ptr(status), st) == 0
    assert int(status) == C.STATUS_RULE_OVERFLOW and torch.equal(size, rule_size)
    used = (torch.arange(capacity, device=DEV) < rule_size[..., None]).unsqueeze(2).expand_as(short)
    assert torch.equal(short[used], rules[..., :capacity][used]) and (short[~used] == -7).all()
    size.zero_()
    assert lib.sph_rule_lists(C.ptr(oz_ptr), ctypes.byref(g), nbr.shape[1], C.ptr(nbr), 0, None, C.ptr(size), 0, C.ptr(status), st) == 0
    assert torch.equal(size, rule_size)
