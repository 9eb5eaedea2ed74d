"""The nine operators of the reference's ``sphconv.sphconv_cuda`` pybind module
(``src/sphconv/all.cpp:14-38``), same names, argument order and return values, over the C ABI.

Differences a caller can see, all documented:
  * feature dtypes fp32, fp16, bf16 and int8 are accepted (the reference hard-codes float);
  * pairs inside one (tile,k) list come in a deterministic order (the reference's is atomics order);
  * entries of ``rules`` past ``rule_size`` are -1 only when ``config.fill_unused_rules`` is set
    (no consumer reads them, ``include/sphconv/iterator.cu.h:173-177``);
  * errors raise ``RuntimeError`` instead of ``printf``/``exit``;
  * ``dilation`` is honoured: kernel offset k reads input o*stride - padding + k*dilation.  The reference's kernels
    ignore the argument (src/sphconv/rules.cu:40-41) while its ``out_spatial`` sizes the output for a dilated kernel
    (sphconv/utils/__init__.py:40-42); dilation 1, the only value its tests use, behaves identically.

``get_rules*`` attach the neighbour tables the convolution kernels read to the returned ``rules``
tensor (attribute ``_sph``).  Rules without it - cloned, loaded from disk, made elsewhere - are
converted on first use and the result is cached on the tensor until it is modified in place.
"""
import ctypes
import functools
from typing import List, Optional

import torch

from . import _capi as C
from . import profiling


class config:
    """Process-wide switches."""
    fill_unused_rules = True   # -1 padding of `rules` as the reference (rules.cu:364-366)
    materialize_rules = True   # False: module path skips the padded `rules` tensor (rules/rule_size come back None)
    transposed_table = None    # None: build the dgrad table when grad mode is on; True/False forces it
    overlap_rule_lists = True  # module path: write the reference-format pair lists on a side stream, beside the conv
    exact_rule_capacity = False  # True: tile_n_max = the longest list (two passes + a host read), never an overflow


class _Tables:
    """Neighbour tables of one rule set.  nbr[k, o] = input row or -1; nbr_t[k, i] = output row or -1."""
    __slots__ = ("nbr", "nbr_t", "n_in", "n_out", "version", "symmetric")

    def __init__(self, nbr, nbr_t, n_in, n_out, version, symmetric):
        self.nbr, self.nbr_t, self.n_in, self.n_out = nbr, nbr_t, n_in, n_out
        self.version, self.symmetric = version, symmetric


def _want_transposed():
    if config.transposed_table is None:
        return torch.is_grad_enabled()
    return bool(config.transposed_table)


@functools.lru_cache(maxsize=256)
def lists_beside(dtype, kv, in_channels, out_channels, padded):
    """Whether a layer gains from pair lists written on a side stream beside its convolution (us, lists on the side / the caller's
    stream; submanifold layers where not said otherwise).
    The CUDA-core kernels of more than 16 channels do: fp32 32 -> 32 on 284 k / 567 k rows 238 / 260 and 495 / 534, 64 -> 64 500 / 538
    and 977 / 1028, strided 16 -> 32 497 / 503 and 940 / 950, bf16 48 -> 40 on 205 k rows 567 / 591; but fp32 16 -> 16 94 / 91 and 171 / 150.
    The tensor-memory kernel fills the SMs and its blocks start one after the other behind lists beside it: fp16 32 -> 32 99 / 88 and
    180 / 147, 64 -> 64 127 / 112 and 225 / 191, padded lists 191 / 178 and 333 / 298; encoders of 8 layers: fp16 8 scans 1728 / 1706, bf16 training
    16 scans 10340 / 10270, int8 wide 11819 / 11830.
    The other 16-bit kernels gain where the lists are padded, because those wait for the padding: bf16 on 205 k rows 24 -> 40 255 / 260,
    4 -> 16 181 / 186 (16 -> 16 176 / 174), strided on 756 k rows 16 -> 16 451 / 462, 24 -> 40 1016 / 1033; without padding it goes
    either way by 3 %, and by up to 14 % for the caller's stream below 150 k rows (fp16 4 -> 16 on 142 k rows 52 / 44)."""
    if dtype not in C.DTYPE_CODE:
        return False
    layer = (C.DTYPE_CODE[dtype], kv, in_channels, out_channels)
    if C.lib().sph_conv_kernel(*layer, 0) == 0:                  # SPH_KERNEL_GENERAL
        return max(in_channels, out_channels) > 16
    return padded and dtype is not torch.float32 and not C.lib().sph_conv_uses_tmem(*layer)


def _timed_lists(dev, oz_ptr, nbr, nnz, geom, beside):
    """The pair lists as a timed section of their own, on the side stream (`beside`) or behind the table, where the section of the
    rules ends -> (rules, rule_size, ready)."""
    h = C.host()
    side = torch.cuda.ExternalStream(h.side_stream(dev.index), device=dev) if beside else None
    if not beside:
        profiling.mark_stop()
    with profiling.section("lists:" + profiling.current_rule_tag, stream=side):
        return h.lists_of_table(oz_ptr, nbr, nnz, *geom, config.fill_unused_rules, beside)


def _join_lists(rules):
    """Orders the current stream behind the side-stream work that fills `rules` (if any is outstanding).  Called
    by every op right AFTER it has enqueued its own kernel, so that kernel overlaps the lists and everything the
    caller enqueues later sees them complete."""
    ready = getattr(rules, "_sph_ready", None)
    if ready is not None:
        ready.join()
        rules._sph_ready = None


def _attach(rules, rule_size, ready, nbr, nbr_t, n_in, n_out, symmetric):
    """(rules, rule_size) with the tables and the lists' event attached, or (tables, None) without lists."""
    tables = _Tables(nbr, nbr_t, n_in, n_out, 0, symmetric)
    if rules is None:
        return tables, None
    tables.version = rules._version
    rules._sph = tables
    if ready is not None:
        rules._sph_ready = ready
    return rules, rule_size


def get_rules_subm(zIndices: torch.Tensor, zPtr: torch.Tensor, batchSize: int, spatialShape: List[int],
                   outSpatialShape: List[int], kernelSize: List[int], stride: List[int], padding: List[int],
                   dilation: List[int], tileSize: List[int], defer_lists: bool = False, lists_beside: bool = True):
    """ref: get_rules_subm, src/sphconv/rules.cu:326-390.  Returns [zIndices, zPtr, rules, ruleSize]
    (the first two are the input objects, as in the reference).  `defer_lists` (extension, used by the modules):
    rules / ruleSize of large rule sets are written on a side stream and are complete on the current stream only after one of the
    rule_conv* ops has been called with them; not so with `lists_beside` off, for layers that gain nothing from it."""
    geom = (batchSize, spatialShape, outSpatialShape, kernelSize, stride, padding, dilation, tileSize)
    lists = config.materialize_rules
    exact = lists and config.exact_rule_capacity
    defer = defer_lists and config.overlap_rule_lists and lists and not exact
    timed = defer and profiling.is_active() and zIndices.shape[0] > 0
    rules, rule_size, nbr, ready = C.host().rules_subm(zIndices, zPtr, *geom, config.fill_unused_rules,
                                                       lists and not exact and not timed, defer and lists_beside)
    if timed:
        rules, rule_size, ready = _timed_lists(zIndices.device, zPtr, nbr, zIndices.shape[0], geom, lists_beside)
    if exact:
        rules, rule_size = C.host().exact_lists(zPtr, nbr, *geom, config.fill_unused_rules)
    symmetric = all(k % 2 == 1 and p == d * (k // 2) and s == 1 for k, p, s, d in zip(kernelSize, padding, stride, dilation))
    nnz = zIndices.shape[0]
    return [zIndices, zPtr, *_attach(rules, rule_size, ready, nbr, None, nnz, nnz, symmetric)]


def get_rules_begin(zIndices: torch.Tensor, zPtr: torch.Tensor, batchSize: int, spatialShape: List[int],
                    outSpatialShape: List[int], kernelSize: List[int], stride: List[int], padding: List[int],
                    dilation: List[int], tileSize: List[int]):
    """Enqueues step 1 of get_rules (the output sparsity pattern) without waiting for the row count.  Work enqueued after
    this call (the convolution of the previous layer, say) keeps the GPU busy while the host later waits for the count.
    Returns a handle for `get_rules(..., pending=...)`, which completes it."""
    return C.host().strided_begin(zIndices, zPtr, batchSize, spatialShape, outSpatialShape, kernelSize, stride, padding,
                                  dilation, tileSize)


def get_rules(zIndices: torch.Tensor, zPtr: torch.Tensor, batchSize: int, spatialShape: List[int],
              outSpatialShape: List[int], kernelSize: List[int], stride: List[int], padding: List[int],
              dilation: List[int], tileSize: List[int], pending=None, defer_lists: bool = False, lists_beside: bool = True):
    """ref: get_rules, src/sphconv/rules.cu:405-486.  Returns [ozIndices, ozPtr, rules, ruleSize].
    `pending` (extension): the result of get_rules_begin on the same arguments; step 1 is then not run again (a handle of
    other arguments is ignored).  `defer_lists`, `lists_beside` (extensions): as for get_rules_subm."""
    geom = (batchSize, spatialShape, outSpatialShape, kernelSize, stride, padding, dilation, tileSize)
    lists = config.materialize_rules
    exact = lists and config.exact_rule_capacity
    defer = defer_lists and config.overlap_rule_lists and lists and not exact
    timed = defer and profiling.is_active()
    if pending is None:
        pending = get_rules_begin(zIndices, zPtr, *geom)
    oz_idx, oz_ptr, rules, rule_size, nbr, nbr_t, ready = C.host().strided_rules(
        zIndices, zPtr, *geom, pending, config.fill_unused_rules, lists and not exact and not timed, _want_transposed(),
        defer and lists_beside)
    if timed:
        rules, rule_size, ready = _timed_lists(zIndices.device, oz_ptr, nbr, zIndices.shape[0], geom, lists_beside)
    if exact:
        rules, rule_size = C.host().exact_lists(oz_ptr, nbr, *geom, config.fill_unused_rules)
    return [oz_idx, oz_ptr, *_attach(rules, rule_size, ready, nbr, nbr_t, zIndices.shape[0], oz_idx.shape[0], False)]


def _tables_for(rules, rule_size, n_in: int, n_out: int, need_t: bool) -> _Tables:
    """Neighbour tables of a rule set: the ones attached by get_rules*, or a conversion of the
    reference-format tensors (cached on `rules`)."""
    if isinstance(rules, _Tables):
        tb = rules
        if tb.n_in != n_in or tb.n_out != n_out:
            raise RuntimeError("this rule set has %d input and %d output rows, the call %d and %d" % (tb.n_in, tb.n_out, n_in, n_out))
    else:
        tb = getattr(rules, "_sph", None)
        if tb is not None and (tb.version != rules._version or tb.n_in != n_in or tb.n_out != n_out):
            tb = None
    if tb is not None and (not need_t or tb.nbr_t is not None or tb.symmetric):
        return tb
    if isinstance(rules, _Tables):
        raise RuntimeError("this rule set was generated without the transposed table; enable grad mode (or "
                           "config.transposed_table) before generating rules that backward will use")
    nbr, nbr_t = C.host().rules_to_nbr(rules, rule_size, n_in, n_out, tb is None, need_t)
    if tb is not None:
        nbr = tb.nbr
    new = _Tables(nbr, nbr_t, n_in, n_out, rules._version, tb.symmetric if tb is not None else False)
    rules._sph = new
    return new


def _packed_weight(weight: torch.Tensor):
    """UMMA image of a [KV, K, N] weight, or None when the CUDA-core kernel will run.  Cached on the tensor."""
    cached = getattr(weight, "_sph_packed", None)
    if cached is not None and cached[0] == weight._version:
        return cached[1]
    packed = C.host().pack_weight(weight)
    weight._sph_packed = (weight._version, packed)
    return packed


def _gather(rows, weight, nbr, n_out, flip_k, scale, bias, relu, out_dtype):
    return C.host().conv_gather(rows, weight, _packed_weight(weight), nbr, n_out, flip_k, scale, bias, relu, out_dtype)


def rule_conv(feature: torch.Tensor, weight: torch.Tensor, rules, ruleSize, outNNZ: int, *,
              scale: Optional[torch.Tensor] = None, bias: Optional[torch.Tensor] = None, relu: bool = False,
              out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """ref: rule_conv, src/sphconv/rule_conv.cu:286-336.  feature [NNZ,iC], weight [KV,iC,oC] ->
    [outNNZ,oC].  Keyword arguments are extensions (fused epilogue relu(acc*scale + bias), output dtype); `scale` is
    float32, `bias` float32 or of the features' 16-bit type."""
    tb = _tables_for(rules, ruleSize, feature.shape[0], int(outNNZ), need_t=False)
    out = _gather(feature, weight, tb.nbr, int(outNNZ), False, scale, bias, relu, out_dtype)
    if getattr(rules, "_sph_ready", None) is not None:
        profiling.mark_stop()          # a timed section around this call ends with the kernel, not with the join
        _join_lists(rules)
    return out


def rule_conv_d_feature(feature: torch.Tensor, weight: torch.Tensor, rules, ruleSize,
                        tile_grid_shape: List[int], outNNZ: int) -> torch.Tensor:
    """ref: rule_conv_d_feature, src/sphconv/rule_conv.cu:520-575.  `feature` is the upstream gradient
    [outNNZ_fwd, oC], `weight` the [KV,oC,iC] transpose, `outNNZ` the number of input rows; returns [outNNZ, iC].
    tile_grid_shape is accepted for signature compatibility (the reference needs it for its 9-colour launches)."""
    n_in = int(outNNZ)
    tb = _tables_for(rules, ruleSize, n_in, feature.shape[0], need_t=True)
    if tb.nbr_t is not None:
        return _gather(feature, weight, tb.nbr_t, n_in, False, None, None, False, None)
    # odd-kernel submanifold layer: (i,o) at k  <=>  (o,i) at KV-1-k, so the forward table serves
    return _gather(feature, weight, tb.nbr, n_in, True, None, None, False, None)


def rule_conv_d_weight(feature: torch.Tensor, d_featureOut: torch.Tensor, rules, ruleSize, *,
                       out: Optional[torch.Tensor] = None, accumulate: bool = False) -> torch.Tensor:
    """ref: rule_conv_d_weight, src/sphconv/rule_conv.cu:469-518.  Returns float32 [KV,iC,oC].
    Keyword arguments are extensions: `out` is a caller-owned contiguous float32 [KV,iC,oC] tensor (e.g. a slice
    of a flat gradient buffer) the kernel writes instead of a fresh one; with `accumulate` it adds to what is there."""
    tb = _tables_for(rules, ruleSize, feature.shape[0], d_featureOut.shape[0], need_t=False)
    dw = C.host().conv_wgrad(feature, d_featureOut, tb.nbr, out, accumulate)
    _join_lists(rules)
    return dw


def rule_conv_backward(d_featureOut: torch.Tensor, feature: torch.Tensor, weight: torch.Tensor, rules, ruleSize,
                       tile_grid_shape: List[int]):
    """ref: rule_conv_backward, src/sphconv/rule_conv.cu:577-597.  `weight` is [KV,oC,iC].
    Returns [d_feature [NNZ,iC], d_weight [KV,iC,oC]] in the dtype of `feature`."""
    d_featureOut = d_featureOut.contiguous()
    d_feature = rule_conv_d_feature(d_featureOut, weight, rules, ruleSize, tile_grid_shape, feature.shape[0])
    d_weight = rule_conv_d_weight(feature, d_featureOut, rules, ruleSize).to(feature.dtype)
    return [d_feature, d_weight]


def conv_layer(feature, weight, bias, rules, tables, n_out, relu):
    """relu(conv + bias) as one differentiable native call (extension): what functional.ConvFunction does, for a rule set
    whose tables serve both directions."""
    out = C.host().conv_layer(feature, weight, bias, tables.nbr, None if tables.symmetric else tables.nbr_t, n_out, relu)
    _join_lists(rules)
    return out


# ---- tensor ops on either side of the path: COO -> range-voxel, range-voxel <-> dense -----------------------

def init_tensor(feature: torch.Tensor, indicesBZYX: torch.Tensor, batchSize: int, spatialShape: List[int]):
    """ref: init_tensor, src/sphconv/tensor.cu:78-127.  COO (b, s0, s1, s2) -> range-voxel.
    Returns [feature', zIndices, zPtr, permutation] with permutation[n] = new row of input row n.
    Rows inside a column are ordered by depth (the reference's order is atomics arrival order).  Any dtype."""
    return list(C.host().init_tensor(feature, indicesBZYX, batchSize, spatialShape))


def init_tensor_backward(d_featureOut: torch.Tensor, permutation: torch.Tensor) -> torch.Tensor:
    """ref: init_tensor_backward, src/sphconv/tensor.cu:147-162: d_feature[n] = d_featureOut[permutation[n]]."""
    return C.host().gather_rows(d_featureOut, permutation)


def _shape3(spatialShape):
    return (ctypes.c_int32 * 3)(*[int(v) for v in spatialShape])


def to_dense(feature: torch.Tensor, zIndices: torch.Tensor, zPtr: torch.Tensor, D: int, out: torch.Tensor):
    """ref: to_dense, src/sphconv/tensor.cu:222-264.  Fills out [B,H,W,D,C] in place and returns it.
    The integer argument is unused, as in the reference kernel, which takes every size from `out`."""
    C.require_cuda(feature, zIndices, zPtr, out)
    if not out.is_contiguous() or out.dim() != 5 or out.dtype != feature.dtype or out.shape[4] != feature.shape[1]:
        raise RuntimeError("out must be a contiguous [B,H,W,D,C] tensor of the feature dtype")
    f = feature.contiguous()
    with torch.cuda.device(f.device):
        C.check(C.lib().sph_to_dense(C.ptr(f), f.shape[1] * f.element_size(), f.shape[0], C.ptr(zIndices.contiguous()),
                                     C.ptr(zPtr.contiguous()), out.shape[0], _shape3(out.shape[1:4]), C.ptr(out), 0,
                                     C.ptr(C.status_tensor(f.device)), C.stream_ptr(f.device)))
    return out


def to_dense_backward(d_featureOut: torch.Tensor, zIndices: torch.Tensor, zPtr: torch.Tensor) -> torch.Tensor:
    """ref: to_dense_backward, src/sphconv/tensor.cu:266-309.  d_featureOut [B,H,W,D,C] -> [NNZ,C]."""
    C.require_cuda(d_featureOut, zIndices, zPtr)
    d = d_featureOut.contiguous()
    nnz = zIndices.shape[0]
    out = torch.empty((nnz, d.shape[4]), dtype=d.dtype, device=d.device)
    with torch.cuda.device(d.device):
        C.check(C.lib().sph_to_dense(C.ptr(out), d.shape[4] * d.element_size(), nnz, C.ptr(zIndices.contiguous()),
                                     C.ptr(zPtr.contiguous()), d.shape[0], _shape3(d.shape[1:4]), C.ptr(d), 1,
                                     C.ptr(C.status_tensor(d.device)), C.stream_ptr(d.device)))
    return out


def dense_in_one_pass(t: torch.Tensor, batch: int, channels: int, depth: int) -> bool:
    """Whether dense_channels_first takes these sizes (elements of 1 to 8 bytes, columns of up to 2048 cells)."""
    return depth <= 2048 and 0 < batch <= 65535 and channels > 0 and t.element_size() <= 8


def dense_channels_first(feature: torch.Tensor, zIndices: torch.Tensor, zPtr: torch.Tensor, shape: List[int]):
    """Rows [NNZ,C] -> dense [B,C,s0,s1,s2], written in one pass (extension; the reference scatters channels-last and
    permutes, sphconv/functional.py:81-106).  shape = [B, C, s0, s1, s2]."""
    return C.host().dense_channels_first(feature, zIndices, zPtr, shape, False)


def dense_channels_first_backward(d_dense: torch.Tensor, zIndices: torch.Tensor, zPtr: torch.Tensor):
    """Dense gradient [B,C,s0,s1,s2] -> rows [NNZ,C]."""
    return C.host().dense_channels_first(d_dense, zIndices, zPtr, list(d_dense.shape), True)


def epilogue_backward(d_out: torch.Tensor, out: Optional[torch.Tensor], relu: bool, need_bias: bool):
    """Backward of the fused epilogue relu(acc + bias) (extension, no reference counterpart): returns
    (d_pre, d_bias fp32 [C] or None) with d_pre = d_out masked by (out > 0) when `relu`."""
    d_pre, d_bias = C.host().epilogue_backward(d_out.contiguous(), None if out is None else out.contiguous(), bool(relu),
                                               bool(need_bias))
    return (d_pre if relu else d_out), d_bias
