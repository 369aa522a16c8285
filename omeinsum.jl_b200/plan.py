"""Contraction-tree execution (NestedEinsum, SlicedEinsum, cost_and_gradient)
through the library's plan API (ome_plan_* in include/ome_b200.h).

A tree is flattened once into post-order arrays, planned once per (tree,
sizes, slicing, dtype, precision) and cached; evaluation is one library call
that runs every node from the device workspace.
"""
from __future__ import annotations

import ctypes as C
import weakref
from typing import Any, Dict, List, Sequence, Tuple

import torch

from . import _lib
from ._lib import ArgumentError, check
from .backends import B200Backend, get_einsum_backend
from .core import NestedEinsum, SlicedEinsum, get_size_dict
from .engine import (_TLS, _TORCH_TO_OME, TropicalTensor, _alloc, _colmajor_strides, _current_device, _f_contig,
                     _LabelMap, _Prepared, _raw_stream, _require_b200, _scalar_buf, _stream, plain_layout)


class Plan:
    """A planned contraction tree in the library (owns an ome_plan*)."""

    def __init__(self, ne: NestedEinsum, slicing: Sequence[Any], size_dict: Dict[Any, int], ome_dtype: int,
                 prec: int):
        lm = _LabelMap()
        nodes: List[Tuple[List[int], List[int]]] = []
        inputs: Dict[int, List[int]] = {}

        def rec(n: NestedEinsum) -> int:
            refs = []
            for ix, a in zip(n.eins.ixs, n.args):
                if a.isleaf:
                    inputs[a.tensorindex] = [lm(l) for l in ix]
                    refs.append(-a.tensorindex - 1)
                else:
                    refs.append(rec(a))
            nodes.append((refs, [lm(l) for l in n.eins.iy]))
            return len(nodes) - 1

        rec(ne)
        self.ninputs = len(inputs)
        if sorted(inputs) != list(range(self.ninputs)):
            raise ArgumentError("leaf tensor indices must be 0..n-1, each used once")
        for l in slicing:
            lm(l)
        self.labels = lm.ids
        self.out_labels = list(ne.eins.iy)
        in_n = [len(inputs[t]) for t in range(self.ninputs)]
        in_l = [x for t in range(self.ninputs) for x in inputs[t]]
        nn = [len(r) for r, _ in nodes]
        na = [x for r, _ in nodes for x in r]
        ny = [len(y) for _, y in nodes]
        nyl = [x for _, y in nodes for x in y]
        lab_ids = list(range(len(lm.ids)))
        inv = {v: k for k, v in lm.ids.items()}
        for i in lab_ids:
            if inv[i] not in size_dict:
                raise ArgumentError(f"label {inv[i]} has no size")
        exts = [int(size_dict[inv[i]]) for i in lab_ids]
        sl = [lm.ids[l] for l in slicing]
        arr = lambda T, v: (T * max(len(v), 1))(*v)
        h = C.c_void_p()
        check(_lib.load().ome_plan_create(
            None, ome_dtype, self.ninputs, arr(C.c_int32, in_n), arr(C.c_int32, in_l), len(nodes),
            arr(C.c_int32, nn), arr(C.c_int32, na), arr(C.c_int32, ny), arr(C.c_int32, nyl), len(lab_ids),
            arr(C.c_int32, lab_ids), arr(C.c_int64, exts), len(sl), arr(C.c_int32, sl), prec, C.byref(h)))
        self.handle = h
        fb, gb = C.c_size_t(), C.c_size_t()
        check(_lib.load().ome_plan_peak_bytes(h, C.byref(fb), C.byref(gb)))
        self.forward_bytes = fb.value
        self.grad_bytes = gb.value
        check(_lib.load().ome_plan_min_bytes(h, C.byref(fb), C.byref(gb)))
        self.forward_min, self.grad_min = fb.value, gb.value
        self.ome_dtype = ome_dtype

    def __del__(self):
        try:
            if self.handle:
                _lib.load().ome_plan_destroy(self.handle)
        except Exception:
            pass


_CACHE: Dict[Any, Plan] = {}


def _tree_key(ne: NestedEinsum):
    if ne.isleaf:
        return ne.tensorindex
    return (tuple(_tree_key(a) for a in ne.args), tuple(map(tuple, ne.eins.ixs)), tuple(ne.eins.iy))


def get_plan(code, size_dict, ome_dtype, prec) -> Plan:
    if isinstance(code, SlicedEinsum):
        ne, slicing = code.eins, list(code.slicing)
    else:
        ne, slicing = code, []
    labels = set(l for ix in ne.getixsv() for l in ix) | set(ne.getiyv())
    key = (_tree_key(ne), tuple(slicing), tuple(sorted((repr(l), size_dict[l]) for l in labels if l in size_dict)),
           ome_dtype, prec)
    p = _CACHE.get(key)
    if p is None:
        p = Plan(ne, slicing, size_dict, ome_dtype, prec)
        _CACHE[key] = p
    return p


# ----------------------------------------------------------------------------
# repeated calls: what a tree's evaluation needs besides its data
# ----------------------------------------------------------------------------

# An input of at most this many elements is read in place whatever its strides;
# larger ones in another order than column-major are copied once per call, as
# every slice and every gradient reads them again.
_IN_PLACE = 4096


class _TreeState:
    """What was seen of a tree object: its nodes with copies of their lists, so
    that a later call notices any change, and the calls prepared for trees of
    its structure.  The tree itself (`code` and its root) is not kept alive."""

    def __init__(self, code, root, calls):
        self.slicing = tuple(code.slicing) if code is not root else ()
        self.root = (tuple(root.args), root.eins, tuple(root.eins.ixs), root.eins.iy)
        self.nodes = []
        todo = list(root.args)
        while todo:
            n = todo.pop()
            if n.tensorindex < 0:
                self.nodes.append((n, tuple(n.args), n.eins, tuple(n.eins.ixs), n.eins.iy))
                todo.extend(n.args)
            else:
                self.nodes.append((n, n.tensorindex, None, None, None))
        self.calls: Dict[Any, "_TreeCall"] = calls

    def holds(self, code, root) -> bool:
        if code is not root and tuple(code.slicing) != self.slicing:
            return False
        args, eins, ixs, iy = self.root
        if root.tensorindex >= 0 or root.eins is not eins or tuple(root.args) != args or tuple(eins.ixs) != ixs or \
                eins.iy != iy:
            return False
        for n, args, eins, ixs, iy in self.nodes:
            if eins is None:
                if n.tensorindex != args:
                    return False
            elif n.eins is not eins or tuple(n.args) != args or tuple(eins.ixs) != ixs or eins.iy != iy:
                return False
        return True


class _TreeCall:
    """A tree evaluated on one layout of plain CUDA inputs (per host thread)."""

    def __init__(self, code, ne, xs, dt, dev, ome, prec, grad):
        size_dict = get_size_dict(ne.getixsv() if grad else code.getixsv(), xs)
        self.plan = get_plan(ne if grad else code, size_dict, ome, prec)
        self.shape = tuple(size_dict[l] for l in ne.eins.iy)
        self.strides = _colmajor_strides(self.shape)
        self.device, self.dtype, self.dev = torch.device("cuda", dev), dt, dev
        self.copied = [i for i, t in enumerate(xs)
                       if t.numel() > _IN_PLACE and tuple(t.stride()) != _colmajor_strides(t.shape)]
        self.xlay = [(tuple(t.shape), _colmajor_strides(t.shape)) for t in xs]
        st = [s for i, t in enumerate(xs) for s in (self.xlay[i][1] if i in self.copied else t.stride())]
        self.str = (C.c_int64 * max(len(st), 1))(*st)
        self.one, self.zero = _scalar_buf(ome, True), _scalar_buf(ome, False)

    def prepare(self, xs):
        """The inputs (kept alive by the caller until the launch returns) and their pointers."""
        if self.copied:
            xs = list(xs)
            for i in self.copied:
                xs[i] = _f_contig(xs[i])
        return xs, _ptrs(xs)


_STATES_MAX = 128


def _tree_state(code, root) -> _TreeState:
    """The state of a tree object, per host thread: kept while the object lives
    and is unchanged.  An object seen for the first time takes over the calls
    that were prepared for another of the same structure (a two-node tree
    parsed and called 42 us, 74 when planned by itself; the same object 21)."""
    states = getattr(_TLS, "trees", None)
    if states is None:
        states = _TLS.trees = {}
        _TLS.tree_calls = {}
    key = id(code)
    held = states.get(key)
    if held is not None and held[0]() is code and held[1].holds(code, root):
        return held[1]
    by_structure = _TLS.tree_calls
    structure = (_tree_key(root), tuple(code.slicing) if code is not root else None)
    calls = by_structure.pop(structure, None)   # (last used last)
    if calls is None:
        calls = {}
        if len(by_structure) >= _STATES_MAX:
            by_structure.pop(next(iter(by_structure)), None)
    by_structure[structure] = calls

    def forget(ref):
        if states.get(key, (None,))[0] is ref:
            states.pop(key, None)

    if len(states) >= _STATES_MAX:
        states.pop(next(iter(states)), None)
    states[key] = (weakref.ref(code, forget), _TreeState(code, root, calls))
    return states[key][1]


def _tree_call(code, xs, grad):
    """(call, tropical, raw inputs) of a tree on plain CUDA inputs, or None."""
    be = get_einsum_backend()
    if not isinstance(be, B200Backend) or len(xs) == 0 or type(code) not in (NestedEinsum, SlicedEinsum):
        return None
    root = code.eins if type(code) is SlicedEinsum else code
    if type(root) is not NestedEinsum or root.tensorindex >= 0:
        return None
    trop = type(xs[0]) is TropicalTensor
    if trop:
        if any(type(x) is not TropicalTensor for x in xs):
            return None
        xs = [x.data for x in xs]
    lay = plain_layout(xs)
    if lay is None:
        return None
    dt, dev, shapes = lay
    if dev != _current_device():
        return None
    calls = _tree_state(code, root).calls
    key = (grad, trop, be.prec, dt, dev, *shapes)
    call = calls.get(key)
    if call is None:
        ome = (_lib.TROP_F32 if dt == torch.float32 else _lib.TROP_F64) if trop else _TORCH_TO_OME[dt]
        call = _TreeCall(code, root, xs, dt, dev, ome, be.prec, grad)
        if len(calls) >= 16:
            calls.pop(next(iter(calls)))
        calls[key] = call
    return call, trop, xs


def tree_plain(code, xs):
    """The tree's value for plain CUDA inputs, or None if the call needs the
    general path (which also raises the errors)."""
    try:
        got = _tree_call(code, xs, False)
    except TypeError:   # unhashable labels
        return None
    if got is None:
        return None
    call, trop, raw = got
    raw, ptrs = call.prepare(raw)
    ctx = _lib.context(call.dev, call.plan.forward_bytes, call.plan.forward_min)
    y = torch.empty_strided(call.shape, call.strides, dtype=call.dtype, device=call.device)
    check(_lib.load().ome_plan_execute_strided(ctx.handle, call.plan.handle, _raw_stream(call.dev), ptrs, call.str,
                                               y.data_ptr(), call.one, call.zero))
    return TropicalTensor(y) if trop else y


def gradient_plain(code, xs):
    """cost_and_gradient of a scalar tree on plain CUDA inputs, or None."""
    try:
        got = _tree_call(code, xs, True)
    except TypeError:
        return None
    if got is None or got[0].shape != ():
        return None
    call, trop, raw = got
    raw, ptrs = call.prepare(raw)
    ctx = _lib.context(call.dev, call.plan.grad_bytes, call.plan.grad_min)
    y = torch.empty_strided(call.shape, call.strides, dtype=call.dtype, device=call.device)
    new, dt, dev = torch.empty_strided, call.dtype, call.device
    dxs = [new(sh, st, dtype=dt, device=dev) for sh, st in call.xlay]
    check(_lib.load().ome_plan_gradient_strided(ctx.handle, call.plan.handle, _raw_stream(call.dev), ptrs, call.str,
                                                None, y.data_ptr(), _ptrs(dxs)))
    if trop:
        return TropicalTensor(y), [TropicalTensor(d) for d in dxs]
    return y, dxs


def _ptrs(ts: Sequence[torch.Tensor]):
    return (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def run_tree(code, xs, size_dict=None, y=None, sx=True, sy=False):
    """einsum / einsum! for NestedEinsum and SlicedEinsum."""
    be = _require_b200()
    ne = code.eins if isinstance(code, SlicedEinsum) else code
    if size_dict is None:
        size_dict = get_size_dict(code.getixsv(), xs)
    if ne.isleaf:
        raise ArgumentError("a bare leaf is not a contraction")
    out_dtype = None
    if y is not None:
        out_dtype = (y.data if isinstance(y, TropicalTensor) else y).dtype
    p = _Prepared(xs, out_dtype=out_dtype)
    plan = get_plan(code, size_dict, p.ome, be.prec)
    dev = p.device
    ctx = _lib.context(dev.index, plan.forward_bytes, plan.forward_min)
    ins = [_f_contig(t) for t in p.tensors]
    shape = [size_dict[l] for l in ne.eins.iy]
    if y is None:
        yt = _alloc(shape, p.dtype, dev)
    else:
        yt = y.data if isinstance(y, TropicalTensor) else y
        if tuple(yt.shape) != tuple(shape):
            raise _lib.DimensionMismatch(f"output shape {tuple(yt.shape)} != {tuple(shape)}")
    work = yt if (y is None or tuple(yt.stride()) == tuple(_f_contig(yt).stride())) else _f_contig(yt)
    with torch.cuda.device(dev):
        check(_lib.load().ome_plan_execute(ctx.handle, plan.handle, _stream(dev), _ptrs(ins), work.data_ptr(),
                                           _scalar_buf(p.ome, sx), _scalar_buf(p.ome, sy)))
    if work is not yt:
        yt.copy_(work)
    if y is not None:
        return y
    return p.wrap(yt)


def tree_gradient(code, xs, dy=None):
    """cost_and_gradient on the device: forward with cached intermediates, then
    einsum_grad per node (src/bp.jl:99-130)."""
    be = _require_b200()
    if dy is None:
        got = gradient_plain(code, xs)
        if got is not None:
            return got
    ne = code.eins if isinstance(code, SlicedEinsum) else code
    if isinstance(code, NestedEinsum) or isinstance(code, SlicedEinsum):
        pass
    else:
        # a flat EinCode: a one-node tree
        ne = NestedEinsum([NestedEinsum(i) for i in range(len(code.ixs))], code)
    size_dict = get_size_dict(ne.getixsv(), xs)
    p = _Prepared(xs)
    plan = get_plan(ne, size_dict, p.ome, be.prec)
    dev = p.device
    ctx = _lib.context(dev.index, plan.grad_bytes, plan.grad_min)
    ins = [_f_contig(t) for t in p.tensors]
    shape = [size_dict[l] for l in ne.eins.iy]
    yt = _alloc(shape, p.dtype, dev)
    dxs = [_alloc(t.shape, p.dtype, dev) for t in ins]
    dyp = None
    if dy is not None:
        dyt = dy.data if isinstance(dy, TropicalTensor) else torch.as_tensor(dy)
        dyt = _f_contig(dyt.to(device=dev, dtype=p.dtype).resolve_conj().resolve_neg())
        if tuple(dyt.shape) != tuple(shape):
            raise _lib.DimensionMismatch("dy has the wrong shape")
        dyp = dyt
    elif len(shape) != 0:
        raise ArgumentError(f"The output must be a scalar! Or you need to feed the gradient manually. Got: {len(shape)}!")
    with torch.cuda.device(dev):
        check(_lib.load().ome_plan_gradient(ctx.handle, plan.handle, _stream(dev), _ptrs(ins),
                                            dyp.data_ptr() if dyp is not None else None, yt.data_ptr(),
                                            _ptrs(dxs)))
    return p.wrap(yt), [p.wrap(d) for d in dxs]
