"""`Tree` / `EvoTree` containers with the reference's field layout (src/structs.jl:77-138) and inference."""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass, field
from operator import is_

import numpy as np

from . import _lib
from .binning import binarize


@dataclass
class Tree:
    """Heap-indexed complete binary tree of 2^depth - 1 nodes (the bias tree has one node).
    feat / cond_bin are 1-based, 0 = no split, exactly as in the reference."""
    feat: np.ndarray      # int64 [nn]
    cond_bin: np.ndarray  # uint8 [nn]
    w: np.ndarray         # float32 [nn]
    gain: np.ndarray      # float32 [nn]
    pred: np.ndarray      # float32 [nn, K]; row n is the reference's pred[:, n]
    split: np.ndarray     # bool [nn]

    def __setattr__(self, name, value):
        _Packed.rebinds += 1      # a tree may have been given other arrays: packed models look again
        object.__setattr__(self, name, value)

    @staticmethod
    def empty(depth: int, K: int) -> "Tree":
        nn = 2 ** depth - 1
        t = object.__new__(Tree)  # a new tree is in no packed model yet
        t.__dict__.update(feat=np.zeros(nn, np.int64), cond_bin=np.zeros(nn, np.uint8), w=np.zeros(nn, np.float32),
                          gain=np.zeros(nn, np.float32), pred=np.zeros((nn, K), np.float32), split=np.zeros(nn, np.uint8))
        return t

    @staticmethod
    def bias(mu: np.ndarray) -> "Tree":
        t = Tree.empty(1, mu.size)
        t.pred[0, :] = mu
        return t


@dataclass
class EvoTree:
    loss: str
    K: int
    trees: list = field(default_factory=list)
    info: dict = field(default_factory=dict)

    def __getstate__(self):      # copies and pickles of a model pack its trees anew
        return {k: v for k, v in self.__dict__.items() if k != "_dev"}

    def __call__(self, x, ntree_limit: int | None = None, device: int = 0):
        return predict(self, x, ntree_limit=ntree_limit, device=device)


def _pack(m: EvoTree, ntree_limit: int):
    nn = max(t.feat.size for t in m.trees[:ntree_limit])
    K = m.K
    feat = np.zeros((ntree_limit, nn), np.int64)
    cb = np.zeros((ntree_limit, nn), np.uint8)
    sp = np.zeros((ntree_limit, nn), np.uint8)
    lp = np.zeros((ntree_limit, nn, K), np.float32)
    for i, t in enumerate(m.trees[:ntree_limit]):
        k = t.feat.size
        feat[i, :k], cb[i, :k], sp[i, :k], lp[i, :k] = t.feat, t.cond_bin, t.split, t.pred
    return nn, feat, cb, sp, lp


_TREE_TYPES = [np.dtype(d) for d in (np.int64, np.uint8, np.uint8, np.float32)]


_addressof, _from_buffer = C.addressof, C.c_char.from_buffer


def _tree_arrays(t: Tree):
    return t.feat, t.cond_bin, t.split, t.pred


class _Packed:
    """A model's trees, packed on one device (`evb_model_create`), and the arrays they were packed from.  `current` says
    whether the model still consists of those arrays; whether their contents are still the same is checked by
    `evb_model_predict` itself, while the GPU works."""
    rebinds = 0     # attribute assignments on any `Tree` so far

    def __init__(self, m: EvoTree, device: int):
        self.rebinds = _Packed.rebinds
        self.device, self.loss, self.K = device, m.loss, m.K
        self.trees = list(m.trees)
        self.edges, self.feattypes = m.info["edges"], m.info["feattypes"]
        self.shared = True                  # the library reads the model's own arrays, not copies
        arrays = [a for t in self.trees for a in (t.feat, t.cond_bin, t.split, t.pred)]
        n, src = len(self.trees), None
        size = [a.size for a in arrays]
        if size[1::4] != size[::4] or size[2::4] != size[::4] or size[3::4] != [s * m.K for s in size[::4]]:
            raise ValueError("the arrays of a tree must have one entry per node")
        if [a.dtype for a in arrays] == _TREE_TYPES * n:
            try:                            # C-contiguous and writable, or it raises; a third of the time of the array interface
                src = [_addressof(_from_buffer(a)) for a in arrays]
            except (TypeError, ValueError):
                pass
        if src is None:
            for i, a in enumerate(arrays):
                dt = _TREE_TYPES[i % 4]
                if a.dtype != dt and not (dt.itemsize == 1 and a.dtype == bool) or not a.flags.c_contiguous:
                    arrays[i], self.shared = np.ascontiguousarray(a, dt), False
            src = [a.__array_interface__["data"][0] for a in arrays]
        e, ft = np.asarray(self.edges), np.asarray(self.feattypes)
        if e.dtype not in (np.float32, np.float64) or not e.flags.c_contiguous:
            e, self.shared = np.ascontiguousarray(e, np.float64), False
        if ft.dtype not in (bool, np.uint8) or not ft.flags.c_contiguous:
            ft, self.shared = np.ascontiguousarray(ft, np.uint8), False
        self.arrays = arrays
        self.keep = (e, ft)
        src = np.array(src, np.uint64)
        nodes = np.array(size[::4], np.int32)
        self.handle = C.c_void_p()
        _lib.check(_lib.lib().evb_model_create(
            C.byref(self.handle), C.c_int32(device), C.c_int32(_lib.LOSS_CODES[m.loss]), C.c_int32(m.K), C.c_int32(n), _lib.ptr(src), _lib.ptr(nodes),
            _lib.ptr(e), C.c_int32(_lib.EVB_F32 if e.dtype == np.float32 else _lib.EVB_F64), C.c_int32(e.shape[1]), C.c_int32(e.shape[0]), _lib.ptr(ft)))
        self.ptr = self.handle.value
        self.nfeats = e.shape[0]

    def current(self, m: EvoTree, device: int) -> bool:
        if not (self.shared and self.device == device and self.loss == m.loss and self.K == m.K and self.edges is m.info["edges"] and
                self.feattypes is m.info["feattypes"] and len(self.trees) == len(m.trees) and all(map(is_, self.trees, m.trees))):
            return False
        if self.rebinds != _Packed.rebinds:
            now = _Packed.rebinds
            if not all(map(is_, self.arrays, [a for t in m.trees for a in _tree_arrays(t)])):
                return False
            self.rebinds = now
        return True

    def __del__(self):
        try:
            _lib.lib().evb_model_destroy(self.handle)
        except Exception:
            pass


def _packed(m: EvoTree, device: int, fresh: bool = False) -> _Packed:
    c = None if fresh else m.__dict__.get("_dev")
    if c is None or not c.current(m, device):
        m.__dict__.pop("_dev", None)
        c = m.__dict__["_dev"] = _Packed(m, device)
    return c


def _run(m: EvoTree, x, ntree_limit, device, apply_link: bool, want_leaf: bool, stats: dict | None = None):
    """Binarize on the device and apply the trees in one call (`evb_model_predict`).  `x` may be C- or Fortran-ordered:
    no host-side transpose is made."""
    ntrees = len(m.trees)
    ntree_limit = ntrees if ntree_limit is None else ntree_limit
    if ntree_limit > ntrees:
        raise ValueError(f"ntree_limit is larger than number of trees {ntrees}.")
    x = np.asarray(x)
    if x.dtype not in (np.float32, np.float64):
        x = x.astype(np.float64)
    row_major = x.flags.c_contiguous      # one row, one column: either order describes it
    if not (row_major or x.flags.f_contiguous):
        x = np.asfortranarray(x)
    nobs, nfeats = x.shape
    lib = _lib.lib()
    p = _packed(m, device)
    if nfeats != p.nfeats:
        raise ValueError(f"x has {nfeats} columns, the model was trained on {p.nfeats}")
    out = np.empty(nobs, np.float32) if m.K == 1 else np.empty((nobs, m.K), np.float32, order="F")
    leaf = np.empty((nobs, ntree_limit), np.uint32, order="F") if want_leaf else None
    kms = None if stats is None else C.c_double(0.0)
    while True:
        rc = lib.evb_model_predict(p.ptr, ntree_limit, x.ctypes.data, 0 if x.dtype == np.float32 else 2, row_major, nobs, apply_link,
                                   out.ctypes.data, None if leaf is None else leaf.ctypes.data, None if kms is None else C.addressof(kms))
        if rc != _lib.ERR_STALE:
            break
        p = _packed(m, device, fresh=True)
    _lib.check(rc)
    if stats is not None:
        stats["kernel_ms"] = kms.value
    return out, leaf


def predict_binned(m: EvoTree, x_bin: np.ndarray, ntree_limit: int | None = None, device: int = 0, apply_link: bool = True):
    """Inference from an already binned matrix (uint8, Fortran order) through `evb_predict`."""
    ntree_limit = len(m.trees) if ntree_limit is None else ntree_limit
    nobs, nfeats = x_bin.shape
    nn, feat, cb, sp, lp = _pack(m, ntree_limit)
    out = np.empty((nobs, m.K), np.float32, order="F")
    ft = np.ascontiguousarray(m.info["feattypes"], np.uint8)
    _lib.check(_lib.lib().evb_predict(C.c_int32(device), C.c_int32(_lib.LOSS_CODES[m.loss]), C.c_int32(m.K),
                                      C.c_int32(ntree_limit), C.c_int32(nn), _lib.ptr(feat), _lib.ptr(cb), _lib.ptr(sp),
                                      _lib.ptr(lp), _lib.ptr(x_bin), C.c_int64(nobs), C.c_int32(nfeats), _lib.ptr(ft),
                                      C.c_int32(1 if apply_link else 0), _lib.ptr(out), None))
    return out


def predict(m: EvoTree, x, ntree_limit: int | None = None, device: int = 0, stats: dict | None = None) -> np.ndarray:
    """`predict(m, data; ntree_limit, device=:gpu)` (src/predict.jl:93-96): sums the trees and applies the
    loss's inverse link.  Returns [nobs] when K == 1, else [nobs, K]."""
    out, _ = _run(m, x, ntree_limit, device, True, False, stats)
    return out


def predict_leaf_idx(m: EvoTree, x, ntree_limit: int | None = None, device: int = 0) -> np.ndarray:
    """`predict_leaf_idx(m, data; ntree_limit)` (src/predict.jl:173-185): uint32 [nobs, ntree_limit]."""
    _, leaf = _run(m, x, ntree_limit, device, False, True)
    return leaf
