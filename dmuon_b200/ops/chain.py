"""Newton-Schulz as one launch: plans for the product-chain kernel
(``csrc/chain_sm100.cu``).

A *group* is a batch of ``L`` matrices of one shape.  A *program* covers one or more
groups: the list of products and the tile list, on the device, used by every call with
the same shapes.  A *plan* is a program with work memory: the buffers of one stream and
the tensor maps over them (which travel as parameters of each launch).  A call supplies
only what changes: where the results go and the scale of the last product (plus the
operands, written into ``plan.X[group][matrix]`` beforehand).

The tile list is ordered product by product, all groups side by side; every entry
names the number of finished warps its matrix must show before the tile may start
(see the kernel source for why that cannot deadlock).
"""
from __future__ import annotations

import ctypes
import math
import threading
from collections import OrderedDict
from dataclasses import dataclass
from functools import lru_cache
from typing import Optional, Sequence

import numpy as np
import torch

from . import build as _build
from . import gemm as G

MAX_OPS = 76
MAX_GROUPS = 16
MAX_MAPS = 128                # tensor maps, which travel in the kernel's parameters
SMS = 148
PAIRS = SMS // 2
_KB = 64                      # inner elements per pipeline stage
_SUM_COLS = 64                # columns of one entry of a sum of partial products
WARPS_PER_TILE = 8            # epilogue warps per CTA: each reports a finished tile
PAIR = 256                    # tile width that stands for CTA pairs on 256 x 256 tiles

_VP, _LL, _I, _F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float


class _Op(ctypes.Structure):
    _fields_ = [
        ("map_a", _I), ("map_b", _I), ("a_mn_major", _I), ("b_mn_major", _I), ("ab_fp16", _I),
        ("M", _I), ("N", _I), ("K", _I), ("kb_per_split", _I), ("splits", _I), ("out_kind", _I), ("final_slot", _I),
        ("alpha", _F), ("beta", _F), ("diag", _F), ("pad_", _I),
        ("alpha_vec", _LL), ("C", _LL), ("D", _LL), ("partials", _LL),
        ("ldc", _LL), ("ldd", _LL), ("strideC", _LL), ("strideD", _LL),
    ]


class _Final(ctypes.Structure):
    _fields_ = [
        ("C", _VP), ("D", _VP), ("C_tab", _VP), ("D_tab", _VP), ("D2_tab", _VP), ("alpha_vec", _VP),
        ("ldc", _LL), ("ldd", _LL), ("ldd2", _LL), ("strideC", _LL), ("strideD", _LL),
        ("alpha", _F), ("beta", _F), ("out_kind", _I), ("pad_", _I),
    ]


class _Map(ctypes.Structure):
    _fields_ = [
        ("base", _VP), ("rows", _LL), ("cols", _LL), ("batch", _LL), ("ld", _LL), ("batch_stride", _LL),
        ("fp16", _I), ("box_cols", _I), ("box_rows", _I), ("pad_", _I),
    ]


class _Args(ctypes.Structure):
    _fields_ = [
        ("ops", _VP), ("maps", _VP), ("tab", _VP), ("counters", _VP), ("work", _VP), ("status", _VP),
        ("n_ops", _I), ("n_maps", _I), ("total", _I), ("n_counters", _I), ("n_final", _I),
        ("bn", _I), ("wide", _I),
        ("fin", _Final * MAX_GROUPS),
    ]


@lru_cache(maxsize=None)
def _lib():
    lib = _build.load()
    lib.dmuon_chain_encode_maps.argtypes = [ctypes.POINTER(_Map), _I, _VP]
    lib.dmuon_chain_encode_maps.restype = _I
    lib.dmuon_chain_launch.argtypes = [ctypes.POINTER(_Args), _VP]
    lib.dmuon_chain_launch.restype = _I
    return lib


def fp16_prescale(m0: int, n0: int) -> float:
    return float(2 ** round(math.log2(math.sqrt(min(m0, n0)))))


# ---------------------------------------------------------------------------- the products of one group
@dataclass
class Product:
    """``out = alpha * A B^T + beta * C + diag * I`` on named buffers of a group."""

    A: str
    B: str
    out: str                        # "final": the caller's output
    a_mn: bool = False
    b_mn: bool = False
    C: Optional[str] = None
    alpha: float = 1.0
    beta: float = 0.0
    diag: float = 0.0
    vec: Optional[str] = None       # per-matrix factor: "vec" or "vec2"
    symmetric: bool = False
    after: int = -1                 # index of the last product that has to be finished first (-1: none)


def iteration_products(left: bool, coefs, restarts, formulation: str, h: float, with_vec: bool) -> list[Product]:
    """The products of the iteration in issue order (the recurrences of
    :mod:`dmuon_b200.optim.newton_schulz`); ``h`` is the host factor between the
    stored operand and the normalised matrix, ``with_vec`` adds the per-matrix one."""
    out: list[Product] = []

    def add(**kw) -> int:
        out.append(Product(**kw))
        return len(out) - 1

    def gram(X: str, dst: str, after: int) -> int:
        return add(A=X, B=X, out=dst, a_mn=not left, b_mn=not left, alpha=h * h, vec="vec2" if with_vec else None,
                   symmetric=True, after=after)

    def apply(Q: str, X: str, dst: str, after: int, **kw) -> int:
        if left:
            return add(A=Q, B=X, out=dst, b_mn=True, after=after, **kw)
        return add(A=X, B=Q, out=dst, after=after, **kw)

    X, Xn = "X", "X2"
    last = len(coefs) - 1
    if formulation == "direct":
        done = -1
        for i, (a, b, c) in enumerate(coefs):
            done = gram(X, "R", done)
            done = add(A="R", B="R", out="P", C="R", alpha=c, beta=b, symmetric=True, after=done)
            done = apply("P", X, "final" if i == last else Xn, done, C=X, beta=a)
            X, Xn = Xn, X
        return out

    done = gram(X, "R", -1)
    R, Rn = "R", "R2"
    pool = ("Qa", "Qb", "P")
    Q: Optional[str] = None
    for i, (a, b, c) in enumerate(coefs):
        if i in restarts and i != 0:
            done = apply(Q, X, Xn, done)
            X, Xn = Xn, X
            done = gram(X, R, done)
            Q = None
        P = next(t for t in pool if t != Q)
        done = add(A=R, B=R, out=P, C=R, alpha=c, beta=b, diag=a, symmetric=True, after=done)
        more = i < last and (i + 1) not in restarts
        after_p = done
        if Q is None:
            Q = P
        else:
            T = next(t for t in pool if t not in (Q, P))
            done = add(A=P, B=Q, out=T, symmetric=True, after=after_p)
            Q = T
        if more:
            # needs only P: runs beside the product above
            done = add(A=R, B=P, out="RP", symmetric=True, after=after_p)
            done = add(A="RP", B=P, out=Rn, symmetric=True, after=done)
            R, Rn = Rn, R
    apply(Q, X, "final", done, alpha=h, vec="vec" if with_vec else None)
    return out


# ---------------------------------------------------------------------------- groups and plans
@dataclass(frozen=True)
class GroupSpec:
    L: int
    m0: int
    n0: int
    dtype: torch.dtype
    formulation: str
    coefs: tuple
    restarts: tuple
    h: float
    with_vec: bool

    def __hash__(self) -> int:
        # a key of every call: the nested coefficients are hashed once
        h = self.__dict__.get("_hash")
        if h is None:
            h = hash((self.L, self.m0, self.n0, self.dtype, self.formulation, self.coefs, self.restarts, self.h,
                      self.with_vec))
            object.__setattr__(self, "_hash", h)
        return h

    @property
    def left(self) -> bool:
        return self.m0 <= self.n0

    @property
    def m(self) -> int:
        return min(self.m0, self.n0)

    @property
    def n(self) -> int:
        return max(self.m0, self.n0)


@lru_cache(maxsize=4096)
def _products_of(spec: GroupSpec) -> tuple[Product, ...]:
    return tuple(iteration_products(spec.left, spec.coefs, spec.restarts, spec.formulation, spec.h, spec.with_vec))


def tile_rows(bn: int) -> int:
    return 256 if bn == PAIR else G.BM


def _tiles(m: int, n: int, bn: int, symmetric: bool) -> np.ndarray:
    """[T, 3] of (row tile, column tile, mirror)."""
    bm = tile_rows(bn)
    t = G.symmetric_tiles(m, bn, bm) if symmetric else G.dense_tiles(m, n, bn, bm)
    return np.asarray(t, dtype=np.int64).reshape(-1, 3)


@lru_cache(maxsize=4096)
def sym_tile_count(m: int, bn: int) -> int:
    return len(G.symmetric_tiles(m, bn, tile_rows(bn)))


def sym_tiles(specs: Sequence[GroupSpec], bn: int) -> int:
    """Tiles of one symmetric product of every group."""
    return sum(s.L * sym_tile_count(s.m, bn) for s in specs)


def _operands(pr: Product, bn: int) -> tuple:
    """The tensor maps of a product's A and B: (buffer, columns and rows of the box)."""
    return tuple((name, (64, _KB) if mn else (_KB, rows))
                 for name, mn, rows in ((pr.A, pr.a_mn, G.BM), (pr.B, pr.b_mn, min(bn, G.BM))))


@lru_cache(maxsize=4096)
def _map_count(spec: GroupSpec, bn: int) -> int:
    return len({m for pr in _products_of(spec) for m in _operands(pr, bn)})


def fits(specs: Sequence[GroupSpec]) -> bool:
    """Within what a plan's tables can express, matrices the kernels take."""
    if len(specs) > MAX_GROUPS or sum(s.L for s in specs) > MAX_MATRICES:
        return False
    if any(s.L < 1 or s.m0 % 8 or s.n0 % 8 or s.m < 8 or not s.coefs for s in specs):
        return False
    bn = choose_bn(specs)
    if sum(_map_count(s, bn) for s in specs) > MAX_MAPS:
        return False
    # a Gram product that is split over K counts twice
    split = bn != PAIR
    return sum(len(p) + split * sum(q.symmetric and q.A in ("X", "X2") for q in p) for p in map(_products_of, specs)) <= MAX_OPS


#: tile width -> (CTAs or pairs that work at once; microseconds per k-block of a tile when few of them work; when
#: all do; microseconds from the first load of a product to the first load of the next beyond its k-blocks)
_COST = {64: (SMS, 0.31, 0.40, 4.2), 128: (SMS, 0.41, 0.52, 5.0), PAIR: (PAIRS, 0.42, 0.46, 7.0)}


def estimate_us(specs: Sequence[GroupSpec], bn: int) -> float:
    """Time of a chain with this tile width: product by product, the k-blocks of its longest
    round plus the way from one product to the next.  An SM is fed about 80 bytes per
    nanosecond, so a k-block costs what its operands weigh (24, 32 and 32 KB per SM here), a
    little more when all SMs pull.  Measured / estimated on a B200: 256 x 256 97 / 98, 1024 x
    1024 in 64-wide tiles 222 / 180, 1536 x 1536 in 128-wide ones 278 / 295, 4096 x 4096 on
    pairs 1301 / 1304, 4096 x 14336 2114 / 2128."""
    units, alone, busy, step = _COST[bn]
    tiles_all = sym_tiles(specs, bn)
    matrices = sum(s.L for s in specs)
    per_group = [_products_of(s) for s in specs]
    total = 0.0
    for i in range(max(len(p) for p in per_group)):
        tiles = work = longest = 0
        total += step
        for s, products in zip(specs, per_group):
            if i >= len(products):
                continue
            pr = products[i]
            is_gram = pr.symmetric and pr.A in ("X", "X2")
            splits, per = gram_splits(s, bn, tiles_all) if is_gram else (1, 0)
            kb = per if splits > 1 else -(-(s.n if is_gram else s.m) // _KB)
            if splits > 1:
                total += step
            n = splits * s.L * (sym_tile_count(s.m, bn) if pr.symmetric else
                                -(-s.m0 // tile_rows(bn)) * -(-s.n0 // bn))
            tiles, work, longest = tiles + n, work + n * kb, max(longest, kb)
        # one or two matrices: whole rounds; more: tiles of other matrices fill the last one
        rounds = max(longest, work / units) if matrices > 2 else -(-tiles // units) * longest
        total += rounds * (alone + (busy - alone) * min(1.0, tiles / units))
    return total


@lru_cache(maxsize=4096)
def _best_bn(specs: tuple) -> int:
    return min(_COST, key=lambda bn: estimate_us(specs, bn))


def choose_bn(specs: Sequence[GroupSpec]) -> int:
    """The tile width with the lowest estimate.  64-wide tiles where products are small (more
    SMs with less each), CTA pairs where they fill the GPU or are long."""
    return _best_bn(tuple(specs))


def choose_wide(specs: Sequence[GroupSpec], bn: int) -> bool:
    """Two tiles side by side per entry?  Only in lists with several rounds of tiles in every
    product: an entry takes twice as long, so the last round of a product costs twice as much.
    Measured (ms, single / two): four 14336 x 4096 (544 tiles a symmetric product) 9.89 / 8.91,
    eight 4096 x 4096 (1088) 10.24 / 10.11, four 3072 x 8192 (312) 3.44 / 3.57, one
    4096 x 14336 (136) 2.39 / 2.49."""
    return bn == PAIR and sym_tiles(specs, PAIR) >= 3 * SMS


def gram_splits(spec: GroupSpec, bn: int, tiles_all: int) -> tuple[int, int]:
    """(splits, k-blocks per split) of the Gram product: as many splits as keep
    the SMs busy, each with at least eight k-blocks to amortise its partial tile.
    CTA pairs are taken only where there are tiles enough."""
    num_kb = -(-spec.n // _KB)
    splits = 1 if bn == PAIR else max(1, min(SMS // max(1, tiles_all), num_kb // 8, 16))
    per = -(-num_kb // splits)
    return -(-num_kb // per), per


def _up(n: int) -> int:
    return -(-n // 1024) * 1024


#: matrices of a plan; their counters and sums of squares stand at the head of the work memory
MAX_MATRICES = 4096
CONTROL_BYTES = _up(4 * (2 + 2 * MAX_MATRICES))


class Arena:
    """Work memory of one stream.  Plans of a stream use it one after the other (the
    operands are written, the chain runs, the result leaves), so they share it; the
    lock spans those steps on the host.

    At its head lie ticket, exits, one counter per matrix and the sums of squares of the
    plan that runs: all zero between calls, the kernel clears them itself."""

    def __init__(self, nbytes: int, device):
        self.lock = threading.RLock()
        self.buf = torch.empty(nbytes, dtype=torch.uint8, device=device)
        self.control = self.buf[:CONTROL_BYTES].view(torch.int32)
        self.control.zero_()
        self.dirty = False          # a call was abandoned half-way: the head has to be cleared

    def at(self, offset: int, shape, dtype) -> torch.Tensor:
        n = math.prod(shape) * torch.empty(0, dtype=dtype).element_size()
        return self.buf[offset : offset + n].view(dtype).view(shape)


def _buffer_shapes(spec: GroupSpec, splits: int) -> dict:
    L, m = spec.L, spec.m
    names = ("R", "P") if spec.formulation == "direct" else ("R", "R2", "RP", "P", "Qa", "Qb")
    out = {b: ((L, m, m), spec.dtype) for b in names}
    out["X"] = out["X2"] = ((L, spec.m0, spec.n0), spec.dtype)
    if splits > 1:
        out["partials"] = ((L * splits, m, m), torch.float32)
    return out


def _layout(specs: Sequence[GroupSpec], bn: int) -> tuple[list[dict], tuple, int]:
    """Where everything lies in the work memory: per group ``{buffer: (offset, shape,
    dtype)}``, the offsets of three words per matrix (two factors, a flag), and the bytes in all."""
    tiles = sym_tiles(specs, bn)
    n = sum(s.L for s in specs)
    vec = CONTROL_BYTES
    vec2 = vec + _up(4 * n)
    again = vec2 + _up(4 * n)
    at = again + _up(4 * n)
    groups = []
    for s in specs:
        group = {}
        for name, (shape, dtype) in _buffer_shapes(s, gram_splits(s, bn, tiles)[0]).items():
            group[name] = (at, shape, dtype)
            at += _up(math.prod(shape) * (4 if dtype == torch.float32 else 2))
        groups.append(group)
    return groups, (vec, vec2, again), at


def plan_bytes(specs: Sequence[GroupSpec]) -> int:
    return _layout(specs, choose_bn(specs))[2]


def _two_wide(e: np.ndarray) -> np.ndarray:
    """Entries of 256 x 256 tiles joined into pairs that lie side by side (they share
    their A rows, see the kernel): bit 9 = there is a second half, bit 10 = its mirror
    flag.  What is left of a last round of single tiles stays single, at the end: a
    round of wide tiles takes twice as long."""
    left = len(e) % SMS
    wide = len(e) - (left if left <= PAIRS else 0)
    if wide == 0:
        return e
    row = (e[:wide, 0] & 0xFF) | ((e[:wide, 1] & 0xFFFF) << 8) | (e[:wide, 2] << 24)     # product, row of tiles, matrix
    col = e[:wide, 1] >> 16
    order = np.lexsort((col, row))
    r, c = row[order], col[order]
    at = np.arange(wide)
    starts = np.r_[True, (r[1:] != r[:-1]) | (c[1:] != c[:-1] + 1)]              # runs of neighbours
    inside = at - np.maximum.accumulate(np.where(starts, at, 0))
    last = np.r_[starts[1:], True]
    first = (inside % 2 == 0) & ~last
    second = np.r_[False, first[:-1]]
    joined = e[order[first]].copy()
    joined[:, 0] |= (1 << 9) | (((e[order[second], 0] >> 8) & 1) << 10)
    joined = joined[np.argsort(order[first], kind="stable")]                     # the list's own order: L2 locality
    single = np.sort(np.r_[order[~first & ~second], np.arange(wide, len(e))])
    return np.concatenate([joined, e[single]])


def build_entries(specs: Sequence[GroupSpec], bn: int):
    """Products and tile list of a plan, without touching a device.

    Returns ``(ops, entries)``: ``ops`` are ``(group, Product, splits, kb_per_split, is_sum)``
    and ``entries`` is an int32 array ``[T, 4]`` in the kernel's packing."""
    per_group = [_products_of(s) for s in specs]
    tiles_all = sym_tiles(specs, bn)
    splits = [gram_splits(s, bn, tiles_all) for s in specs]
    first_matrix = np.cumsum([0] + [s.L for s in specs])
    ops: list = []
    chunks: list[np.ndarray] = []
    # finished warps of one matrix of group g after product i (all tiles of products 0..i)
    total = [0] * len(specs)
    upto: list[list[int]] = [[] for _ in specs]

    def emit(g: int, op: int, tiles: np.ndarray, want: int, split: int = 0) -> None:
        L = specs[g].L
        b = np.repeat(np.arange(L), len(tiles))
        t = np.tile(tiles, (L, 1))
        e = np.empty((len(b), 4), dtype=np.int64)
        e[:, 0] = op | (t[:, 2] << 8) | (split << 16)
        e[:, 1] = t[:, 0] | (t[:, 1] << 16)
        e[:, 2] = b | ((first_matrix[g] + b) << 16)
        e[:, 3] = want
        level.append(e)
        total[g] += len(tiles) * WARPS_PER_TILE * (2 if bn == PAIR else 1)

    wide = choose_wide(specs, bn)
    for i in range(max(len(p) for p in per_group)):
        level: list[np.ndarray] = []
        for g, s in enumerate(specs):
            if i >= len(per_group[g]):
                continue
            pr = per_group[g][i]
            want = upto[g][pr.after] if pr.after >= 0 else 0
            is_gram = pr.symmetric and pr.A == pr.B and pr.A in ("X", "X2")
            ns, per = splits[g] if is_gram else (1, 0)
            rows = s.m if pr.symmetric else s.m0
            cols = s.m if pr.symmetric else s.n0
            tiles = _tiles(rows, cols, bn, pr.symmetric)
            if ns > 1:
                plain = tiles.copy()
                plain[:, 2] = 0
                ops.append((g, pr, ns, per, False))
                for k in range(ns):
                    emit(g, len(ops) - 1, plain, want, k)
                ops.append((g, pr, ns, 0, True))
                emit(g, len(ops) - 1, _tiles(rows, cols, _SUM_COLS, True), total[g])
            else:
                ops.append((g, pr, 1, 0, False))
                emit(g, len(ops) - 1, tiles, want)
            upto[g].append(total[g])
        entries = np.concatenate(level)
        chunks.append(_two_wide(entries) if wide else entries)
    entries = np.concatenate(chunks) if chunks else np.zeros((0, 4), dtype=np.int64)
    # the packing holds 31 bits per word; the sign bit of the first word marks the end of the list
    return ops, (entries & 0xFFFFFFFF).astype(np.uint32).view(np.int32)


class Program:
    """What a plan knows before it has work memory: the operations (with offsets into that
    memory), the tile list and the operands' tensor maps.  The lists lie on the device in
    one piece and serve every stream."""

    def __init__(self, specs: Sequence[GroupSpec], device: torch.device):
        self.specs = tuple(specs)
        self.device = device
        self.captured = False       # a CUDA graph names the lists
        self.bn = choose_bn(self.specs)
        self.wide = choose_wide(self.specs, self.bn)
        self.groups, (self.vec, self.vec2, self.again), self.nbytes = _layout(self.specs, self.bn)
        self.n_matrices = sum(s.L for s in self.specs)
        assert self.n_matrices <= MAX_MATRICES
        self.first = [0]
        for s in self.specs:
            self.first.append(self.first[-1] + s.L)
        ops, entries = build_entries(self.specs, self.bn)
        assert len(ops) <= MAX_OPS
        self.n_ops, self.total = len(ops), int(entries.shape[0])
        self.maps: list[tuple] = []          # (group, buffer, box)
        self.finals = {g: pr for g, pr, *_ in ops if pr.out == "final"}
        # the power of two that keeps fp16 operands clear of the subnormals, per matrix
        k = np.repeat([fp16_prescale(s.m0, s.n0) for s in self.specs], [s.L for s in self.specs]).astype(np.float32)
        parts = [np.frombuffer(bytes(self._operations(ops)), dtype=np.uint8), entries.view(np.uint8).reshape(-1),
                 k.view(np.uint8)]
        at = np.cumsum([0] + [_up(len(x)) for x in parts])
        host = np.zeros(at[-1], dtype=np.uint8)
        for lo, x in zip(at, parts):
            host[lo : lo + len(x)] = x
        self.lists = torch.from_numpy(host).to(device)
        self.ops_at, self.tab_at = (self.lists.data_ptr() + int(lo) for lo in at[:2])
        self.k = self.lists[at[2] : at[2] + len(parts[2])].view(torch.float32)

    def _operations(self, ops):
        index: dict[tuple, int] = {}

        def map_of(key: tuple) -> int:
            if key not in index:
                index[key] = len(self.maps)
                self.maps.append(key)
            return index[key]

        arr = (_Op * len(ops))()
        for i, (g, pr, ns, per, is_sum) in enumerate(ops):
            s, bufs = self.specs[g], self.groups[g]
            o = arr[i]
            o.M = s.m if pr.symmetric else s.m0
            o.N = s.m if pr.symmetric else s.n0
            o.K = s.n if (pr.symmetric and pr.A in ("X", "X2")) else s.m
            o.a_mn_major, o.b_mn_major = int(pr.a_mn), int(pr.b_mn)
            o.ab_fp16 = int(s.dtype == torch.float16)
            o.final_slot, o.splits, o.kb_per_split = -1, ns, per
            o.map_a, o.map_b = (-1, -1) if is_sum else (map_of((g, *x)) for x in _operands(pr, self.bn))
            o.alpha_vec = o.C = o.D = o.partials = -1
            if ns > 1 and not is_sum:
                o.alpha, o.out_kind = 1.0, 2
                o.D, o.ldd, o.strideD = bufs["partials"][0], s.m, s.m * s.m
                continue
            o.alpha, o.beta, o.diag = pr.alpha, pr.beta, pr.diag
            o.out_kind = G._OUT_KIND[s.dtype]
            if pr.vec is not None:
                o.alpha_vec = (self.vec if pr.vec == "vec" else self.vec2) + 4 * self.first[g]
            if is_sum:
                o.partials = bufs["partials"][0]
            if pr.C is not None:
                o.C, (_, rows, o.ldc), _ = bufs[pr.C]
                o.strideC = rows * o.ldc
            if pr.out == "final":
                o.final_slot = g
            else:
                o.D, (_, rows, o.ldd), _ = bufs[pr.out]
                o.strideD = rows * o.ldd
        return arr

    def encode(self, base: int):
        """The tensor maps over the work memory at ``base``: (their owner, their address)."""
        n = len(self.maps)
        marr = (_Map * n)()
        for m, (g, name, box) in zip(marr, self.maps):
            offset, (L, r, c), dtype = self.groups[g][name]
            m.base, m.rows, m.cols, m.batch, m.ld, m.batch_stride = base + offset, r, c, L, c, r * c
            m.fp16, m.box_cols, m.box_rows = int(dtype == torch.float16), box[0], box[1]
        raw = ctypes.create_string_buffer(128 * n + 64)
        at = (ctypes.addressof(raw) + 63) & ~63      # tensor maps are aligned to 64 bytes
        rc = _lib().dmuon_chain_encode_maps(marr, n, at)
        if rc != 0:
            raise RuntimeError(f"dmuon_chain_encode_maps failed with code {rc}")
        return raw, at


class Plan:
    """A program and its work memory."""

    def __init__(self, program: Program, arena: Arena):
        self.program, self.arena, self.lock = program, arena, arena.lock
        self.specs, self.device, self.n_matrices, self.k = program.specs, program.device, program.n_matrices, program.k
        n = self.n_matrices
        self.sumsq = arena.control[2 + n : 2 + 2 * n].view(torch.float32)
        self.vec = arena.at(program.vec, (n,), torch.float32)
        self.vec2 = arena.at(program.vec2, (n,), torch.float32)
        self.again = arena.at(program.again, (n,), torch.int32)
        # per group: the operands, their sums of squares and flags
        bounds = list(zip(program.first, program.first[1:]))
        self.X = [list(arena.at(*g["X"])) for g in program.groups]
        self.group_sumsq = [self.sumsq[lo:hi] for lo, hi in bounds]
        self.group_again = [self.again[lo:hi] for lo, hi in bounds]
        base = arena.buf.data_ptr()
        self._maps, maps_at = program.encode(base)
        a = _Args()
        a.ops, a.maps, a.tab = program.ops_at, maps_at, program.tab_at
        a.counters, a.work, a.status = base, base, G.status_buffer(self.device).data_ptr()
        a.n_ops, a.n_maps, a.total = program.n_ops, len(program.maps), program.total
        a.n_counters, a.n_final, a.bn, a.wide = 2 + 2 * n, len(self.specs), program.bn, int(program.wide)
        self._args = a

    def begin(self) -> None:
        """Call before the sums of squares are accumulated."""
        if self.arena.dirty:
            self.arena.control.zero_()
        self.arena.dirty = True

    def run(self, finals: Sequence[dict]) -> None:
        """Launch the chain on the current stream.  ``finals[g]``: ``out`` (a
        ``[L, m0, n0]`` tensor) or ``out_tab`` / ``c_tab`` / ``out2_tab`` (device tables
        of addresses, multiples of 16 bytes) with ``out_dtype``; ``alpha`` multiplies the plan's own factor."""
        a, program = self._args, self.program
        for g, f in enumerate(finals):
            s, pr, fin = self.specs[g], program.finals[g], a.fin[g]
            fin.alpha = float(f.get("alpha", 1.0)) * pr.alpha
            fin.alpha_vec = self.vec.data_ptr() + 4 * program.first[g] if pr.vec is not None else None
            fin.C = fin.C_tab = fin.D = fin.D_tab = fin.D2_tab = None
            fin.ldc = fin.ldd = fin.ldd2 = s.n0
            fin.strideC = fin.strideD = s.m0 * s.n0
            fin.beta = 0.0
            out = f.get("out")
            if out is not None:
                fin.D, fin.out_kind = out.data_ptr(), G._OUT_KIND[out.dtype]
                if pr.C is not None:
                    assert out.dtype == s.dtype
                    fin.C, fin.beta = self.arena.buf.data_ptr() + program.groups[g][pr.C][0], pr.beta
                continue
            assert pr.C is None
            fin.D_tab, fin.out_kind = f["out_tab"].data_ptr(), G._OUT_KIND[f["out_dtype"]]
            if f.get("c_tab") is not None:
                fin.C_tab, fin.beta = f["c_tab"].data_ptr(), float(f["beta"])
            if f.get("out2_tab") is not None:
                fin.D2_tab = f["out2_tab"].data_ptr()
        stream = ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(self.device.index))
        rc = _lib().dmuon_chain_launch(ctypes.byref(a), stream)
        if rc != 0:
            raise RuntimeError(f"dmuon_chain_launch failed with code {rc}")
        self.arena.dirty = False


# ---------------------------------------------------------------------------- plans that are kept
#: what the buffers of one plan may take together (the largest batch of a Muon step fills it to the byte for powers of
#: two), and with what stands at the head of the work memory
MAX_BUFFER_BYTES = 6 << 30
MAX_PLAN_BYTES = MAX_BUFFER_BYTES + CONTROL_BYTES + 3 * _up(4 * MAX_MATRICES)
MAX_PLANS = 256
MAX_ARENAS = 8
#: and those of all streams: two of the largest
MAX_ARENA_BYTES = 2 * MAX_PLAN_BYTES + (1 << 20)
_programs: "OrderedDict[tuple, Program]" = OrderedDict()
_plans: "OrderedDict[tuple, Plan]" = OrderedDict()
_arenas: "OrderedDict[tuple, Arena]" = OrderedDict()
_lock = threading.RLock()


@lru_cache(maxsize=4096)
def possible(specs: tuple[GroupSpec, ...]) -> bool:
    """These groups can be one plan."""
    return fits(specs) and plan_bytes(specs) <= MAX_PLAN_BYTES


def _program_for(sig: tuple) -> Program:
    p = _programs.get(sig)
    if p is None:
        if len(_programs) >= MAX_PLANS:
            _programs.pop(next((k for k, q in _programs.items() if not q.captured), None), None)
        p = _programs[sig] = Program(*sig)
    _programs.move_to_end(sig)
    return p


def _arena_for(where: tuple, nbytes: int, device: torch.device) -> Arena:
    arena = _arenas.get(where)
    if arena is None or arena.buf.numel() < nbytes:
        # plans on the smaller memory go: only their work memory's addresses are lost, the programs stay
        _drop(lambda k: k[1] == where)
        _arenas.pop(where, None)
        arena = None
        arena = _arenas[where] = Arena(nbytes, device)
    _arenas.move_to_end(where)
    while len(_arenas) > MAX_ARENAS or (len(_arenas) > 1 and
                                        sum(a.buf.numel() for a in _arenas.values()) > MAX_ARENA_BYTES):
        old, _ = _arenas.popitem(last=False)
        _drop(lambda k: k[1] == old)
    return arena


def plan_for(specs: Sequence[GroupSpec], device: torch.device) -> Optional[Plan]:
    """The plan of these groups for the current stream: work memory is never shared
    between streams, nor between a captured call and any other.

    While a CUDA graph is captured, the work memory is allocated like every other
    temporary of the captured call: it belongs to the graph, whatever stream replays it,
    and the head is cleared by the graph itself.  The program is one that an earlier call
    made (nothing can be uploaded now; ``None`` if there is none) and is kept for good,
    because the graph names its lists: 16 bytes a tile, far less than the work memory that
    the graph itself holds."""
    sig = (tuple(specs), device)
    if torch.cuda.is_current_stream_capturing():
        with _lock:
            program = _programs.get(sig)
            if program is None:
                return None
            program.captured = True
        return Plan(program, Arena(program.nbytes, device))
    where = (device.index, torch._C._cuda_getCurrentRawStream(device.index))
    key = (sig, where)
    with _lock:
        p = _plans.get(key)
        if p is None:
            program = _program_for(sig)
            # freed only when this stream has finished with them
            program.lists.record_stream(torch.cuda.current_stream(device))
            p = Plan(program, _arena_for(where, program.nbytes, device))
            if len(_plans) >= MAX_PLANS:
                _plans.popitem(last=False)
            _plans[key] = p
        _plans.move_to_end(key)
        return p


def _drop(which) -> None:
    for k in [k for k in _plans if which(k)]:
        del _plans[k]


def release() -> None:
    with _lock:
        for k in [k for k, p in _programs.items() if not p.captured]:
            del _programs[k]
        _plans.clear()
        _arenas.clear()
