"""Host side of the htree operator: the reference's Python entry points over the C ABI of libhtree_b200.

Same names, keyword arguments, tensor layouts and return values as the reference (skywong14/htree):
    htree_forward                  src/parallel.py:874-1159
    htree_backward                 src/backward.py:941-1119
    HTreeTritonFunction            src/backward.py:1126-1193   (alias of HTreeFunction here)
    htree_forward_triton_autograd  src/backward.py:1196-1208
    LayerTrace                     src/naive.py:13-19
PyTorch supplies device memory and the current stream only; all arithmetic runs in the CUDA library.  There is no
CPU path: tensors must live on a CUDA device and the library must have been built.

Differences from the reference that callers can rely on:
  * `max_top_nodes` may be smaller than `top_k_per_layer * compression_rate` (the reference asserts equality).  The
    additional top levels then hold at most top_k nodes, every candidate is kept and nothing is accumulated there, so
    the result equals the reference called with max_top_nodes = top_k_per_layer * compression_rate.
  * sizes need not be powers of two, and top_k_per_layer need not be a multiple of 64 or of compression_rate.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Dict, List, Optional, Tuple

import torch

from . import _lib

HTREE_SCORE_NEG_INF: float = -1.0e10                                  # src/parallel.py:75
HTREE_SCORE_VALID_THRESHOLD: float = HTREE_SCORE_NEG_INF * 0.9         # src/parallel.py:81

_DTYPES = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}

# Keep the per-level selections from the forward for the backward of the autograd function (True), or rebuild them
# in the backward with the selection-only pass like the reference does (False; saves L*B*T*H_kv*top_k*4 bytes).
SAVE_SELECTIONS_FOR_BACKWARD = True

# Storage of the per-level selections (bwd_ctx["per_layer_parents"]): "int32" is the reference's layout
# (src/parallel.py:1044, -1 = none); "uint16" halves that memory (torch.int16 tensors holding the unsigned bit
# pattern, 0xFFFF = none; decode_parents() converts) and needs every pooled level to have at most 65535 nodes.
SELECTION_STORAGE = "int32"

# Largest temporary the forward may allocate for handing selections from its selection kernel to its accumulation
# kernel when the caller does not keep them (see htree_forward); above it the queries run window by window.
SPLIT_FORWARD_MAX_BYTES = 4 << 30


# Scratch of the two-pass backward (htree_b200_run_backward): P and dS of the queries of one launch.  Larger means fewer
# launches; a shape that does not fit at all takes the one-pass backward, which needs none.
BACKWARD_MAX_BYTES = 4 << 30


def _parents_dtype(layers_k, top_k: int):
    if SELECTION_STORAGE == "int32":
        return torch.int32
    if SELECTION_STORAGE != "uint16":
        raise ValueError(f"SELECTION_STORAGE must be 'int32' or 'uint16', not {SELECTION_STORAGE!r}")
    if top_k > 65535 or any(x.shape[1] > 65535 for x in layers_k[1:]):
        raise ValueError("SELECTION_STORAGE='uint16' needs pooled levels of at most 65535 nodes")
    return torch.int16


def _parents_flag(parents) -> int:
    first = parents[0] if parents is not None else None
    return _lib.PARENTS_U16 if first is not None and first.dtype == torch.int16 else 0


def decode_parents(t: torch.Tensor) -> torch.Tensor:
    """Selections in the reference's layout (int32, -1 = none) from either storage format."""
    if t.dtype == torch.int32:
        return t
    x = t.to(torch.int32) & 0xFFFF
    return torch.where(x == 0xFFFF, torch.full_like(x, -1), x)


@dataclass
class LayerTrace:
    layer_idx: int
    selected_parents: Optional[torch.Tensor]
    layer_max: torch.Tensor
    layer_sum: torch.Tensor
    layer_output: torch.Tensor


_rope_tables: Dict[Tuple, Tuple[torch.Tensor, torch.Tensor]] = {}
_status_words: Dict[torch.device, torch.Tensor] = {}


def rope_cache(k_dim: int, cache_size: int, rope_base: float, device) -> Tuple[torch.Tensor, torch.Tensor]:
    """cos/sin tables [cache_size, k_dim/2] fp32 (src/parallel.py:983-988), built once per configuration.

    The tables are evaluated with torch's CPU float32 kernels and copied to the device: the angle pos*inv_freq is
    rounded to float32 before the cosine, so results only match the reference's CPU oracle bit for bit when
    inv_freq comes out of the same pow implementation."""
    key = (int(k_dim), int(cache_size), float(rope_base), torch.device(device))
    hit = _rope_tables.get(key)
    if hit is None:
        inv_freq = 1.0 / (rope_base ** (torch.arange(0, k_dim, 2, dtype=torch.float32) / k_dim))
        freqs = torch.outer(torch.arange(cache_size, dtype=torch.float32), inv_freq)
        hit = (freqs.cos().to(device).contiguous(), freqs.sin().to(device).contiguous())
        _rope_tables[key] = hit
    return hit


_rope_half: Dict[Tuple, Tuple[torch.Tensor, torch.Tensor]] = {}


def rope_cache_half(k_dim: int, cache_size: int, rope_base: float, scale: float, device):
    """cos*scale and sin*scale as float16 tables (same shape as rope_cache), for the packed-half query rotation of the
    tensor-core kernels in the passes that do not decide the Top-K."""
    key = (int(k_dim), int(cache_size), float(rope_base), float(scale), torch.device(device))
    hit = _rope_half.get(key)
    if hit is None:
        c, s = rope_cache(k_dim, cache_size, rope_base, device)
        hit = ((c * float(scale)).to(torch.float16).contiguous(), (s * float(scale)).to(torch.float16).contiguous())
        _rope_half[key] = hit
    return hit


_rope_rows: Dict[Tuple, torch.Tensor] = {}


def rope_rows(k_dim: int, cache_size: int, rope_base: float, scale: Optional[float], device) -> torch.Tensor:
    """The rotary table of the transposed tensor-core kernels: rows [cos | sin] of width k_dim, float16 multiplied by
    `scale`, or plain fp32 when scale is None (split-half kernels)."""
    key = (k_dim, cache_size, rope_base, scale, device)
    hit = _rope_rows.get(key)
    if hit is None:
        c, s = rope_cache(k_dim, cache_size, rope_base, device)
        if scale is None:
            hit = torch.cat([c, s], dim=1).contiguous()
        else:
            hit = torch.cat([(c * float(scale)).to(torch.float16), (s * float(scale)).to(torch.float16)], dim=1).contiguous()
        _rope_rows[key] = hit
    return hit


def rope_rows_select(k_dim: int, cache_size: int, rope_base: float, device) -> torch.Tensor:
    """The rotary table of the selection kernel: fp32 rows [cos | sin | -sin], each part ordered [k-step pair][r][4] over the pairs
    (k_dim/8)*r + 4*(k-step pair) + {0..3} that lane r of a quad rotates.  (The format of the C interface; the third part is not read.)"""
    key = (k_dim, cache_size, rope_base, "select", device)
    hit = _rope_rows.get(key)
    if hit is None:
        c, s = rope_cache(k_dim, cache_size, rope_base, device)
        perm = torch.arange(k_dim // 2).view(4, -1, 4).transpose(0, 1).reshape(-1).to(device)
        hit = torch.cat([c[:, perm], s[:, perm], -s[:, perm]], dim=1).contiguous()
        _rope_rows[key] = hit
    return hit


def _status(device) -> torch.Tensor:
    device = torch.device(device)
    w = _status_words.get(device)
    if w is None:
        w = torch.zeros(1, dtype=torch.int32, device=device)
        _status_words[device] = w
    return w


def check_status(device=None) -> None:
    """Synchronise and raise if a kernel flagged a problem since the last check: an out-of-range node index (bits 0-3), or a
    bounded wait of the pipelined forward that ran out (bit 4)."""
    device = torch.device(device if device is not None else torch.cuda.current_device())
    if device.type == "cuda" and device.index is None:
        device = torch.device("cuda", torch.cuda.current_device())
    w = _status_words.get(device)
    if w is not None:
        v = int(w.item())
        if v:
            w.zero_()
            what = []
            if v & 0xF:
                what.append("a node index outside its tree level (clamped)")
            if v & 16:
                what.append("an asynchronous operand copy of the pipelined forward did not complete within its bounded wait "
                            "(the affected outputs were not written)")
            raise RuntimeError(f"htree_b200 kernels reported device-side status 0x{v:x}: " + "; ".join(what or ["unknown bits"]))


def _stream() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


class _on_device:
    """torch.cuda.device for the common case that the tensors' device is the current one (a tenth of its cost)."""

    __slots__ = ("index", "guard")

    def __init__(self, index: int):
        self.index, self.guard = index, None

    def __enter__(self):
        if torch._C._cuda_getDevice() != self.index:
            self.guard = torch.cuda.device(self.index)
            self.guard.__enter__()

    def __exit__(self, *exc):
        if self.guard is not None:
            self.guard.__exit__(*exc)


_table_sets: Dict[Tuple, Tuple] = {}


def _tables(k_dim: int, n_pos: int, rope_base: float, scale: float, split: bool, index: int):
    """(cos, sin, rows of the transposed kernels, rows of the selection kernel, status word) of one configuration and the
    addresses of the five: what a call would otherwise look up one by one."""
    key = (k_dim, n_pos, rope_base, scale, split, index)
    hit = _table_sets.get(key)
    if hit is None:
        dev = torch.device("cuda", index)
        ts = rope_cache(k_dim, n_pos, rope_base, dev) + (rope_rows(k_dim, n_pos, rope_base, None if split else scale, dev),
                                                         rope_rows_select(k_dim, n_pos, rope_base, dev), _status(dev))
        if len(_table_sets) >= 256:
            _table_sets.clear()
        hit = _table_sets[key] = ts + tuple(t.data_ptr() for t in ts)
    return hit


def _validate(q, k, v, compression_rate, max_top_nodes, top_k_per_layer, q_offset=None):
    if q.dim() != 4 or k.dim() != 4 or v.dim() != 4:
        raise ValueError("q/k/v must be rank-4 tensors")          # src/naive.py:141-142
    if not (q.is_cuda and k.is_cuda and v.is_cuda):
        raise RuntimeError("htree_b200 runs on CUDA tensors only; there is no CPU implementation")
    B, T_q, H, K = q.shape
    T = T_q if q_offset is None else k.shape[1]
    H_kv, V = k.shape[2], v.shape[-1]
    assert H % H_kv == 0, f"H ({H}) must be divisible by H_kv ({H_kv})"                      # src/parallel.py:912
    assert k.shape[2] == v.shape[2], "K and V must have same number of heads"                # src/parallel.py:914
    assert tuple(k.shape[:2]) == (B, T) and tuple(v.shape[:2]) == (B, T) and k.shape[3] == K  # src/naive.py:146
    if q_offset is not None:
        assert 0 <= q_offset and q_offset + T_q <= T, "query window must lie inside the key/value sequence"
    assert q.dtype == k.dtype == v.dtype and q.dtype in _DTYPES, "q, k, v must share one of fp32/bf16/fp16"
    assert max_top_nodes <= top_k_per_layer * compression_rate, (
        f"max_top_nodes ({max_top_nodes}) must not exceed top_k_per_layer*compression_rate "
        f"({top_k_per_layer}*{compression_rate})")                                            # cf. src/parallel.py:917-920
    return _lib.HtreeShape(B, T, H, H_kv, K, V, int(compression_rate), int(top_k_per_layer), int(max_top_nodes),
                           _DTYPES[q.dtype], 0 if q_offset is None else T_q, 0 if q_offset is None else int(q_offset))


def _ptrs(tensors) -> ctypes.Array:
    return _lib.ptr_array([t.data_ptr() if t is not None else None for t in tensors])


def build_tree(k: torch.Tensor, v: torch.Tensor, compression_rate: int, max_top_nodes: int,
               rope_base: Optional[float] = None):
    """Mean-pool tree (src/parallel.py:941-976).  Returns (layers_k, layers_v); level 0 are k and v themselves.

    With `rope_base` given, (layers_k, layers_v, layers_k_rot, layers_v_blk) is returned; the last two are the operand
    copies the tensor-core kernels read (None where no such kernel exists: fp32, or head sizes / compression rates they
    do not cover): the keys of every level rotated by their child index (node % compression_rate), float16 for bf16
    inputs too (one rounding of the rotated value, with half's finer significand), and the values of every level grouped
    per parent in the order the kernel's lanes consume them ([B, ceil(N/CR)*CR, H_kv, V], rows past N zero)."""
    k = k.contiguous(); v = v.contiguous()
    B, T, H_kv, K = k.shape
    V = v.shape[-1]
    sizes = _lib.level_sizes(T, compression_rate, max_top_nodes)
    layers_k, layers_v = [k], [v]
    for n in sizes[1:]:
        layers_k.append(torch.empty(B, n, H_kv, K, dtype=k.dtype, device=k.device))
        layers_v.append(torch.empty(B, n, H_kv, V, dtype=v.dtype, device=v.device))
    want_rot = rope_base is not None and _rotatable(k.dtype, K, V, compression_rate)
    layers_kr = [_rotated_like(x) for x in layers_k] if want_rot else None
    want_blk = want_rot and _blockable(V, compression_rate)
    layers_vb = [_blocked_like(x, compression_rate) for x in layers_v] if want_blk else None
    want_kblk = want_blk and _pipelined(k.dtype, K, compression_rate)
    layers_kb = [_blocked_like(x, compression_rate) for x in layers_kr] if want_kblk else None
    if len(sizes) > 1 or want_rot:
        shape = _lib.HtreeShape(B, T, H_kv, H_kv, K, V, int(compression_rate), 1, int(max_top_nodes),
                                _DTYPES[k.dtype])   # H and top_k play no role in the tree
        cos_c = sin_c = None
        if want_rot:
            cos_c, sin_c = rope_cache(K, max(int(compression_rate), 16), rope_base, k.device)
        with _on_device(k.get_device()):
            _lib.check(_lib.lib().htree_b200_build_tree(
                ctypes.byref(shape), _ptrs(layers_k), _ptrs(layers_v), _ptrs(layers_kr) if want_rot else None,
                _ptrs(layers_kb) if want_kblk else None, _ptrs(layers_vb) if want_blk else None,
                cos_c.data_ptr() if want_rot else None, sin_c.data_ptr() if want_rot else None, _stream()),
                "build_tree")
    if rope_base is not None:
        return layers_k, layers_v, layers_kr, OperandBlocks(layers_vb, layers_kb) if layers_vb is not None else None
    return layers_k, layers_v


class OperandBlocks(list):
    """Per-parent operand copies of every level.  As written by build_tree(rope_base=...) and block_values: the blocked values
    (the list itself) and the blocked keys (`.keys`, or None).  As written by build_operands and kept in a forward's context:
    the combined key/value blocks the transposed kernels read (the list itself, also `.keys` and `.blocks`) and, when a
    backward follows, its part (`.blocks_bwd`)."""

    def __init__(self, values, keys=None, blocks=None, blocks_bwd=None):
        super().__init__(values)
        self.keys = keys
        self.blocks = blocks
        self.blocks_bwd = blocks_bwd


def _transposed(dtype, K: int, V: int, G: int, compression_rate: int) -> bool:
    """Shapes with transposed tensor-core kernels (any storage type)."""
    return K == V and K in (32, 64, 128) and int(compression_rate) in (8, 16) and G <= 16


def _split(dtype, K: int) -> bool:
    """Operands carried as hi + lo half planes: fp32 storage, and 32-wide heads in every storage type."""
    return dtype == torch.float32 or K == 32


def _selects_on_tensor_cores(dtype, K: int) -> bool:
    return K == 64 or (K == 128 and dtype != torch.float32)


_plans: Dict[Tuple, Tuple] = {}


def _plan(shape: "_lib.HtreeShape", flags: int) -> "_lib.HtreePlan":
    """Workspace layout of a forward (htree_b200_plan), kept per shape."""
    key = (shape.B, shape.T, shape.H, shape.H_kv, shape.K, shape.compression_rate, shape.top_k, shape.max_top_nodes, shape.dtype,
           shape.T_q, flags)
    plan = _plans.get(key)
    if plan is None:
        plan = _lib.HtreePlan()
        _lib.check(_lib.lib().htree_b200_plan(shape, flags, plan), "plan")
        if len(_plans) >= 512:       # layouts are cheap to redo: callers with ever-changing lengths do not grow this for ever
            _plans.clear()
        _plans[key] = plan
    return plan


def _carve(ws: torch.Tensor, offset: int, shape, dtype) -> torch.Tensor:
    n = dtype.itemsize
    for x in shape:
        n *= x
    return ws[offset:offset + n].view(dtype).view(shape)


class _Workspace:
    """One buffer with everything a forward derived from k and v, and views of its parts in the reference's layouts."""

    def __init__(self, ws, plan, k, v, cr):
        self.ws, self.plan, self.k, self.v, self.cr = ws, plan, k, v, cr

    def _levels(self, offsets, first, D, dtype, lead=()):
        B, _, H_kv, _ = self.k.shape
        out = [first] if first is not None else []
        for l in range(len(out), self.plan.levels):
            out.append(_carve(self.ws, offsets[l], tuple(lead) + (B, self.plan.nodes[l], H_kv, D), dtype) if offsets[l] >= 0 else None)
        return out

    def layers_k(self):
        return self._levels(self.plan.layers_k, self.k, self.k.shape[3], self.k.dtype)

    def layers_v(self):
        return self._levels(self.plan.layers_v, self.v, self.v.shape[3], self.v.dtype)

    def blocks(self):
        L, p = self.plan.levels, self.plan
        ends = [self._block_bytes(l) for l in range(L)]
        fwd = [self.ws[p.blocks[l]:p.blocks[l] + ends[l][0]] for l in range(L)]
        bwd = [self.ws[p.blocks_bwd[l]:p.blocks_bwd[l] + ends[l][1]] for l in range(L)] if p.blocks_bwd[0] >= 0 else None
        return OperandBlocks(fwd, keys=fwd, blocks=fwd, blocks_bwd=bwd)

    def _block_bytes(self, l):
        B, _, H_kv, K = self.k.shape
        blocks, split = B * ((self.plan.nodes[l] + self.cr - 1) // self.cr) * H_kv, _split(self.k.dtype, K)
        n = blocks * (2 if split else 1) * K * 2 * self.cr
        return n * (2 if self.cr == 16 or not split else 3) + (128 * blocks if split else 0), n


class BwdContext(dict):
    """The forward's context: the reference's keys (bwd_ctx of src/parallel.py:1139-1159).  Views of the tree levels and operand
    copies are made when they are asked for."""

    _LAZY = ("layers_k", "layers_v", "layers_k_rot", "layers_v_blk", "rope_half", "per_layer_parents")
    workspace: Optional[_Workspace] = None
    parents: Optional[torch.Tensor] = None         # the kept selections of all levels, [L, B, T_q, H_kv, top_k]

    def __missing__(self, key):
        if key == "per_layer_parents" and self.parents is not None:
            val = dict(enumerate(self.parents.unbind(0)))
        elif key == "rope_half":
            k = self.workspace.k if self.workspace is not None else (self["layers_k"] or [None])[0]
            ok = k is not None and _selects_on_tensor_cores(k.dtype, k.shape[3])
            val = rope_cache_half(k.shape[3], self["cos_cache"].shape[0], self["rope_base"], self["scale"], k.device) if ok else None
        elif key == "layers_k_rot":      # the row-major K' that the one-kernel forms read; the transposed kernels do not
            lk = self["layers_k"]
            ok = lk is not None and _selects_on_tensor_cores(lk[0].dtype, lk[0].shape[3])
            val = rotate_keys(lk, self["compression_rate"], self["max_top_nodes"], self["rope_base"]) if ok else None
        elif key in self._LAZY and self.workspace is not None:
            val = self.workspace.blocks() if key == "layers_v_blk" else getattr(self.workspace, key)()
        else:
            raise KeyError(key)
        self[key] = val
        return val

    def get(self, key, default=None):
        try:
            return self[key]
        except KeyError:
            return default

    def __contains__(self, key):
        return super().__contains__(key) or key in self._LAZY

    def drop_tree(self):
        """Forget everything derived from k and v (a backward then rebuilds it)."""
        self.workspace = None
        for key in ("layers_k", "layers_v", "layers_k_rot", "layers_v_blk"):
            dict.__setitem__(self, key, None)


def build_operands(k: torch.Tensor, v: torch.Tensor, compression_rate: int, max_top_nodes: int, rope_base: float,
                   layers=None, backward: bool = False):
    """(layers_k, layers_v, None, OperandBlocks) in the form the transposed tensor-core kernels read, for a forward with
    `_layers`; from k, v alone, or from existing levels `layers` = (layers_k, layers_v).  None in the last two places for
    shapes without such kernels."""
    k = k.contiguous(); v = v.contiguous()
    B, T, H_kv, K = k.shape
    if not _transposed(k.dtype, K, v.shape[-1], 1, compression_rate):
        lk, lv = (list(layers[0]), list(layers[1])) if layers is not None else build_tree(k, v, compression_rate, max_top_nodes)
        return lk, lv, None, None
    cr = int(compression_rate)
    sizes = _lib.level_sizes(T, cr, max_top_nodes)
    shape = _lib.HtreeShape(B, T, H_kv, H_kv, K, K, cr, sizes[-1], int(max_top_nodes), _DTYPES[k.dtype])
    dev = k.device
    if layers is None:
        lk = [k] + [torch.empty(B, n, H_kv, K, dtype=k.dtype, device=dev) for n in sizes[1:]]
        lv = [v] + [torch.empty(B, n, H_kv, K, dtype=v.dtype, device=dev) for n in sizes[1:]]
    else:
        lk, lv = list(layers[0]), list(layers[1])
    n_blk = lambda l, bwd: int(_lib.lib().htree_b200_operand_block_bytes(ctypes.byref(shape), l, bwd))
    blocks = [torch.empty(n_blk(l, 0), dtype=torch.uint8, device=dev) for l in range(len(sizes))]
    bwd = [torch.empty(n_blk(l, 1), dtype=torch.uint8, device=dev) for l in range(len(sizes))] if backward else None
    cos_c, sin_c = rope_cache(K, 16, rope_base, dev)
    with _on_device(torch.device(dev).index):
        _lib.check(_lib.lib().htree_b200_prepare(ctypes.byref(shape), _ptrs(lk), _ptrs(lv), _ptrs(blocks), _ptrs(bwd) if bwd else None,
                                                 int(layers is None), cos_c.data_ptr(), sin_c.data_ptr(),
                                                 _stream()), "prepare")
    return lk, lv, None, OperandBlocks(blocks, keys=blocks, blocks=blocks, blocks_bwd=bwd)


def _pipelined(dtype, K: int, compression_rate: int) -> bool:
    """Shapes with a pipelined forward (operand blocks streamed through shared memory): 16-bit types, 128-wide heads,
    16 children per parent."""
    return dtype != torch.float32 and K == 128 and int(compression_rate) == 16


def build_tree_into(k: torch.Tensor, v: torch.Tensor, out_k, out_v, compression_rate: int, max_top_nodes: int) -> None:
    """Mean-pool tree of (k, v) with the pooled levels written into caller-provided tensors out_k[i], out_v[i]
    (level i+1; contiguous, shaped [B, N_{i+1}, H_kv, *]).  Sequence-sharded runs pool their slice of the leaves straight
    into their slot of the buffers that the all-gather then completes."""
    B, T, H_kv, K = k.shape
    V = v.shape[-1]
    sizes = _lib.level_sizes(T, compression_rate, max_top_nodes)
    assert len(out_k) == len(out_v) == len(sizes) - 1
    layers_k, layers_v = [k] + list(out_k), [v] + list(out_v)
    for x, n in zip(layers_k, sizes):
        assert x.is_contiguous() and x.shape[1] == n, "level tensors must be contiguous and of the level's length"
    for x in layers_v:
        assert x.is_contiguous()
    if len(sizes) == 1:
        return
    shape = _lib.HtreeShape(B, T, H_kv, H_kv, K, V, int(compression_rate), 1, int(max_top_nodes), _DTYPES[k.dtype])
    with _on_device(k.get_device()):
        _lib.check(_lib.lib().htree_b200_build_tree(ctypes.byref(shape), _ptrs(layers_k), _ptrs(layers_v), None, None, None, None,
                                                    None, _stream()), "build_tree")


def _split_half(dtype, K: int, V: int, compression_rate: int) -> bool:
    """fp32 storage on the tensor cores (operands carried as hi + lo half planes): 64-wide heads only."""
    return dtype == torch.float32 and K == 64 and V == 64 and int(compression_rate) in (8, 16)


def _rotatable(dtype, K: int, V: int, compression_rate: int) -> bool:
    return (dtype != torch.float32 and K % 16 == 0) or _split_half(dtype, K, V, compression_rate)


def _rotated_like(x: torch.Tensor) -> torch.Tensor:
    """K' buffer of one level: float16, for fp32 storage two planes (hi, lo)."""
    shape = ((2,) if x.dtype == torch.float32 else ()) + tuple(x.shape)
    return torch.empty(shape, dtype=torch.float16, device=x.device)


def _blockable(V: int, compression_rate: int) -> bool:
    return V in (64, 128) and int(compression_rate) in (8, 16)


def _blocked_like(x: torch.Tensor, compression_rate: int) -> torch.Tensor:
    B, N, H_kv, V = x.shape
    cr = int(compression_rate)
    if x.dtype == torch.float32:      # split-half planes (hi, lo) of float16
        return torch.empty(2, B, (N + cr - 1) // cr * cr, H_kv, V, dtype=torch.float16, device=x.device)
    return torch.empty(B, (N + cr - 1) // cr * cr, H_kv, V, dtype=x.dtype, device=x.device)


def block_values(layers_v, compression_rate: int, max_top_nodes: int, layers_k_rot=None):
    """Blocked copies of existing value levels (see build_tree) and, given the K' levels, of the keys where the pipelined
    forward applies; None for shapes the tensor-core forward does not cover."""
    v = layers_v[0]
    B, T, H_kv, V = v.shape
    if not _blockable(V, compression_rate) or (v.dtype == torch.float32 and V != 64):
        return None
    out = [_blocked_like(x, compression_rate) for x in layers_v]
    shape = _lib.HtreeShape(B, T, H_kv, H_kv, V, V, int(compression_rate), 1, int(max_top_nodes), _DTYPES[v.dtype])
    keys = None
    with _on_device(v.get_device()):
        _lib.check(_lib.lib().htree_b200_block_values(ctypes.byref(shape), _ptrs(layers_v), _ptrs(out), _stream()), "block_values")
        if layers_k_rot is not None and _pipelined(v.dtype, layers_k_rot[0].shape[-1], compression_rate):
            keys = [_blocked_like(x, compression_rate) for x in layers_k_rot]
            _lib.check(_lib.lib().htree_b200_block_keys(ctypes.byref(shape), _ptrs(layers_k_rot), _ptrs(keys), _stream()), "block_keys")
    return OperandBlocks(out, keys)


def rotate_keys(layers_k, compression_rate: int, max_top_nodes: int, rope_base: float):
    """K' levels (keys rotated by their child index) for existing tree levels; None where no tensor-core kernel reads them
    (K % 16 != 0, or fp32 storage with heads other than 64 wide)."""
    k = layers_k[0]
    B, T, H_kv, K = k.shape
    if not _rotatable(k.dtype, K, K, compression_rate):
        return None
    out = [_rotated_like(x) for x in layers_k]
    shape = _lib.HtreeShape(B, T, H_kv, H_kv, K, K, int(compression_rate), 1, int(max_top_nodes), _DTYPES[k.dtype])
    cos_c, sin_c = rope_cache(K, max(int(compression_rate), 16), rope_base, k.device)
    with _on_device(k.get_device()):
        _lib.check(_lib.lib().htree_b200_rotate_keys(ctypes.byref(shape), _ptrs(layers_k), _ptrs(out),
                                                     cos_c.data_ptr(), sin_c.data_ptr(), _stream()), "rotate_keys")
    return out


def _run_forward(shape, q, layers_k, layers_v, cos_cache, sin_cache, scale, out, gmax, gsum, parents, trace, flags,
                 layers_kr=None, half_tables=None, layers_vb=None):
    with _on_device(q.get_device()):
        rc = _lib.lib().htree_b200_forward(
            ctypes.byref(shape), q.data_ptr(), _ptrs(layers_k), _ptrs(layers_v),
            _ptrs(layers_kr) if layers_kr is not None else None,
            _ptrs(layers_vb.keys) if getattr(layers_vb, "keys", None) is not None else None,
            _ptrs(layers_vb) if layers_vb is not None else None,
            cos_cache.data_ptr(), sin_cache.data_ptr(),
            half_tables[0].data_ptr() if half_tables else None, half_tables[1].data_ptr() if half_tables else None,
            cos_cache.shape[0], float(scale),
            out.data_ptr() if out is not None else None, gmax.data_ptr() if gmax is not None else None,
            gsum.data_ptr() if gsum is not None else None, _ptrs(parents) if parents is not None else None,
            ctypes.byref(trace) if trace is not None else None, _status(q.device).data_ptr(), flags, _stream())
    _lib.check(rc, "forward")


def htree_forward(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
    compression_rate: int = 16, max_top_nodes: int = 8192, top_k_per_layer: int = 512,
    scale: Optional[float] = None, rope_base: float = 10000.0,
    _save_for_backward: bool = False, _save_parents: bool = True,
    return_trace: bool = False, _force_generic: bool = False, _q_offset: Optional[int] = None, _layers=None,
    _fused: bool = False, _tiled: bool = False, _no_pipeline: bool = False,
):
    """htree forward.  q [B,T,H,K], k [B,T,H_kv,K], v [B,T,H_kv,V] -> out [B,T,H,V] in q's dtype.

    Returns `out`, or `(out, bwd_ctx)` with `_save_for_backward` (the reference's contract, src/parallel.py:1139-1159),
    with a third element — {"num_layers", "num_groups", "layers": {l: LayerTrace}} — when `return_trace` is set
    (the shape of htree_forward_naive's trace, src/naive.py:225-234).

    `_fused` bounds the temporaries of a call that keeps no selections (windows of queries, see SPLIT_FORWARD_MAX_BYTES; no effect
    where they are kept);
    `_no_pipeline` is accepted and has no effect (there is one accumulation kernel); `_tiled` concerns the generic kernels.

    Sequence sharding: with `_q_offset` = t0, q holds only the query positions t0 .. t0+q.shape[1]-1 while k, v (or the
    prebuilt tree `_layers` = (layers_k, layers_v)) cover the whole sequence; outputs have q's length."""
    shape = _validate(q, k, v, compression_rate, max_top_nodes, top_k_per_layer, _q_offset)
    B, T, H, K = q.shape
    H_kv, V = k.shape[2], v.shape[-1]
    if scale is None:
        scale = K ** -0.5
    q = q.contiguous(); k = k.contiguous(); v = v.contiguous()
    if (not (_force_generic or return_trace) and _transposed(q.dtype, K, V, H // H_kv, compression_rate) and q.data_ptr() % 32 == 0
            and k.data_ptr() % 16 == 0 and v.data_ptr() % 16 == 0):
        if not (_save_for_backward or _fused or _layers is not None) and _lib.glue():
            n_pos = top_k_per_layer * compression_rate + 1024
            out = _lib.glue().plain_forward(q, k, v, _tables(K, n_pos, rope_base, scale, _split(q.dtype, K), q.get_device())[:5],
                                            compression_rate, max_top_nodes, top_k_per_layer, scale,
                                            -1 if _q_offset is None else _q_offset, SPLIT_FORWARD_MAX_BYTES)
            if out is not None:
                return out
        return _forward_transposed(shape, q, k, v, scale, rope_base, _save_for_backward, _save_parents, _layers, _fused)
    dev = q.device
    if _layers is not None:
        layers_k, layers_v = _layers[0], _layers[1]
    else:
        layers_k, layers_v = build_tree(k, v, compression_rate, max_top_nodes)
    L = len(layers_k)
    cos_cache, sin_cache = rope_cache(K, top_k_per_layer * compression_rate + 1024, rope_base, dev)
    out = torch.empty(B, T, H, V, dtype=q.dtype, device=dev)
    gmax = torch.empty(B, T, H, dtype=torch.float32, device=dev)
    gsum = torch.empty(B, T, H, dtype=torch.float32, device=dev)
    want_parents = (_save_for_backward and _save_parents) or return_trace
    parents = [torch.empty(B, q.shape[1], H_kv, top_k_per_layer, dtype=_parents_dtype(layers_k, top_k_per_layer), device=dev)
               for _ in range(L)] if want_parents else None
    trace = tr = None
    if return_trace:
        tr = (torch.empty(L, B, T, H, dtype=torch.float32, device=dev),
              torch.empty(L, B, T, H, dtype=torch.float32, device=dev),
              torch.empty(L, B, T, H, V, dtype=torch.float32, device=dev))
        trace = _lib.HtreeTrace(tr[0].data_ptr(), tr[1].data_ptr(), tr[2].data_ptr())
    flags = _lib.FWD_GENERIC | (_lib.FWD_TILED if _tiled else 0) | _parents_flag(parents)
    _run_forward(shape, q, layers_k, layers_v, cos_cache, sin_cache, scale, out, gmax, gsum, parents, trace, flags)
    if not (_save_for_backward or return_trace):
        return out
    result = [out]
    if _save_for_backward:
        result.append(dict(
            _context_fields(gmax, gsum, cos_cache, sin_cache, L, shape, rope_base, scale),
            per_layer_parents={l: parents[l] for l in range(L)} if (_save_parents and want_parents) else None,
            layers_k=layers_k, layers_v=layers_v, layers_k_rot=None, layers_v_blk=None, rope_half=None))
    if return_trace:
        check_status(dev)
        layers = {l: LayerTrace(l, decode_parents(parents[l - 1]) if l > 0 else None, tr[0][l], tr[1][l], tr[2][l])
                  for l in range(L)}
        result.append({"num_layers": L, "num_groups": H // H_kv, "selection_mode": "parallel_importance",
                       "layers": layers})
    return tuple(result)


def _context_fields(gmax, gsum, cos_cache, sin_cache, L, shape, rope_base, scale) -> dict:
    G = shape.H // shape.H_kv
    return dict(global_max=gmax, global_sum=gsum, cos_cache=cos_cache, sin_cache=sin_cache, num_layers=L, rope_base=rope_base,
                compression_rate=shape.compression_rate, top_k_per_layer=shape.top_k, max_top_nodes=shape.max_top_nodes, scale=scale,
                NUM_GROUPS=G,
                # tuning constants of the reference's Triton kernels; kept so that code reading them keeps working
                G_PAD=max(16, 1 << (G - 1).bit_length()), TILE_P=4, DROP_BLOCK=64)


def _forward_transposed(shape, q, k, v, scale, rope_base, save, save_parents, given_layers, windows):
    """The forward on the transposed tensor-core kernels: operand preparation, selection, accumulation."""
    B, Tq, H, K = q.shape
    H_kv, TK, CR = shape.H_kv, shape.top_k, shape.compression_rate
    dev, dtype, index = q.device, q.dtype, q.get_device()
    n_pos = TK * CR + 1024
    cos_cache, sin_cache, table, table32, _, cos_ptr, sin_ptr, tab_ptr, tab32_ptr, status_ptr = _tables(
        K, n_pos, rope_base, scale, _split(dtype, K), index)
    keep = save and save_parents
    # Callers that do not keep the selections get them only as temporaries (int32 whatever SELECTION_STORAGE says), and only up
    # to SPLIT_FORWARD_MAX_BYTES at a time: beyond it the queries run window by window over the same tree, with the same results.
    plan = _plan(shape, _lib.PLAN_BACKWARD if save else 0)
    L = plan.levels
    out = torch.empty_like(q)
    stats = torch.empty((2, B, Tq, H), dtype=torch.float32, device=dev)
    per_query = L * H_kv * TK * 4
    ws = layers = parents = None
    if not keep and (windows or B * Tq * per_query > SPLIT_FORWARD_MAX_BYTES):
        layers = _operand_layers(k, v, shape, rope_base, given_layers, save)
        _forward_windows(shape, q, layers, cos_cache, sin_cache, (table, table32), scale, out, stats[0], stats[1], per_query)
    else:
        pdt = _parents_dtype_of(plan, TK) if keep else torch.int32
        parents = torch.empty((L, B, Tq, H_kv, TK), dtype=pdt, device=dev)
        flags = (0 if save or given_layers is not None else _lib.FWD_INFERENCE) | (_lib.PARENTS_U16 if pdt == torch.int16 else 0)
        pptr = _lib.address_array(parents.data_ptr(), B * Tq * H_kv * TK * pdt.itemsize, L)
        gmax_ptr = stats.data_ptr()
        gsum_ptr = gmax_ptr + B * Tq * H * 4
        with _on_device(index):
            if given_layers is None:
                ws = torch.empty(plan.bytes, dtype=torch.uint8, device=dev)
                rc = _lib.lib().htree_b200_run_forward(
                    shape, plan, q.data_ptr(), k.data_ptr(), v.data_ptr(), cos_ptr, sin_ptr, tab_ptr, tab32_ptr, n_pos, scale,
                    ws.data_ptr(), out.data_ptr(), gmax_ptr, gsum_ptr, pptr, status_ptr, flags,
                    torch._C._cuda_getCurrentRawStream(index))
            else:
                layers = _operand_layers(k, v, shape, rope_base, given_layers, save)
                rc = _attend(shape, q, layers, cos_cache, sin_cache, (table, table32), scale, out.data_ptr(), gmax_ptr, gsum_ptr, pptr, flags)
        if rc:
            _lib.check(rc, "forward")
    if not save:
        return out
    ctx = BwdContext(_context_fields(stats[0], stats[1], cos_cache, sin_cache, L, shape, rope_base, scale))
    if keep:
        ctx.parents = parents
    else:
        ctx["per_layer_parents"] = None
    if ws is not None:
        ctx.workspace = _Workspace(ws, plan, k, v, CR)
    else:
        ctx.update(layers_k=layers[0], layers_v=layers[1], layers_v_blk=layers[3])
    return out, ctx


def _parents_dtype_of(plan, top_k: int):
    if SELECTION_STORAGE == "int32":
        return torch.int32
    if SELECTION_STORAGE != "uint16":
        raise ValueError(f"SELECTION_STORAGE must be 'int32' or 'uint16', not {SELECTION_STORAGE!r}")
    if top_k > 65535 or any(plan.nodes[l] > 65535 for l in range(1, plan.levels)):
        raise ValueError("SELECTION_STORAGE='uint16' needs pooled levels of at most 65535 nodes")
    return torch.int16


def _operand_layers(k, v, shape, rope_base, given, backward):
    """(layers_k, layers_v, layers_k_rot, OperandBlocks) for the transposed kernels, from the caller's levels where given."""
    if given is None:
        return build_operands(k, v, shape.compression_rate, shape.max_top_nodes, rope_base, backward=backward)
    if len(given) > 3 and getattr(given[3], "blocks", None) is not None and (not backward or given[3].blocks_bwd is not None):
        return given
    return build_operands(given[0][0], given[1][0], shape.compression_rate, shape.max_top_nodes, rope_base, layers=given, backward=backward)


def _attend(shape, q, layers, cos_cache, sin_cache, tables, scale, out_ptr, gmax_ptr, gsum_ptr, pptr, flags) -> int:
    return _lib.lib().htree_b200_attend(
        ctypes.byref(shape), q.data_ptr(), _ptrs(layers[0]), _ptrs(layers[1]), _ptrs(layers[3].blocks),
        cos_cache.data_ptr(), sin_cache.data_ptr(), tables[0].data_ptr(), tables[1].data_ptr(), cos_cache.shape[0], float(scale),
        out_ptr, gmax_ptr, gsum_ptr, pptr, _status(q.device).data_ptr(), flags, _stream())


def _forward_windows(shape, q, layers, cos_cache, sin_cache, tables, scale, out, gmax, gsum, per_query):
    """The forward over windows of query positions, one batch element at a time, whose selections fit
    SPLIT_FORWARD_MAX_BYTES."""
    B, Tq, H, K = q.shape
    L = len(layers[0])
    step = max(1, min(Tq, SPLIT_FORWARD_MAX_BYTES // per_query))
    parents = torch.empty(L, step, shape.H_kv, shape.top_k, dtype=torch.int32, device=q.device)
    pptr = _ptrs(parents.unbind(0))
    t_offset = shape.t_offset
    with _on_device(q.get_device()):
        for b in range(B):
            blocks = OperandBlocks([])
            blocks.blocks = [x.view(B, -1)[b] for x in layers[3].blocks]
            one = [[x[b:b + 1] for x in layers[0]], [x[b:b + 1] for x in layers[1]], None, blocks]
            for a in range(0, Tq, step):
                n = min(step, Tq - a)
                w = _lib.HtreeShape(1, shape.T, shape.H, shape.H_kv, shape.K, shape.V, shape.compression_rate, shape.top_k,
                                    shape.max_top_nodes, shape.dtype, n, t_offset + a)
                _lib.check(_attend(w, q[b:b + 1, a:a + n], one, cos_cache, sin_cache, tables, scale, out[b, a:].data_ptr(),
                                   gmax[b, a:].data_ptr(), gsum[b, a:].data_ptr(), pptr, 0), "forward")


def recompute_parents(q, layers_k, layers_v, cos_cache, sin_cache, compression_rate, top_k_per_layer,
                      max_top_nodes, scale, layers_k_rot=None, _force_generic=False, layers_v_blk=None,
                      rope_base: Optional[float] = None) -> Dict[int, torch.Tensor]:
    """Selection-only replay of the forward (the reference's _recompute_parents, src/backward.py:881-934)."""
    B, T, H, K = q.shape
    H_kv, V = layers_k[0].shape[2], layers_v[0].shape[-1]
    shape = _lib.HtreeShape(B, T, H, H_kv, K, V, int(compression_rate), int(top_k_per_layer), int(max_top_nodes),
                            _DTYPES[q.dtype])
    L = len(layers_k)
    parents = [torch.empty(B, T, H_kv, top_k_per_layer, dtype=_parents_dtype(layers_k, top_k_per_layer), device=q.device)
               for _ in range(L)]
    if rope_base is not None and getattr(layers_v_blk, "blocks", None) is not None and not _force_generic and q.is_contiguous() and q.data_ptr() % 32 == 0:
        rows = rope_rows_select(K, cos_cache.shape[0], rope_base, q.device)
        tables = (rows, rows)                            # the selection reads the second only
        with _on_device(q.get_device()):
            _lib.check(_attend(shape, q, (layers_k, layers_v, None, layers_v_blk), cos_cache, sin_cache, tables, scale, None, None, None,
                               _ptrs(parents), _lib.FWD_SELECT_ONLY | _parents_flag(parents)), "select")
        return {l: parents[l] for l in range(L)}
    _run_forward(shape, q.contiguous(), layers_k, layers_v, cos_cache, sin_cache, scale, None, None, None, parents,
                 None, _lib.FWD_SELECT_ONLY | (_lib.FWD_GENERIC if _force_generic else 0) | _parents_flag(parents),
                 layers_k_rot, None, layers_v_blk)
    return {l: parents[l] for l in range(L)}


_DO_DTYPE = ("dO has dtype {} but q has {}: pass the output gradient in the operator's storage type (cast it explicitly if the loss "
             "of precision is acceptable)")
_bwd_plans: Dict[Tuple, Optional[Tuple[int, int]]] = {}


def _backward_operands(q, ctx):
    """(blocks pointers, blocks_bwd pointers, T, H_kv) of a context with the transposed kernels' operands, else None."""
    ws = getattr(ctx, "workspace", None)
    if ws is not None and not dict.__contains__(ctx, "layers_k"):
        p, base = ws.plan, ws.ws.data_ptr()
        if p.blocks_bwd[0] < 0:
            return None
        L = range(p.levels)
        return ([base + p.blocks[l] for l in L], [base + p.blocks_bwd[l] for l in L], ws.k.shape[1], ws.k.shape[2])
    blk = ctx.get("layers_v_blk")
    if getattr(blk, "blocks_bwd", None) is None:
        return None
    k = ctx["layers_k"][0]
    return ([x.data_ptr() for x in blk.blocks], [x.data_ptr() for x in blk.blocks_bwd], k.shape[1], k.shape[2])


def _backward_two_pass(dO, q, output, ctx, operands, typed, window):
    """The backward on the two-pass kernels; None where their scratch does not fit BACKWARD_MAX_BYTES or an operand is not
    32-byte aligned (the one-pass backward then runs)."""
    B, Tq, H, K = q.shape
    blocks, blocks_bwd, T, H_kv = operands
    if (q.data_ptr() | dO.data_ptr() | output.data_ptr()) % 32:
        return None
    CR, TK, MTN = int(ctx["compression_rate"]), int(ctx["top_k_per_layer"]), int(ctx["max_top_nodes"])
    budget = BACKWARD_MAX_BYTES
    key = (B, T, H, H_kv, K, CR, TK, MTN, q.dtype, Tq, budget)
    shape = _lib.HtreeShape(B, T, H, H_kv, K, K, CR, TK, MTN, _DTYPES[q.dtype], 0 if window is None else Tq,
                            0 if window is None else int(window["t0"]))
    if key not in _bwd_plans:
        a, s = ctypes.c_int64(), ctypes.c_int64()
        rc = _lib.lib().htree_b200_backward_plan(shape, budget, ctypes.byref(a), ctypes.byref(s))
        if len(_bwd_plans) >= 512:
            _bwd_plans.clear()
        _bwd_plans[key] = ((a.value + 255) // 256 * 256, s.value) if rc == 0 else None
    plan = _bwd_plans[key]
    if plan is None or window is not None and not window["first"] and "two_pass" not in window["acc"]:
        return None
    dev, dtype, index = q.device, q.dtype, q.get_device()
    L = len(blocks)
    kept = getattr(ctx, "parents", None)
    if kept is not None and not dict.__contains__(ctx, "per_layer_parents"):
        pptr = _lib.address_array(kept.data_ptr(), kept.stride(0) * kept.element_size(), L)
        pflag = _lib.PARENTS_U16 if kept.dtype == torch.int16 else 0
    else:
        parents = ctx.get("per_layer_parents")
        if parents is None:
            parents = recompute_parents(q, ctx["layers_k"], ctx["layers_v"], ctx["cos_cache"], ctx["sin_cache"], CR, TK, MTN, ctx["scale"],
                                        layers_v_blk=ctx["layers_v_blk"], rope_base=ctx["rope_base"])
        kept = [parents[l] for l in range(L)]
        pptr, pflag = _ptrs(kept), _parents_flag(kept)
    n_pos, scale = ctx["cos_cache"].shape[0], float(ctx["scale"])
    t = _tables(K, n_pos, ctx["rope_base"], scale, _split(dtype, K), index)
    if window is None:
        scratch = torch.empty(plan[0] + plan[1], dtype=torch.uint8, device=dev)
        acc_ptr, flags, final = scratch.data_ptr(), 0, True
        scratch_ptr = acc_ptr + plan[0]
    else:
        if window["first"]:
            window["acc"]["two_pass"] = torch.empty(plan[0], dtype=torch.uint8, device=dev)
        acc_ptr, final = window["acc"]["two_pass"].data_ptr(), window["last"]
        flags = (0 if window["first"] else _lib.BWD_KEEP_ACCUM) | (0 if final else _lib.BWD_NO_FOLD)
        scratch = torch.empty(plan[1], dtype=torch.uint8, device=dev)
        scratch_ptr = scratch.data_ptr()
    gdt = dtype if typed else torch.float32
    dq = torch.empty((B, Tq, H, K), dtype=gdt, device=dev)
    dk = dv = None
    if final:
        dk = torch.empty((B, T, H_kv, K), dtype=gdt, device=dev)
        dv = torch.empty((B, T, H_kv, K), dtype=gdt, device=dev)
    with _on_device(index):
        rc = _lib.lib().htree_b200_run_backward(
            shape, q.data_ptr(), _lib.ptr_array(blocks), _lib.ptr_array(blocks_bwd), t[5], t[6], t[7], n_pos, scale, output.data_ptr(),
            dO.data_ptr(), ctx["global_max"].data_ptr(), ctx["global_sum"].data_ptr(), pptr, acc_ptr, scratch_ptr, budget, dq.data_ptr(),
            dk.data_ptr() if final else None, dv.data_ptr() if final else None, 1 if typed else 0, t[9], flags | pflag,
            torch._C._cuda_getCurrentRawStream(index))
    if rc:
        _lib.check(rc, "backward")
    return dq, dk, dv


def htree_backward(dO: torch.Tensor, q: torch.Tensor, output: torch.Tensor, bwd_ctx: dict, _force_generic: bool = False,
                   _typed: bool = False, _window: Optional[dict] = None):
    """Backward given the forward context; returns fp32 (dq, dk, dv) with the shapes of q, k, v
    (src/backward.py:941-1119).  If bwd_ctx['per_layer_parents'] is None the selections are rebuilt first.

    `_typed=True` returns the three gradients in q's dtype instead, rounded once inside the kernels: what the
    reference's autograd function produces by casting the fp32 results afterwards (src/backward.py:1193), without the
    fp32 dq tensor and the extra passes over memory.
    dO must have q's dtype (the kernels read it in the storage type; the reference up-casts both to fp32,
    src/backward.py:966): a wider dO is refused rather than rounded silently.

    `_window` runs the backward over consecutive query windows that share the dK/dV accumulators (what the host-buffer
    pipeline does to overlap transfers with kernels): {"t0": first position of this window, "first": bool, "last": bool,
    "acc": dict kept by the caller across the windows of one backward}.  q, dO, output and bwd_ctx then belong to the
    window (a forward called with `_q_offset`); dq is returned for the window, dk and dv only with the last window
    (None before)."""
    B, T, H, K = q.shape
    two_pass = None if _force_generic else _backward_operands(q, bwd_ctx)
    if two_pass is not None:
        if dO.dtype != q.dtype:
            raise ValueError(_DO_DTYPE.format(dO.dtype, q.dtype))
        res = _backward_two_pass(dO.contiguous(), q.contiguous(), output.contiguous(), bwd_ctx, two_pass, _typed, _window)
        if res is not None:
            return res
    layers_k, layers_v = bwd_ctx["layers_k"], bwd_ctx["layers_v"]
    H_kv, V = layers_k[0].shape[2], layers_v[0].shape[-1]
    L = bwd_ctx["num_layers"]
    CR, TK, MTN = bwd_ctx["compression_rate"], bwd_ctx["top_k_per_layer"], bwd_ctx["max_top_nodes"]
    scale = bwd_ctx["scale"]
    cos_cache, sin_cache = bwd_ctx["cos_cache"], bwd_ctx["sin_cache"]
    layers_kr = bwd_ctx.get("layers_k_rot")
    half_tables = bwd_ctx.get("rope_half")
    dev = q.device
    q = q.contiguous()
    if dO.dtype != q.dtype:
        raise ValueError(_DO_DTYPE.format(dO.dtype, q.dtype))
    dO = dO.contiguous()
    output = output.contiguous()
    parents = bwd_ctx.get("per_layer_parents")
    if parents is None:
        parents = recompute_parents(q, layers_k, layers_v, cos_cache, sin_cache, CR, TK, MTN, scale,
                                    bwd_ctx.get("layers_k_rot"), layers_v_blk=bwd_ctx.get("layers_v_blk"))
    flags = 0
    if _window is None:
        shape = _lib.HtreeShape(B, T, H, H_kv, K, V, int(CR), int(TK), int(MTN), _DTYPES[q.dtype])
        dk_levels = [torch.empty(x.shape, dtype=torch.float32, device=dev) for x in layers_k]
        dv_levels = [torch.empty(x.shape, dtype=torch.float32, device=dev) for x in layers_v]
    else:
        T_full = layers_k[0].shape[1]
        shape = _lib.HtreeShape(B, T_full, H, H_kv, K, V, int(CR), int(TK), int(MTN), _DTYPES[q.dtype], T, int(_window["t0"]))
        acc = _window["acc"]
        if _window["first"]:
            acc["dk"] = [torch.empty(x.shape, dtype=torch.float32, device=dev) for x in layers_k]
            acc["dv"] = [torch.empty(x.shape, dtype=torch.float32, device=dev) for x in layers_v]
        dk_levels, dv_levels = acc["dk"], acc["dv"]
        flags |= (0 if _window["first"] else _lib.BWD_KEEP_ACCUM) | (0 if _window["last"] else _lib.BWD_NO_FOLD)
    final = _window is None or _window["last"]
    typed = None
    if _typed:
        dq = torch.empty(B, T, H, K, dtype=q.dtype, device=dev)
        # before the last window the leaf gradients are not written; the struct still wants valid pointers
        dk_t = torch.empty(layers_k[0].shape if final else (8,), dtype=q.dtype, device=dev)
        dv_t = torch.empty(layers_v[0].shape if final else (8,), dtype=q.dtype, device=dev)
        typed = _lib.HtreeTypedGrads(dq.data_ptr(), dk_t.data_ptr(), dv_t.data_ptr())
    else:
        dq = torch.empty(B, T, H, K, dtype=torch.float32, device=dev)
    with _on_device(torch.device(dev).index):
        rc = _lib.lib().htree_b200_backward(
            ctypes.byref(shape), q.data_ptr(), _ptrs(layers_k), _ptrs(layers_v),
            _ptrs(layers_kr) if layers_kr is not None else None, cos_cache.data_ptr(), sin_cache.data_ptr(),
            half_tables[0].data_ptr() if half_tables else None, half_tables[1].data_ptr() if half_tables else None,
            cos_cache.shape[0], float(scale), output.data_ptr(), dO.data_ptr(),
            bwd_ctx["global_max"].data_ptr(), bwd_ctx["global_sum"].data_ptr(),
            _ptrs([parents[l] for l in range(L)]), None if _typed else dq.data_ptr(), _ptrs(dk_levels), _ptrs(dv_levels),
            ctypes.byref(typed) if typed is not None else None, _status(dev).data_ptr(),
            flags | (_lib.FWD_GENERIC if _force_generic else 0) | _parents_flag([parents[l] for l in range(L)]), _stream())
    _lib.check(rc, "backward")
    if not final:
        return dq, None, None
    if _typed:
        return dq, dk_t, dv_t
    return dq, dk_levels[0], dv_levels[0]


class HTreeFunction(torch.autograd.Function):
    """Differentiable htree attention (the reference's HTreeTritonFunction, src/backward.py:1126-1193)."""

    @staticmethod
    def forward(ctx, q, k, v, compression_rate, max_top_nodes, top_k_per_layer, scale, rope_base):
        save = SAVE_SELECTIONS_FOR_BACKWARD
        output, bwd_ctx = htree_forward(q, k, v, compression_rate=compression_rate, max_top_nodes=max_top_nodes,
                                        top_k_per_layer=top_k_per_layer, scale=scale, rope_base=rope_base,
                                        _save_for_backward=True, _save_parents=save)
        ctx.save_for_backward(q, k, v, output, bwd_ctx["global_max"], bwd_ctx["global_sum"])
        ctx.bwd_ctx = bwd_ctx
        if not save:   # like the reference: drop the pooled levels and rebuild them in backward
            if isinstance(bwd_ctx, BwdContext):
                bwd_ctx.drop_tree()
            else:
                bwd_ctx["layers_k"] = bwd_ctx["layers_v"] = bwd_ctx["layers_k_rot"] = bwd_ctx["layers_v_blk"] = None
        return output

    @staticmethod
    def backward(ctx, dO):
        q, k, v, output, gmax, gsum = ctx.saved_tensors
        c = ctx.bwd_ctx
        if getattr(c, "workspace", None) is None and c["layers_k"] is None:
            c = dict(c)
            c["layers_k"], c["layers_v"], c["layers_k_rot"], c["layers_v_blk"] = build_operands(
                k, v, c["compression_rate"], c["max_top_nodes"], c["rope_base"], backward=True)
        dq, dk, dv = htree_backward(dO.to(q.dtype), q, output, c, _typed=True)    # gradients come back in the input dtype
        return dq, dk, dv, None, None, None, None, None


HTreeTritonFunction = HTreeFunction   # drop-in name of the reference


def htree_forward_autograd(q, k, v, compression_rate: int = 16, max_top_nodes: int = 8192,
                           top_k_per_layer: int = 512, scale: Optional[float] = None, rope_base: float = 10000.0):
    """Differentiable forward (signature of htree_forward_triton_autograd, src/backward.py:1196-1208)."""
    if scale is None:
        scale = q.shape[-1] ** -0.5
    if SAVE_SELECTIONS_FOR_BACKWARD and SELECTION_STORAGE == "int32" and q.dim() == 4 and _lib.glue():
        q = q.contiguous(); k = k.contiguous(); v = v.contiguous()
        _validate(q, k, v, compression_rate, max_top_nodes, top_k_per_layer)
        K = q.shape[3]
        if _transposed(q.dtype, K, v.shape[3], q.shape[2] // k.shape[2], compression_rate):
            out = _lib.glue().autograd_forward(
                q, k, v, _tables(K, top_k_per_layer * compression_rate + 1024, rope_base, scale, _split(q.dtype, K), q.get_device())[:5],
                compression_rate, max_top_nodes, top_k_per_layer, scale, BACKWARD_MAX_BYTES)
            if out is not None:
                return out
    return HTreeFunction.apply(q.contiguous(), k.contiguous(), v.contiguous(), compression_rate, max_top_nodes,
                               top_k_per_layer, scale, rope_base)


htree_forward_triton_autograd = htree_forward_autograd   # drop-in name of the reference

__all__ = [
    "decode_parents", "HTREE_SCORE_NEG_INF", "HTREE_SCORE_VALID_THRESHOLD", "LayerTrace", "build_tree", "rope_cache",
    "rotate_keys", "block_values", "build_operands",
    "htree_forward", "htree_backward", "recompute_parents", "HTreeFunction", "HTreeTritonFunction",
    "htree_forward_autograd", "htree_forward_triton_autograd", "check_status",
]
