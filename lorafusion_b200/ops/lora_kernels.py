"""Kernel-level building blocks of the fused (multi-)LoRA linear layer.

The functions of the table are one launch each, of the tcgen05 GEMM kernels or of the rank-wide
kernel (``csrc/gemm/lora_skinny.cu``); ``linear_fwd`` / ``linear_bwd`` issue a whole layer's launches
in one native call.  Together they replace the reference's Triton kernels K1-K11 and its
cuBLAS calls for the skinny products (``lorafusion/ops/lora_v1.py:87-166``,
``lorafusion/ops/multi_lora.py:456-600``):

================  =========================================  ===============================
function          computes                                   reference counterpart
================  =========================================  ===============================
``lora_down``     ``S' = alpha_a * drop(X) A_a^T``            dropout.py + ``X̂ @ Aᵀ`` (cuBLAS),
                                                              fused_dropout_matmul.py
``base_lora_fwd`` ``Y = X W^T + S' B_a^T (+ bias)``           fused_(multi_)lora_xw_sb(_tma).py
``lora_ds``       ``dS = alpha_a * dY B_a``                   fused_(multi_)lora_dys_dyb.py (dS half)
``lora_db``       ``dB_a += dY^T S'``                         fused_(multi_)lora_dys_dyb.py (dB half)
``lora_da``       ``dA_a += dS^T drop(X)``                    ``dSᵀ @ X̂`` (cuBLAS loop)
``base_lora_dx``  ``dX = dY W + keep (.) (dS A_a)/(1-p)``     fused_(multi_)lora_dyw_dsa(_tma).py
================  =========================================  ===============================

Conventions
-----------
* Tokens are packed ``[M, features]``; every 128-row tile belongs to one adapter
  (``tile_adapter[m_tile]``, ``-1`` = no adapter) -- the solver pads each adapter's
  segment to a multiple of 128 tokens.
* Adapters are stacked and rank-padded to ``R`` (64, 128, 192 or 256) with zeros:
  ``A_all [n, R, K]``, ``B_all [n, N, R]``; the kernels index them by adapter id, so there
  are no per-call pointer tables and no limit of four adapters.
* ``alpha`` (= lora_alpha / r) is applied to the fp32 accumulator when ``S'`` and ``dS``
  are produced, never folded into bf16 weights.
* The dropout mask is regenerated from Philox (``ops/philox.py``) -- nothing is stored.
"""

from __future__ import annotations

import ctypes as C
import functools
from dataclasses import dataclass, field
from typing import Optional, Sequence

import torch

from . import _native as nv
from .gemm import check2d, launch_gemm, launch_skinny, pair_scratch, use_pair
from .philox import dropout_threshold
from .tile_config import get_kernel_config

RANK_PAD = 64
RANK_PADS = (64, 128, 192, 256)  # stacked-rank widths the skinny kernels are built for
TILE_M = 128
# N tile of the dX kernel with dropout: 256 = two single-buffered accumulators,
# 128 = two double-buffered accumulators
DROPMIX_BN = int(__import__('os').environ.get('LORAFUSION_B200_DROPMIX_BN', '256'))


@dataclass
class DropoutSpec:
    """Dropout state of one LoRA linear call: a seed, a stream id unique to the call site
    (layer / projection) and either one ``p`` or per-adapter thresholds."""

    seed: int = 0
    stream_id: int = 0
    p: float = 0.0
    adapter_thresh16: Optional[torch.Tensor] = None  # int32/uint32 [n_adapters]
    adapter_inv_keep: Optional[torch.Tensor] = None  # fp32 [n_adapters]
    row_offset: int = 0
    col_offset: int = 0

    @property
    def active(self) -> bool:
        return self.p > 0.0 or self.adapter_thresh16 is not None

    def kwargs(self) -> dict:
        return dict(
            thresh16=dropout_threshold(self.p),
            inv_keep=1.0 / (1.0 - self.p) if self.p > 0 else 1.0,
            adapter_thresh16=self.adapter_thresh16,
            adapter_inv_keep=self.adapter_inv_keep,
            seed=self.seed,
            stream_id=self.stream_id,
            row_offset=self.row_offset,
            col_offset=self.col_offset,
        )


NO_DROPOUT = DropoutSpec()


# How many CTAs share the reduction of one 128-row output tile of a rank-wide product.  Two such
# CTAs fit on an SM, so a launch has 296 places: the reduction is cut in two, four or eight while
# all pieces still run at once and each keeps at least two 64-deep blocks to sum.  Measured (us for
# 1, 2, 4, 8 CTAs a tile, S' with dropout): 100 x 1024 16.6 11.8 8.7 7.7; 8192 x 4096 60.9 35.8 28.5
# 37.0 (eight no longer fit); 16384 x 4096 63.1 50.2 56.3 69.8.
_SPLIT_PLACES = 2 * 148
_SPLIT_MIN_BLOCKS = 2
_SPLIT_MAX = 8


@functools.lru_cache(maxsize=4096)
def reduction_split(tiles: int, k_blocks: int) -> int:
    """CTAs per output tile (1, 2, 4 or 8) for ``tiles`` tiles that sum ``k_blocks`` blocks each."""
    c = 1
    while c < _SPLIT_MAX and tiles * c * 2 <= _SPLIT_PLACES and k_blocks >= _SPLIT_MIN_BLOCKS * c * 2:
        c *= 2
    return c


@dataclass
class SegmentTable:
    """Token segments of one packed microbatch: ``(adapter, start, end)`` with ``start`` and
    ``end`` multiples of 128 and at most one segment per adapter (but see :meth:`passes`).  ``staged`` (optional):
    ``(int32 device tensor, first, end)`` where the :func:`segment_rows` of the segments already lie."""

    segments: Sequence[tuple[int, int, int]]
    device: torch.device
    total_rows: Optional[int] = None
    staged: Optional[tuple] = None
    _cache: dict = field(default_factory=dict)

    @property
    def repeats(self) -> bool:
        """Whether an adapter owns more than one segment."""
        return len(self._passes()) > 1

    def _passes(self) -> list:
        """How many rows of :func:`segment_rows` belong to each launch: first segments, second ones, ..."""
        n = self._cache.get("passes")
        if n is None:
            n = [len(g) for g in _by_occurrence(self.segments)] or [0]
            self._cache["passes"] = n
        return n

    def _rows(self) -> torch.Tensor:
        """:func:`segment_rows` on the device."""
        t = self._cache.get("rows")
        if t is None:
            for adapter, start, end in self.segments:
                last = self.total_rows is not None and end >= self.total_rows
                if adapter >= 0 and end > start and (start % TILE_M or (end % TILE_M and not last)):
                    raise ValueError("segment bounds must be multiples of 128 tokens")
            if self.staged is not None:
                src, first, end = self.staged
                t = src[first:end].view(-1, 4)
            else:
                t = torch.tensor(segment_rows(self.segments), dtype=torch.int32).reshape(-1, 4).to(self.device)
            self._cache["rows"] = t
        return t

    def device_rows(self) -> torch.Tensor:
        """int32 ``[n, 4]`` work list ``(adapter, start, end, 0)`` of the gradient kernels; every adapter once."""
        if self.repeats:
            raise ValueError("an adapter may own only one token segment per microbatch")
        return self._rows()

    def passes(self, features: int) -> list:
        """The work lists of a gradient product of ``features`` features, to be launched one after the other: one,
        unless an adapter owns several segments.  That is taken for long segments and few features (fewer than
        96 pieces of segment x 128 features, a segment of 2048 tokens or more), where it has always worked."""
        if self.repeats and (sum(self._passes()) * ((features + TILE_M - 1) // TILE_M) >= 96
                             or max(e - s for a, s, e in self.segments if a >= 0) < 2048):
            raise ValueError("an adapter may own only one token segment per microbatch")
        return list(self._rows().split(self._passes()))

    def chunks(self, features: int) -> int:
        """In how many chunks the tokens of a segment are summed."""
        c = self._cache.get(features)
        if c is None:
            rows = segment_rows(self.segments)
            tiles = len(rows) * ((features + TILE_M - 1) // TILE_M)
            c = reduction_split(tiles, (rows[0][2] - rows[0][1] + 63) // 64) if rows else 1
            self._cache[features] = c
        return c


def _by_occurrence(segments) -> list:
    """``(adapter, start, end, 0)`` of every segment that has an adapter and tokens, in lists that name an adapter once:
    the adapters' first segments, their second ones, ...  A list starts with its longest: its tiles start first, and the
    short ones fill the gaps at the end."""
    groups, count = [], {}
    for a, s, e in segments:
        if a >= 0 and e > s:
            k = count[a] = count.get(a, -1) + 1
            if k == len(groups):
                groups.append([])
            groups[k].append((a, s, e, 0))
    for g in groups:
        g.sort(key=lambda r: r[1] - r[2])
    return groups


def segment_rows(segments) -> list:
    """:func:`_by_occurrence` as one list."""
    return [r for g in _by_occurrence(segments) for r in g]


def _flat2d(t: torch.Tensor) -> torch.Tensor:
    return t.reshape(-1, t.shape[-1])


def _rows_split(rows: int, k: int) -> int:
    return reduction_split((rows + TILE_M - 1) // TILE_M, (k + 63) // 64)


def lora_down(x: torch.Tensor, a_all: torch.Tensor, *, tile_adapter: Optional[torch.Tensor],
              adapter_scale: Optional[torch.Tensor], scale: float = 1.0,
              dropout: DropoutSpec = NO_DROPOUT, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``S'[M, R] = alpha_a * dropout(x)[M, K] @ A_a[R, K]^T`` with the adapter of each tile."""
    M, K = x.shape
    n, R, K2 = a_all.shape
    assert K2 == K and R in RANK_PADS
    if out is None:
        out = torch.empty((M, R), dtype=torch.bfloat16, device=x.device)
    launch_skinny(_rows_split(M, K), a=x, b=_flat2d(a_all), out=out, M=M, N=R, K=K, bn=R,
                  epi=nv.EPI_BF16_ADAPTER_SCALE, mask_a=dropout.active,
                  tile_adapter=tile_adapter, b_adapter_rows=R, adapter_scale=adapter_scale,
                  scale=scale, **dropout.kwargs())
    return out


def base_lora_fwd(x: torch.Tensor, w: torch.Tensor, s: Optional[torch.Tensor],
                  b_all: Optional[torch.Tensor], *, tile_adapter: Optional[torch.Tensor],
                  bias: Optional[torch.Tensor] = None,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``Y[M, N] = x[M, K] @ w[N, K]^T + S'[M, R] @ B_a[N, R]^T (+ bias)``."""
    M, K = x.shape
    N = w.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=torch.bfloat16, device=x.device)
    kw = {}
    if s is not None:
        n, N2, R = b_all.shape
        assert N2 == N and s.shape == (M, R)
        kw = dict(a2=s, b2=_flat2d(b_all), K2=R, b2_adapter_rows=N, tile_adapter=tile_adapter)
    launch_gemm(a=x, b=w, out=out, M=M, N=N, K=K, bn=256 if N >= 256 else 128, bias=bias, tuned="fwd", **kw)
    return out


def lora_ds(dy: torch.Tensor, b_all: torch.Tensor, *, tile_adapter: Optional[torch.Tensor],
            adapter_scale: Optional[torch.Tensor], scale: float = 1.0,
            out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``dS[M, R] = alpha_a * dy[M, N] @ B_a[N, R]``."""
    M, N = dy.shape
    n, N2, R = b_all.shape
    assert N2 == N and R in RANK_PADS
    if out is None:
        out = torch.empty((M, R), dtype=torch.bfloat16, device=dy.device)
    launch_skinny(_rows_split(M, N), a=dy, b=_flat2d(b_all), out=out, M=M, N=R, K=N, b_mn=True, bn=R,
                  epi=nv.EPI_BF16_ADAPTER_SCALE, tile_adapter=tile_adapter, b_adapter_rows=N,
                  adapter_scale=adapter_scale, scale=scale)
    return out


def lora_db(dy: torch.Tensor, s: torch.Tensor, segs: SegmentTable, db_all: torch.Tensor) -> None:
    """``dB_all[a][N, R] += dy[seg_a]^T @ S'[seg_a]`` (fp32, one owner CTA per element)."""
    M, N = dy.shape
    n, N2, R = db_all.shape
    assert N2 == N and s.shape == (M, R) and db_all.dtype == torch.float32
    for rows in segs.passes(N):
        if rows.shape[0] > 0:
            launch_skinny(segs.chunks(N), a=dy, b=s, out=db_all, M=N, N=R, K=M, a_mn=True, b_mn=True, bn=R,
                          epi=nv.EPI_F32_ACCUM, seg_tiles=rows, ldo=R, out_adapter_stride=N * R)


def lora_da(x: torch.Tensor, ds: torch.Tensor, segs: SegmentTable, da_all: torch.Tensor, *,
            dropout: DropoutSpec = NO_DROPOUT) -> None:
    """``dA_all[a][R, K] += dS[seg_a]^T @ dropout(x)[seg_a]`` (fp32)."""
    M, K = x.shape
    n, R, K2 = da_all.shape
    assert K2 == K and ds.shape == (M, R) and da_all.dtype == torch.float32
    for rows in segs.passes(K):
        if rows.shape[0] > 0:
            launch_skinny(segs.chunks(K), a=x, b=ds, out=da_all, M=K, N=R, K=M, a_mn=True, b_mn=True, bn=R,
                          epi=nv.EPI_F32_ACCUM, mask_a=dropout.active, seg_tiles=rows, ldo=K,
                          out_transposed=True, out_adapter_stride=R * K, **dropout.kwargs())


@dataclass
class OneAdapter:
    """Every token belongs to adapter 0: what the kernels need to know of a batch in that case,
    without any table on the device (:class:`~.batch_info.MultiLoRABatchInfo` is the general one)."""

    tokens: int
    scale: float
    p: float
    seed: int
    tile_adapter = None
    adapter_scale = None
    segment_table = None

    def __post_init__(self):
        dropout_threshold(self.p)   # refuses what is no rate

    @property
    def segments(self) -> list:
        return [(0, 0, self.tokens)]

    @property
    def alpha_by_adapter(self) -> dict:
        return {0: self.scale}

    @property
    def dropout_by_adapter(self) -> dict:
        return {0: self.p}

    def dropout_spec(self, stream_id: int, training: bool = True) -> DropoutSpec:
        return DropoutSpec(seed=self.seed, stream_id=stream_id, p=self.p) if training and self.p > 0 else NO_DROPOUT


def _matrix(t: torch.Tensor, name: str, rows: int, cols: int) -> tuple[int, int]:
    """Address and row pitch of a bf16 matrix ``[rows, cols]``.  (A layer looks at up to eight operands a call: the
    usual case is one comparison of each property.)"""
    ptr = t.data_ptr()
    if t.shape == (rows, cols) and t.dtype is torch.bfloat16:
        ld, unit = t.stride()
        if unit == 1 and not (2 * ld | ptr) & 15:
            return ptr, ld
    check2d(t, name)
    raise ValueError(f"{name} must have the shape {(rows, cols)}, got {tuple(t.shape)}")


def _stack(t: torch.Tensor, name: str, rows: int, cols: int) -> tuple[int, int, torch.Tensor]:
    """Address and row pitch of ``[n, rows, cols]`` adapters as the bf16 matrix ``[n * rows, cols]`` that the kernels
    read, and the tensor that holds it: a copy where the adapters do not lie one behind the other."""
    if t.dim() != 3 or t.shape != (t.shape[0], rows, cols):
        raise ValueError(f"{name} must have the shape [n, {rows}, {cols}], got {tuple(t.shape)}")
    if not t.is_contiguous() or t.dtype is not torch.bfloat16 or (2 * cols | t.data_ptr()) & 15:
        t = _flat2d(t)
        check2d(t, name)
        return t.data_ptr(), t.stride(0), t
    return t.data_ptr(), cols, t


def _grad_stack(t: Optional[torch.Tensor], name: str, rows: int, cols: int) -> Optional[int]:
    """Address of the fp32 gradient accumulators ``[n, rows, cols]`` of all adapters."""
    if t is None:
        return None
    if t.dim() != 3 or t.shape != (t.shape[0], rows, cols) or t.dtype is not torch.float32 or not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous fp32 [n, {rows}, {cols}], got {t.dtype} {tuple(t.shape)} "
                         f"strides {t.stride()}")
    return t.data_ptr()


def _linear_args(M: int, K: int, N: int, R: int, n: int, info, drop: DropoutSpec, device,
                 **fields) -> nv.LfLoraLinearArgs:
    """Describe one LoRA linear layer (``lf_lora_linear_fwd`` / ``_bwd``) for the current stream.  The operands come as
    addresses: the callers have checked them, since the kernels read and write what the sizes say."""
    if R not in RANK_PADS and not fields.get("have_s"):
        raise ValueError(f"adapter stacks must be {RANK_PADS} wide, got {R}")
    if "y" in fields:
        cfg = get_kernel_config("fwd", M, K, N)
        fields.update(fwd_group_m=cfg.group_m, fwd_max_ctas=cfg.max_ctas)
    else:
        cfg = get_kernel_config("dx_dropout" if drop.active else "dx", M, N, K)
        fields.update(dx_group_m=cfg.group_m, dx_max_ctas=cfg.max_ctas)
    args = nv.LfLoraLinearArgs(
        err=nv.err_word(device).data_ptr(), stream=nv.current_stream_ptr(), M=M, K=K, N=N, R=R, n_adapters=n,
        dropmix_bn=DROPMIX_BN, scale=getattr(info, "scale", 1.0), **fields)
    if info.tile_adapter is not None:
        args.tile_adapter = info.tile_adapter.data_ptr()
    if info.adapter_scale is not None:
        args.adapter_scale = info.adapter_scale.data_ptr()
    if drop.active:
        args.dropout = 1
        args.thresh16 = dropout_threshold(drop.p)
        args.inv_keep = 1.0 / (1.0 - drop.p) if drop.p > 0 else 1.0
        if drop.adapter_thresh16 is not None:
            args.adapter_thresh16 = drop.adapter_thresh16.data_ptr()
            args.adapter_inv_keep = drop.adapter_inv_keep.data_ptr()
        args.seed_lo, args.seed_hi = drop.seed & 0xFFFFFFFF, (drop.seed >> 32) & 0xFFFFFFFF
        args.stream_id = drop.stream_id & 0xFFFFFFFF
        args.row_offset, args.col_offset = drop.row_offset, drop.col_offset
    return args


def _pair_setup(args: nv.LfLoraLinearArgs, M: int, N: int, K: int, max_ctas: int, device) -> Optional[torch.Tensor]:
    """Route the layer's big product (256-wide tiles) and give it the scratch it wants."""
    if N < 256 or not use_pair(M, N, K, max_ctas, device):
        return None
    args.pair = 1
    scratch = pair_scratch(M, N, K, max_ctas, device)
    if scratch is not None:
        args.scratch, args.scratch_bytes = scratch.data_ptr(), scratch.numel()
    return scratch


def linear_fwd(x: torch.Tensor, w: torch.Tensor, a_all: Optional[torch.Tensor], b_all: torch.Tensor, info,
               drop: DropoutSpec, bias: Optional[torch.Tensor] = None, s: Optional[torch.Tensor] = None):
    """``lora_down`` and ``base_lora_fwd`` in one call: ``(y, s)``.  With ``s`` given, ``a_all`` is not read."""
    M, K = x.shape
    n, N, R = b_all.shape
    have_s = s is not None
    x_ptr, x_ld = _matrix(x, "x", M, K)
    w_ptr, w_ld = _matrix(w, "w", N, K)
    b_ptr, b_ld, b_all = _stack(b_all, "B", N, R)
    a_ptr, a_ld = None, 0
    if have_s:
        s_ptr, s_ld = _matrix(s, "S'", M, R)
    else:
        n = min(n, a_all.shape[0])
        a_ptr, a_ld, a_all = _stack(a_all, "A", R, K)
        s = x.new_empty(M, R)
        s_ptr, s_ld = s.data_ptr(), R
    y = x.new_empty(M, N)
    args = _linear_args(M, K, N, R, n, info, drop, x.device, y=y.data_ptr(), have_s=int(have_s), x=x_ptr, x_ld=x_ld,
                        w=w_ptr, w_ld=w_ld, a_all=a_ptr, a_ld=a_ld, b_all=b_ptr, b_ld=b_ld, s=s_ptr, s_ld=s_ld,
                        bias=None if bias is None else bias.data_ptr(), split_s=_rows_split(M, K))
    scratch = _pair_setup(args, M, N, K, args.fwd_max_ctas, x.device)
    nv.note_launch(1 if have_s else 2)
    rc = nv.cuda_lib().lf_lora_linear_fwd(C.byref(args))
    if rc != 0:
        raise RuntimeError(f"lf_lora_linear_fwd failed with code {rc}")
    del scratch   # back to the allocator, in stream order, once the launch is queued
    return y, s


def linear_bwd(dy: torch.Tensor, x: Optional[torch.Tensor], s: Optional[torch.Tensor], w: Optional[torch.Tensor],
               a_all: Optional[torch.Tensor], b_all: torch.Tensor, info, drop: DropoutSpec, da: Optional[torch.Tensor],
               db: Optional[torch.Tensor], need_dx: bool) -> Optional[torch.Tensor]:
    """``lora_ds``, ``lora_db`` into ``db``, ``lora_da`` into ``da`` and ``base_lora_dx`` in one call.  ``x`` is read
    for ``da``, ``s`` for ``db``, ``w`` and ``a_all`` for dX."""
    n, N, R = b_all.shape
    M = dy.shape[0]
    K = w.shape[1] if need_dx else (0 if da is None else x.shape[1])
    dy_ptr, dy_ld = _matrix(dy, "dy", M, N)
    b_ptr, b_ld, b_all = _stack(b_all, "B", N, R)
    da_ptr, db_ptr = _grad_stack(da, "dA", R, K), _grad_stack(db, "dB", N, R)
    x_ptr, x_ld = (None, 0) if da is None else _matrix(x, "x", M, K)
    s_ptr, s_ld = (None, 0) if db is None else _matrix(s, "S'", M, R)
    ds = dy.new_empty(M, R)
    dx = dx_ptr = w_ptr = a_ptr = None
    w_ld = a_ld = 0
    if need_dx:
        n = min(n, a_all.shape[0])
        w_ptr, w_ld = _matrix(w, "w", N, K)
        a_ptr, a_ld, a_all = _stack(a_all, "A", R, K)
        dx = dy.new_empty(M, K)
        dx_ptr = dx.data_ptr()
    if da is None and db is None:
        seg_rows, num_segs, split_da, split_db = None, 0, 1, 1
    elif info.segment_table is None:
        seg_rows, num_segs = None, 1
        split_da, split_db = (reduction_split((f + TILE_M - 1) // TILE_M, (M + 63) // 64) for f in (K, N))
    else:
        rows = info.segment_table.device_rows()
        seg_rows, num_segs = rows.data_ptr(), rows.shape[0]
        split_da, split_db = info.segment_table.chunks(K), info.segment_table.chunks(N)
    args = _linear_args(M, K, N, R, n, info, drop, dy.device, dy=dy_ptr, dy_ld=dy_ld, ds=ds.data_ptr(), x=x_ptr,
                        x_ld=x_ld, s=s_ptr, s_ld=s_ld, w=w_ptr, w_ld=w_ld, a_all=a_ptr, a_ld=a_ld, b_all=b_ptr,
                        b_ld=b_ld, dx=dx_ptr, da=da_ptr, db=db_ptr, seg_rows=seg_rows, num_segs=num_segs,
                        split_ds=_rows_split(M, N), split_db=split_db, split_da=split_da)
    scratch = _pair_setup(args, M, K, N, args.dx_max_ctas, dy.device) if need_dx else None
    nv.note_launch(1 + (da is not None) + (db is not None) + need_dx)
    rc = nv.cuda_lib().lf_lora_linear_bwd(C.byref(args))
    if rc != 0:
        raise RuntimeError(f"lf_lora_linear_bwd failed with code {rc}")
    del scratch
    return dx


def _pieces(entries: Sequence[tuple]):
    """C array of ``(a, b, r)`` adapter entries (tensors or ``None``)."""
    arr = (nv.LfLoraPiece * len(entries))()
    for e, (a, b, r) in zip(arr, entries):
        if a is not None:
            e.a, e.a_ld = a.data_ptr(), a.stride(0)
        if b is not None:
            e.b, e.b_ld = b.data_ptr(), b.stride(0)
        e.r = r
    return arr


def pack_stacks(entries: Sequence[tuple], K: int, N: int, R: int, device):
    """``(A, B, r)`` per adapter (bf16 ``[r, K]`` / ``[N, r]`` with a contiguous last dimension, or
    ``(None, None, 0)``) -> zero-padded stacks ``[n, R, K]``, ``[n, N, R]``."""
    n = len(entries)
    flat = torch.empty(n * R * (K + N), dtype=torch.bfloat16, device=device)
    a_all, b_all = flat[:n * R * K].view(n, R, K), flat[n * R * K:].view(n, N, R)
    nv.call("lf_lora_pack", C.addressof(arr := _pieces(entries)), n, a_all.data_ptr(), b_all.data_ptr(), R, K, N,
            nv.current_stream_ptr())
    del arr
    return a_all, b_all


def unpack_grads(entries: Sequence[tuple], da: Optional[torch.Tensor], db: Optional[torch.Tensor], K: int, N: int,
                 R: int) -> None:
    """fp32 gradient stacks -> the bf16 tensors of ``entries`` (contiguous ``[r, K]`` / ``[N, r]``)."""
    nv.call("lf_lora_unpack", C.addressof(arr := _pieces(entries)), len(entries),
            None if da is None else da.data_ptr(), None if db is None else db.data_ptr(), R, K, N,
            nv.current_stream_ptr())
    del arr


def base_lora_dx(dy: torch.Tensor, w: torch.Tensor, ds: Optional[torch.Tensor],
                 a_all: Optional[torch.Tensor], *, tile_adapter: Optional[torch.Tensor],
                 dropout: DropoutSpec = NO_DROPOUT,
                 out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``dX[M, K] = dy[M, N] @ w[N, K] + keep (.) (dS[M, R] @ A_a[R, K]) / (1 - p)``."""
    M, N = dy.shape
    K = w.shape[1]
    if out is None:
        out = torch.empty((M, K), dtype=torch.bfloat16, device=dy.device)
    kw = {}
    if ds is not None:
        n, R, K2 = a_all.shape
        assert K2 == K and ds.shape == (M, R)
        kw = dict(a2=ds, b2=_flat2d(a_all), K2=R, b2_adapter_rows=R, tile_adapter=tile_adapter)
    if ds is not None and dropout.active:
        launch_gemm(a=dy, b=w, out=out, M=M, N=K, K=N, b_mn=True, b2_mn=True,
                    bn=DROPMIX_BN if K >= 256 else 128, nacc=2,
                    epi=nv.EPI_BF16_DROPMIX, tuned="dx_dropout", **kw, **dropout.kwargs())
    else:
        launch_gemm(a=dy, b=w, out=out, M=M, N=K, K=N, b_mn=True, b2_mn=True,
                    bn=256 if K >= 256 else 128, tuned="dx", **kw)
    return out
