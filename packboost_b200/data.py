"""Binning and bit-packing of features for the B200 backend.

Host-facing names follow the reference's data utilities
(``packboost/data.py``): ``BinningResult``, ``detect_prebinned``,
``quantile_bin``, ``preprocess_features``, ``apply_bins``, ``build_era_index``.
The code assignment (``searchsorted`` against the per-feature edges) and the
packing into 4-bit / 8-bit lanes run on the device; the quantile edges
themselves are order statistics interpolated in float64 by ``np.quantile``,
exactly as the reference computes them, so that bin codes are bit-identical.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Iterable, Sequence

import numpy as np
import torch

from . import backends as B


@dataclass(slots=True)
class BinningResult:
    """Preprocessed training data (``packboost/data.py:12-18``).  ``bins`` is only
    materialised on request; training keeps the packed device matrix instead."""

    bins: np.ndarray | None
    bin_edges: np.ndarray | None
    prebinned: bool


def ensure_numpy(array) -> np.ndarray:
    if isinstance(array, np.ndarray):
        return array
    if isinstance(array, torch.Tensor):
        return array.detach().cpu().numpy()
    return np.asarray(array)


def detect_prebinned(X: np.ndarray, max_bins: int) -> bool:
    """Integer input whose values already are bin ids (``packboost/data.py:32-42``)."""
    if not np.issubdtype(X.dtype, np.integer):
        return False
    if X.size and X.min() < 0:
        return False
    top = int(X.max()) if X.size else 0
    if top >= max_bins:
        return False
    return top <= 127


def detect_prebinned_tensor(X: torch.Tensor, max_bins: int) -> bool:
    """:func:`detect_prebinned` of a tensor where it is: only an integer table is looked at, and only
    its smallest and largest value leave the device."""
    if X.is_floating_point() or X.is_complex() or X.dtype == torch.bool:
        return False
    if X.numel() == 0:
        return max_bins > 0
    if X.dtype in (torch.uint16, torch.uint32, torch.uint64):   # (torch has no minimum of these)
        X = X.to(torch.int32 if X.dtype == torch.uint16 else torch.int64)
    low, top = (int(v) for v in torch.stack(torch.aminmax(X)).tolist())
    return low >= 0 and top < max_bins and top <= 127


def sort_eras(era: np.ndarray | None, n_rows: int) -> tuple[np.ndarray, np.ndarray, np.ndarray | None]:
    """``(era ids ascending, offsets of their row ranges, row order)`` of the rows grouped by era;
    the order is ``None`` when the rows are grouped already.  The runs of equal ids give the ids and
    the offsets, so rows that come in ascending order cost one comparison pass."""
    if era is None:
        return np.array([0], dtype=np.int16), np.array([0, n_rows], dtype=np.int32), None
    order = None
    for attempt in range(2):
        starts = np.flatnonzero(era[1:] != era[:-1]) + 1
        starts = np.concatenate([[0], starts]) if n_rows else starts
        uniq = era[starts]
        if np.all(uniq[1:] > uniq[:-1]):
            break
        order = np.argsort(era, kind="stable")
        era = era[order]
    return uniq, np.concatenate([starts, [n_rows]]).astype(np.int32), order


def quantile_edges(X: np.ndarray, max_bins: int) -> np.ndarray:
    """``[max_bins-1, F]`` float32 edges at the interior quantiles (``packboost/data.py:49-50``)."""
    q = np.linspace(0.0, 1.0, max_bins + 1, dtype=np.float64)[1:-1]
    return np.quantile(X, q, axis=0, method="linear").astype(np.float32)


def edges_from_sorted(sorted_cols: torch.Tensor, max_bins: int) -> np.ndarray:
    """Interior quantile edges of columns that are already sorted ascending (NaN last), with the
    arithmetic of ``np.quantile(..., method="linear")`` step for step: virtual index
    ``(n - 1) * q`` in float64, the two neighbours taken from the float32 column, their float32
    difference, then ``a + d * t`` (``b - d * (1 - t)`` where ``t >= 0.5``) in float64.  A column
    that holds a NaN gets NaN edges.  Only the two gathers touch the big array; the interpolation
    runs on the host on ``2 * (max_bins - 1) * F`` numbers.  ``float64 [max_bins - 1, F]``."""
    n = int(sorted_cols.shape[0])
    q = np.linspace(0.0, 1.0, max_bins + 1, dtype=np.float64)[1:-1]
    virtual = (n - 1) * q
    prev = np.floor(virtual).astype(np.int64)
    nxt = prev + 1
    above = virtual >= n - 1
    prev[above] = n - 1
    nxt[above] = n - 1
    below = virtual < 0
    prev[below] = 0
    nxt[below] = 0
    dev = sorted_cols.device
    a = sorted_cols[torch.from_numpy(prev).to(dev)].cpu().numpy()
    b = sorted_cols[torch.from_numpy(nxt).to(dev)].cpu().numpy()
    has_nan = torch.isnan(sorted_cols[-1]).cpu().numpy()
    t = (virtual - prev).reshape(-1, 1)
    d = np.subtract(b, a)                      # float32, as in numpy's _lerp
    with np.errstate(invalid="ignore"):
        out = np.add(a, d * t)
        np.subtract(b, d * (1 - t), out=out, where=np.broadcast_to(t >= 0.5, out.shape))
    out[:, has_nan] = np.nan
    return out


def quantile_edges_device(X: np.ndarray | torch.Tensor, max_bins: int) -> np.ndarray:
    """``quantile_edges`` with the sort on the GPU (a column sort of 500 000 x 256 floats takes
    seconds on the host and milliseconds on the device); same result bit for bit up to the sign
    of a zero.  ``X``: float32 ``[N, F]``, host array or tensor on either side."""
    dev = _device()
    n, f = X.shape
    uploads = Uploads()
    # Fewer than 128 columns per sort, in even shares of at most 256 MB: a sort of that many segments
    # goes over all keys at once (500 000 rows: 29 us a column), one of more sorts segment by segment (46).
    most = max(1, min(127, (256 << 20) // max(4 * n, 1)))
    cols = max(1, -(-f // -(-f // most)))
    out = np.empty((max_bins - 1, f), dtype=np.float64)
    for c0 in range(0, f, cols):
        c1 = min(f, c0 + cols)
        if isinstance(X, torch.Tensor) and X.is_cuda:
            block = X[:, c0:c1].to(device=dev, dtype=torch.float32)
        else:
            block = uploads(X[:, c0:c1], torch.float32)
        # (columns made rows first: the sort then copies nothing in or out)
        out[:, c0:c1] = edges_from_sorted(torch.sort(block.t().contiguous(), dim=1).values.t(), max_bins)
    return out.astype(np.float32)


def code_bits_for(max_bins: int) -> int:
    return 4 if max_bins <= 16 else 8


def _device() -> torch.device:
    if not B.cuda_available():
        raise RuntimeError("packboost_b200 needs its CUDA library and a B200-class device; there is no CPU path")
    return torch.device("cuda", torch.cuda.current_device())


_CHUNK_BYTES = 256 << 20


def _row_chunks(n_rows: int, row_bytes: int, chunk_bytes: int = _CHUNK_BYTES) -> Iterable[tuple[int, int]]:
    step = max(256, (chunk_bytes // max(row_bytes, 1)) // 256 * 256)
    for a in range(0, n_rows, step):
        yield a, min(n_rows, a + step)


class PackedMatrix:
    """Feature-major packed bin codes on the device (layout of ``pb_train_state.codes``)."""

    def __init__(self, n_rows: int, n_features_local: int, code_bits: int, device: torch.device,
                 pitch: int | None = None, zero: bool = True):
        self.n_rows = int(n_rows)
        self.rows_padded = (self.n_rows + 255) // 256 * 256
        self.code_bits = int(code_bits)
        self.pitch = (self.rows_padded * code_bits // 8 + 127) // 128 * 128
        if pitch is not None:
            if pitch % 128 or pitch < self.pitch:
                raise ValueError("pitch must be a multiple of 128 that covers the padded rows")
            self.pitch = int(pitch)
        self.n_features_local = int(n_features_local)
        self.max_code = 0   # largest pre-binned code seen while packing (when validation was asked for)
        make = torch.zeros if zero else torch.empty
        self.codes = make((max(self.n_features_local, 1), self.pitch), dtype=torch.uint8, device=device)

    def unpack(self) -> torch.Tensor:
        """``uint8 [F_local, n_rows]`` (tests and the legacy feature-major predictors)."""
        if self.code_bits == 8:
            return self.codes[: self.n_features_local, : self.n_rows].contiguous()
        lo = self.codes & 0xF
        hi = self.codes >> 4
        full = torch.stack([lo, hi], dim=2).reshape(self.codes.shape[0], -1)
        return full[: self.n_features_local, : self.n_rows].contiguous()


class Uploads:
    """Host arrays on their way to the device.  Page-locked tensors go to the copy engine as they are,
    everything else through a page-locked ring filled by the library's copy threads.  The rings stay
    with this object, which has to live until the current stream has passed the copies."""

    def __init__(self) -> None:
        self._rings: list[torch.Tensor] = []

    def __call__(self, host, dtype: torch.dtype, out: torch.Tensor | None = None) -> torch.Tensor:
        """Device copy of a host array or tensor, converted to ``dtype`` on the host where it differs."""
        if isinstance(host, torch.Tensor):
            src = host if host.dtype == dtype else host.to(dtype)
            if src.is_pinned() and src.is_contiguous():
                dev = torch.empty(src.shape, dtype=dtype, device=_device()) if out is None else out
                return dev.copy_(src, non_blocking=True)
            src = src.contiguous()
            shape, at, nbytes = src.shape, src.data_ptr(), src.numel() * src.element_size()
        else:
            src = np.ascontiguousarray(host, dtype=_NUMPY_OF[dtype])
            shape, at, nbytes = src.shape, src.ctypes.data, src.nbytes
        dev = torch.empty(shape, dtype=dtype, device=_device()) if out is None else out
        need = int(B.lib().pb_upload_ring_bytes(nbytes))
        ring = next((r for r in self._rings if r.numel() >= need), None)
        if ring is not None:
            torch.cuda.current_stream().synchronize()   # (the ring's last user)
        else:
            ring = torch.empty(max(need, 1), dtype=torch.uint8, pin_memory=True)
            self._rings.append(ring)
        B.check(B.lib().pb_upload(dev.data_ptr(), at, nbytes, ring.data_ptr(), ring.numel(),
                                  torch.cuda.current_stream().cuda_stream))
        return dev


_NUMPY_OF = {torch.float32: np.float32, torch.uint8: np.uint8, torch.int32: np.int32}


def fits_on_device(nbytes: int) -> bool:
    """Whether to try bringing a whole table to the device for a while: when it is small next to the device
    (asking for the free memory costs 0.1 ms and, now and then, tens of them), else up to a third of what is
    free.  The caller goes on without when there is no room after all."""
    dev = _device()
    if nbytes <= torch.cuda.get_device_properties(dev).total_memory // 64:
        return True
    return nbytes <= torch.cuda.mem_get_info(dev)[0] // 3


def pack_feature_major(
    X: np.ndarray | torch.Tensor,
    edges: np.ndarray | None,
    max_bins: int,
    *,
    row_order: np.ndarray | None = None,
    feature_map: np.ndarray | None = None,
    n_features_local: int | None = None,
    validate_codes: bool = False,
    rows: tuple[int, int] | None = None,
    out: "PackedMatrix | None" = None,
    defer_validation: bool = False,
) -> PackedMatrix:
    """Bin (when ``edges`` is given) and pack host or device data into a device ``PackedMatrix``.

    ``row_order`` lists source rows in destination order (era-sorted rows);
    ``feature_map[j]`` is the destination feature row of column ``j`` or -1.
    ``rows=(r0, r1)`` packs only that range of destination rows, into rows ``0 .. r1 - r0`` of
    ``out`` (one rank's share when several GPUs split the upload).  ``out`` packs into an existing
    matrix.  ``validate_codes`` checks on the device that pre-binned input stays below ``max_bins``
    (negative int8 values show up as codes >= 128) and raises ``ValueError`` otherwise; with
    ``defer_validation`` the largest code seen is only recorded in ``PackedMatrix.max_code`` (several
    ranks must agree before any of them raises).

    A device table of the right type is packed in one launch, rows in any order.  Host input reaches
    the device in pieces (see :class:`Uploads`): the copy of piece ``i + 1`` overlaps the packing of
    piece ``i``.
    """
    dev = _device()
    lib = B.lib()
    n_rows, n_feat = X.shape
    bits = code_bits_for(max_bins)
    r0, r1 = (0, n_rows) if rows is None else (int(rows[0]), int(rows[1]))
    n_local = n_feat if n_features_local is None else n_features_local
    # (the pack kernels write the padding of every row they write: only rows nobody writes need zeros)
    pm = out if out is not None else PackedMatrix(r1 - r0, n_local, bits, dev,
                                                  zero=feature_map is not None or n_local != n_feat or r1 <= r0)
    if r1 <= r0:
        return pm
    fmap_t = None
    if feature_map is not None:
        fmap_t = torch.from_numpy(np.ascontiguousarray(feature_map, dtype=np.int32)).to(dev)
    is_f32 = edges is not None
    edges_t = None
    if is_f32:
        edges_t = edges if isinstance(edges, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(edges, dtype=np.float32))
        edges_t = edges_t.to(dev)
    stream = torch.cuda.current_stream().cuda_stream
    want = torch.float32 if is_f32 else torch.uint8
    top = torch.zeros(1, dtype=torch.int32, device=dev) if validate_codes and not is_f32 else None

    def pack(chunk, n, at, order=None):
        B.check(lib.pb_pack_table(chunk.data_ptr(), 1 if is_f32 else 0, B._ptr(order), n, n_feat, at, B._ptr(edges_t),
                                  edges_t.shape[0] if is_f32 else 0, max_bins if is_f32 else (16 if bits == 4 else 256),
                                  B._ptr(fmap_t), pm.codes.data_ptr(), pm.pitch, bits, B._ptr(top), stream))

    def as_codes(src):
        """int8 is read as the bytes it is: negative values fail the range check."""
        if is_f32:
            return src
        if isinstance(src, torch.Tensor):
            return src.view(torch.uint8) if src.dtype == torch.int8 else src
        return src.view(np.uint8) if src.dtype == np.int8 else src

    uploads = Uploads()
    if isinstance(X, torch.Tensor) and X.device == dev and as_codes(X).dtype == want and X.is_contiguous():
        if row_order is None:
            pack(as_codes(X[r0:r1]), r1 - r0, 0)
        else:
            order = np.ascontiguousarray(row_order[r0:r1], dtype=np.int32)
            pack(as_codes(X), r1 - r0, 0, torch.from_numpy(order).to(dev))
    else:
        order_t = None
        if row_order is not None and isinstance(X, torch.Tensor):
            order_t = torch.from_numpy(np.ascontiguousarray(row_order, dtype=np.int64)).to(X.device)
        for a, b in _row_chunks(r1 - r0, n_feat * (4 if is_f32 else 1)):
            if order_t is not None:
                src = X.index_select(0, order_t[r0 + a:r0 + b])
            else:
                src = X[r0 + a:r0 + b] if row_order is None else X[row_order[r0 + a:r0 + b]]
            src = as_codes(src)
            if isinstance(src, torch.Tensor) and src.is_cuda:
                chunk = src.to(device=dev, dtype=want).contiguous()
            else:
                chunk = uploads(src, want)
            pack(chunk, b - a, a)
            # no synchronisation per chunk: the copy, the pack kernel and the release of `chunk` are
            # ordered on the current stream
    if top is not None:
        pm.max_code = max(pm.max_code, int(top.item()))
    else:
        torch.cuda.current_stream().synchronize()
    if validate_codes and not defer_validation and pm.max_code >= min(max_bins, 128):
        raise ValueError("prebinned=True requires X to contain integer bins within [0, max_bins).")
    return pm


def rows_per_rank(n_rows: int, world: int) -> int:
    """Rows each rank packs when the upload is split by rows: equal shares rounded up to 256 rows
    (128 bytes of 4-bit codes), so that every rank's bytes of a feature row are a whole, aligned
    segment of it."""
    per = (n_rows + world - 1) // max(world, 1)
    return (per + 255) // 256 * 256


def pack_feature_major_distributed(X, edges, max_bins, *, row_order, rank: int, world: int, n_features: int,
                                   keep: tuple[int, int] | None, validate_codes: bool = False) -> PackedMatrix:
    """Pack the matrix with ``world`` GPUs sharing the host -> device transfer.

    Rank ``r`` brings over and packs only rows ``[r * R, (r + 1) * R)`` (``R = rows_per_rank``): a
    contiguous piece of the caller's row-major matrix, 1 / world of the bytes, at the full speed of
    its own host link.  The packed pieces are then exchanged between the GPUs (NVLink): with
    ``keep=None`` every rank ends up with the whole feature-major matrix (all-gather), with
    ``keep=(c0, c1)`` with all rows of its own features ``c0 .. c1`` only (all-to-all; every rank
    owns a block of ``ceil(F / world)`` features).  The result is laid out exactly like the matrix a
    single GPU would pack, with ``pitch = world * R * code_bits / 8``."""
    import torch.distributed as dist
    dev = _device()
    n_rows = X.shape[0]
    bits = code_bits_for(max_bins)
    per = rows_per_rank(n_rows, world)
    seg = per * bits // 8                                   # bytes of one feature row per rank (multiple of 128)
    blk = (n_features + world - 1) // world
    f_pad = blk * world
    slab = PackedMatrix(per, f_pad, bits, dev)
    assert slab.pitch == seg
    r0, r1 = min(n_rows, rank * per), min(n_rows, (rank + 1) * per)
    pack_feature_major(X, edges, max_bins, row_order=row_order, validate_codes=validate_codes, rows=(r0, r1), out=slab,
                       defer_validation=True)
    if keep is None:
        full = PackedMatrix(n_rows, f_pad, bits, dev, pitch=world * seg)
        parts = torch.empty((world, f_pad, seg), dtype=torch.uint8, device=dev)
        dist.all_gather_into_tensor(parts, slab.codes)
        full.codes.view(f_pad, world, seg).copy_(parts.permute(1, 0, 2))
        full.n_features_local = n_features
    else:
        full = PackedMatrix(n_rows, blk, bits, dev, pitch=world * seg)
        parts = torch.empty((world, blk, seg), dtype=torch.uint8, device=dev)
        dist.all_to_all_single(parts, slab.codes.view(world, blk, seg))
        full.codes.view(blk, world, seg).copy_(parts.permute(1, 0, 2))
        full.n_features_local = keep[1] - keep[0]
    full.max_code = slab.max_code
    return full


class PackedRows:
    """Row-major packed codes on the device (input layout of ``pb_predict_rows``)."""

    def __init__(self, n_rows: int, n_features: int, code_bits: int, device: torch.device):
        self.n_rows = int(n_rows)
        self.n_features = int(n_features)
        self.code_bits = int(code_bits)
        need = (n_features + 1) // 2 if code_bits == 4 else n_features
        self.pitch_row = (need + 15) // 16 * 16
        self.codes = torch.empty((max(self.n_rows, 1), self.pitch_row), dtype=torch.uint8, device=device)


def pack_row_major(X: np.ndarray | torch.Tensor, edges: np.ndarray | torch.Tensor | None, max_bins: int, *,
                   top: torch.Tensor | None = None, uploads: Uploads | None = None) -> PackedRows:
    """Bin (when ``edges`` is given) and pack rows for prediction.  ``X`` may already be a
    device tensor (float32 or uint8); edges too.  ``top`` (``int32 [1]`` on the device) takes the largest
    byte of pre-binned input.  With ``uploads`` the call only enqueues and the caller synchronises
    before it lets that object go."""
    dev = _device()
    lib = B.lib()
    bits = code_bits_for(max_bins)
    is_f32 = edges is not None
    n_rows, n_feat = X.shape
    pr = PackedRows(n_rows, n_feat, bits, dev)
    edges_t = None
    if is_f32:
        edges_t = edges if isinstance(edges, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(edges, dtype=np.float32))
        edges_t = edges_t.to(dev)
    stream = torch.cuda.current_stream().cuda_stream
    want = torch.float32 if is_f32 else torch.uint8
    up = Uploads() if uploads is None else uploads
    whole = isinstance(X, torch.Tensor) and X.device == dev and X.dtype == want and X.is_contiguous()
    for a, b in ([(0, n_rows)] if whole else _row_chunks(n_rows, n_feat * (4 if is_f32 else 1))):
        chunk = X[a:b]
        if not whole:
            on_gpu = isinstance(chunk, torch.Tensor) and chunk.is_cuda
            chunk = chunk.to(device=dev, dtype=want).contiguous() if on_gpu else up(chunk, want)
        B.check(lib.pb_pack_rows_top(chunk.data_ptr(), 1 if is_f32 else 0, b - a, n_feat, B._ptr(edges_t),
                                     edges_t.shape[0] if is_f32 else 0, max_bins, pr.codes[a:b].data_ptr(), pr.pitch_row,
                                     bits, B._ptr(top), stream))
    if uploads is None:
        torch.cuda.current_stream().synchronize()
    return pr


# ---- reference-named host helpers ------------------------------------------------------------


def quantile_bin(X: np.ndarray, max_bins: int) -> tuple[np.ndarray, np.ndarray]:
    """Quantile-bin ``X`` column-wise (``packboost/data.py:45-58``): ``(int8 codes [N,F], edges)``."""
    if max_bins > 128:
        raise ValueError("PackBoost currently supports up to 128 bins (int8 storage)")
    Xf = np.ascontiguousarray(X, dtype=np.float32)
    edges = quantile_edges(Xf, max_bins)
    pm = pack_feature_major(Xf, edges, max_bins)
    bins = pm.unpack().t().contiguous().cpu().numpy().astype(np.int8)
    return bins, edges


def preprocess_features(X: np.ndarray, max_bins: int, *, assume_prebinned: bool = False) -> BinningResult:
    """``packboost/data.py:61-93``; the returned ``bins`` are int8 ``[N, F]``."""
    X_np = ensure_numpy(X)
    if assume_prebinned and not detect_prebinned(X_np, max_bins):
        raise ValueError("prebinned=True requires X to contain integer bins within [0, max_bins).")
    if assume_prebinned or detect_prebinned(X_np, max_bins):
        return BinningResult(bins=X_np.astype(np.int8, copy=False), bin_edges=None, prebinned=True)
    bins, edges = quantile_bin(X_np.astype(np.float32, copy=False), max_bins=max_bins)
    return BinningResult(bins=bins, bin_edges=edges, prebinned=False)


def apply_bins(X: np.ndarray, bin_edges: np.ndarray | None, max_bins: int) -> np.ndarray:
    """Bin ``X`` with stored edges (``packboost/data.py:96-111``) -> int8 ``[N, F]``."""
    X_np = ensure_numpy(X)
    if bin_edges is None:
        if not detect_prebinned(X_np, max_bins):
            raise ValueError("Input must already be prebinned when no edges are provided")
        return X_np.astype(np.int8, copy=False)
    Xf = np.ascontiguousarray(X_np, dtype=np.float32)
    pm = pack_feature_major(Xf, bin_edges, max_bins)
    return pm.unpack().t().contiguous().cpu().numpy().astype(np.int8)


def build_era_index(era_ids: Iterable[int] | np.ndarray, num_eras: int | None) -> list[torch.Tensor]:
    """Per-era ascending row-id tensors (``packboost/data.py:114-134``)."""
    era_np = np.asarray(era_ids, dtype=np.int16)
    if era_np.ndim != 1:
        raise ValueError("era_ids must be 1D")
    if num_eras is None:
        num_eras = 1 if era_np.size == 0 else int(era_np.max()) + 1
    order = np.argsort(era_np, kind="stable")
    counts = np.bincount(era_np[era_np >= 0].astype(np.int64), minlength=int(num_eras))[: int(num_eras)]
    offs = np.concatenate([[0], np.cumsum(counts)])
    valid = order[era_np[order] >= 0]
    return [torch.from_numpy(valid[offs[e]:offs[e + 1]].astype(np.int64)) for e in range(int(num_eras))]
