"""Choice among the bfloat16 tensor-core matrix products.

  * up to 8 rows (small decode batches): the persistent TMA-ring streaming kernel (`gemm_stream.cu`) for large
    weights (gate/up, down, the output head), the weight-streaming mma.sync kernel (`gemm_smallm.cu`) for the
    smaller ones (q/k/v, o);
  * 9 to 16 rows: the streaming kernel at every shape;
  * more than 128 rows (prefill, mixed batches): the tcgen05 kernel on pairs of SMs (`gemm_pair.cu`), unless the output has few
    columns (`pair_config`);
  * the rows between (larger decode batches) and those few columns: the persistent tcgen05 kernel (`gemm_tc.cu`) with
    the tile width that fills whole waves of SMs (`tc_config`), cutting K into slices when the output has fewer
    tiles than the GPU has SMs; up to 128 rows and from three slices on, the slices are added inside a cluster
    (`cluster_config`).
The choice depends on the shape alone, so a token's logits do not depend on what else a process ran before.
Shapes all of them refuse (K not a multiple of 8, unaligned operands) go to the generic kernel.
"""
from __future__ import annotations

import ctypes
import functools
from typing import Optional

import torch

from . import build, ops

_UNSUPPORTED = 100001
SMALL_M = 64          # the most rows the weight-streaming kernel takes
SMALL_M_AUTO = 8      # up to here it is chosen (measured); above, the tcgen05 kernel with K slices streams better
_status = {}
_sm_count = {}


def status_flag(device: torch.device) -> torch.Tensor:
    """Device int32 that a timed-out wait inside a tensor-core kernel sets to 1."""
    key = device.index or 0
    if key not in _status:
        _status[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[key]


def check_status(device: torch.device) -> None:
    """Raises if a kernel recorded a timed-out wait (synchronises with the device)."""
    key = device.index or 0
    if key in _status and int(_status[key].item()) != 0:
        _status[key].zero_()
        raise RuntimeError("a tensor-core kernel gave up waiting on a barrier; its results are invalid")


def _sms(device: torch.device) -> int:
    key = device.index or 0
    if key not in _sm_count:
        _sm_count[key] = torch.cuda.get_device_properties(device).multi_processor_count
    return _sm_count[key]


def _ptr(t) -> int:
    return t.data_ptr()


def _stream() -> int:
    return ops._stream()


def _aligned(a, w) -> bool:
    return a.shape[1] % 8 == 0 and a.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0


_rt_override = 0      # tests and tuning runs may pin the row tiles per CTA


def row_tiles(M: int, N: int, device) -> int:
    """Row tiles of 16 per CTA for the small-M kernel.  One: measured fastest at every decode shape of the
    8B model (more, smaller CTAs per SM hide the latency of the weight loads better than fat ones)."""
    return _rt_override or 1


_tc_bn = 0            # tests and tuning runs may pin the tile width (a multiple of 16 up to 256) ...
_tc_splits = 0        # ... and the number of K slices of the tcgen05 kernel
TC_TILE_FIXED = 150   # a tile's fixed cost in columns: tiles of 128 measured 30-45 % slower per flop than tiles of 256


@functools.lru_cache(maxsize=4096)
def _tc_ragged_config(M: int, N: int, K: int, sms: int, swiglu: bool):
    """Tile width and K slices for two or more row tiles, by a model of the time in us that was fitted to 900 measured
    (shape, width, slices), 130 to 1,500 rows by the products of layers 2,048 and 4,096 wide (relative error 9 %): what it picks
    is 1.4 % slower than the best on average, "256 wide, or 128 wide with slices where the tiles do not fill the SMs" was 8 %.
    At 527 rows: 4,096 x 12,288 92 us with tiles of 256 (80 tiles on 148 SMs), 74 with 144 (145 tiles); 4,096 x 4,096 43 and
    36; at 300 rows 72 (128 wide) and 54 (256 wide, three slices)."""
    m_tiles, step = -(-M // 128), 32 if swiglu else 16
    k_blocks = -(-K // 64)
    best = None
    for bn in range(256, 63, -step):
        tiles = m_tiles * -(-N // bn)
        for splits in (1, 2, 3, 4, 6, 8):
            if splits > 1 and (tiles * splits > sms or k_blocks < 8 * splits or (swiglu and (N // 2) % (bn // 2))):
                break
            waves = -(-tiles * splits // sms)
            cost = waves * (k_blocks / splits * (0.198 + 0.000521 * bn) + 0.013 * bn)
            if splits > 1:
                cost += 1.5 + M * N * splits * 1.46e-6        # partial sums written and read, and the launch that adds them
            if best is None or cost < best[0]:
                best = (cost, bn, splits)
    return best[1:]


def tc_config(M: int, N: int, K: int, sms: int, swiglu: bool = False):
    """Tile width (a multiple of 16, of 32 with the SwiGLU epilogue) and number of K slices for the tcgen05 kernel.
    Very many tiles (prefill): the width, from 256 down to 192, whose tiles leave the least of the last wave of SMs
    empty, a tile costing its width plus a fixed part.  Several row tiles but few waves: `_tc_ragged_config`.  One row tile
    (decode batches): with the SwiGLU epilogue, and from 48 columns an SM on, the narrowest tile that needs one wave (no slices: the
    epilogue cannot run on partial sums without a second kernel; 64 rows by 20,544 x 4,096 39.6 us with 81 tiles of 256, 32.4 with
    143 of 144; from 64 columns an SM on where the rows of a are less than 128 KB together, which every tile reads and which come
    slower then: 24 rows by 8,256 x 2,048 15.0 us in one wave of tiles, 13.1 with slices, 32 rows 9.7 and 11.4); else 128- or 256-wide tiles with K cut into slices so that every SM streams a
    share of the weights.  (A finer cost model that also weighed wave tails chose more slices there and measured slower:
    the second kernel that adds the slices has a fixed cost.)"""
    m_tiles = -(-M // 128)
    step = 32 if swiglu else 16
    k_blocks = -(-K // 64)
    if not _tc_bn and m_tiles > 1 and m_tiles * -(-N // 256) < 8 * sms:
        bn, splits = _tc_ragged_config(M, N, K, sms, swiglu)
        return bn, min(_tc_splits, k_blocks) if _tc_splits else splits
    if _tc_bn:
        bn = _tc_bn
    elif m_tiles * -(-N // 256) >= sms:
        best = None
        for cand in range(256, 191, -step):
            waves = -(-(m_tiles * -(-N // cand)) // sms)
            cost = waves * (cand + TC_TILE_FIXED)
            if best is None or cost < best[0]:
                best = (cost, cand)
        bn = best[1]
    elif m_tiles == 1 and (swiglu or N > (48 if M * K >= 1 << 16 else 64) * sms) and N <= 256 * sms:
        bn = min(256, max(32 if swiglu else 64, -(-N // sms + step - 1) // step * step))       # the narrowest tile width that needs one wave
        while bn < 256 and -(-N // bn) > sms:
            bn += step
    else:
        bn = 256 if N >= 256 and m_tiles * -(-N // 256) >= sms // 2 else 128
    tiles = m_tiles * -(-N // bn)
    splits = 1
    if tiles < sms and not (swiglu and (N // 2) % (bn // 2)):
        splits = max(1, min(sms // tiles, k_blocks // 8))
    if _tc_splits:
        splits = min(_tc_splits, k_blocks)
    return bn, splits


STREAM_M = 32         # the most rows the persistent streaming kernel takes
STREAM_M_AUTO = 8     # up to here it is chosen ...
STREAM_MIN_WEIGHTS = 40 << 20    # ... for weights of at least this many elements (see `stream_wanted`)
STREAM_M_AUTO_WIDE = 16          # ... and up to here for weights of any size
_stream_rw = 0        # tests and tuning runs may pin the consumer warps across a tile's rows (8, 4, 2, 1)
_stream_ctas = 0      # tests may run fewer CTAs than SMs to move the places where CTAs hand a tile over
_stream_scratch = {}


STREAM_MAX_N = 1 << 20


def _stream_buffers(device: torch.device, lib):
    """Workspace for partial tiles and the per-tile arrival counters of the streaming kernel, sized once for
    the largest call it takes and never replaced (captured graphs keep their addresses).  One pair per device:
    the engine launches on one stream, and launches that do not overlap may share them."""
    key = device.index or 0
    if key not in _stream_scratch:
        if torch.cuda.is_current_stream_capturing():
            return None
        ws = torch.empty(int(lib.hk_gemm_stream_workspace(STREAM_M, 8)), dtype=torch.float32, device=device)
        ct = torch.zeros(STREAM_MAX_N // 16 + 2, dtype=torch.int32, device=device)
        _stream_scratch[key] = (ws, ct)
    return _stream_scratch[key]


def stream_row_warps(N: int, sms: int) -> int:
    """Consumer warps across a tile's rows (tile = 16 rows each): the widest tile that still gives every CTA a
    whole tile of its own, so that only the left-over tiles are shared between CTAs."""
    if _stream_rw:
        return _stream_rw
    for rw in (4, 2):
        if -(-N // (16 * rw)) >= sms:
            return rw
    return 1


def stream_wanted(M: int, N: int, K: int) -> bool:
    """The streaming kernel pays about two microseconds to fill its ring and to hand shared tiles over.  Measured
    on the 8B model's decode products: up to 8 rows it wins from about 80 MB of weights up (gate/up, down, output
    head) and loses to the small-M kernel below (q/k/v, o); from 9 to 16 rows it wins at every shape, against the
    small-M kernel and against the tcgen05 kernel with K slices; from 17 rows on the tcgen05 kernel is ahead."""
    if K % 64:
        return False
    return (M <= STREAM_M_AUTO and N * K >= STREAM_MIN_WEIGHTS) or STREAM_M_AUTO < M <= STREAM_M_AUTO_WIDE


def run_stream(a, w, out, epilogue: int, ldo: int, limit: float = 0.0, slope: float = 1.0) -> bool:
    """The persistent streaming kernel; epilogue 0 store, 1 add, 2 silu(gate) * up (3: tanh gelu; 4: the clamped form with
    its limit and slope) over w = [gate rows | up rows], 5 slope * max(z, 0)^2 in bf16."""
    M, K = a.shape
    N = w.shape[0]
    if M > STREAM_M or N > STREAM_MAX_N:
        return False
    lib = build.load("gemm_stream")
    scratch = _stream_buffers(a.device, lib)
    if scratch is None:
        return False
    ws, ct = scratch
    if epilogue == 4:
        code = lib.hk_gemm_stream_clamped(_ptr(a), _ptr(w), _ptr(out), M, N, K, ldo,
                                          stream_row_warps(N, _sms(a.device)), _ptr(ws), _ptr(ct), _ptr(status_flag(a.device)),
                                          _stream_ctas, limit, slope, _stream())
    elif epilogue == 5:
        code = lib.hk_gemm_stream_sqrelu(_ptr(a), _ptr(w), _ptr(out), M, N, K, ldo,
                                         stream_row_warps(N, _sms(a.device)), _ptr(ws), _ptr(ct), _ptr(status_flag(a.device)),
                                         _stream_ctas, slope, _stream())
    else:
        code = lib.hk_gemm_stream(_ptr(a), _ptr(w), _ptr(out), M, N, K, ldo, epilogue,
                                  stream_row_warps(N, _sms(a.device)),
                                  _ptr(ws), _ptr(ct), _ptr(status_flag(a.device)), _stream_ctas, _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm (streaming)")
    return True


# Clusters of CTAs with a whole SM's shared memory each that are resident at once on 148 SMs (asked of the driver's occupancy
# call): the groups of SMs a cluster must sit in are not multiples of it.
CLUSTERS_AT_ONCE = {2: 74, 3: 45, 4: 33, 6: 22, 8: 15}
CLUSTER_M = 128


@functools.lru_cache(maxsize=4096)
def cluster_config(M: int, N: int, K: int, sms: int):
    """(tile width, K slices) of the product whose slices are added inside a cluster, or None where the sliced kernel with its
    second launch stays.  It takes what would be cut into three slices or more: with two the partial sums are few, and 64 and
    128 rows by 8,192 x 4,096 measured 19.3 and 21.7 us that way, 19.7 and 23.2 in clusters.  All clusters run at once; among
    the widths and slices that allow it a model picks (a K block costs a fixed part and its bytes; then the tile goes through
    shared memory), within 4 % of the best of all 27 measured shapes of 24 to 128 rows.  64 rows, us before and now: 4,096 x
    4,096 13.9 and 12.8, 6,144 x 4,096 17.0 and 16.1, 4,096 x 12,288 26.9 and 24.9, 2,560 x 2,560 10.6 and 8.9."""
    if M > CLUSTER_M or N % 4 or tc_config(M, N, K, sms)[1] < 3:
        return None
    k_blocks, rows = -(-K // 64), -(-M // 8) * 8
    best = None
    for slices, clusters in CLUSTERS_AT_ONCE.items():
        if k_blocks < 4 * slices:
            break
        for bn in range(64, 257, 32):
            if -(-N // bn) > clusters * sms // 148:
                continue
            cost = k_blocks / slices * (0.25 + 0.0007 * (rows + bn)) + 1.3e-4 * M * bn
            if best is None or cost < best[0]:
                best = (cost, bn, slices)
    return best and best[1:]


def run_cluster(a, w, out, accumulate: bool, bn: int, slices: int) -> bool:
    """out (fp32) = a w^T (+ out) with the K slices added inside clusters.  False when the kernel refuses."""
    M, K = a.shape
    N = w.shape[0]
    code = build.load("gemm_tc").hk_gemm_tc_cluster(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, 1 if accumulate else 0,
                                                    bn, slices, _ptr(status_flag(a.device)), _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm (tcgen05, clusters)")
    return True


PAIR_M = 128            # from here on the rows' padding to 32 instead of 128 and the pairs' larger tiles pay
PAIR_K = 1024           # below, a tile's start and end weigh more than its loop: 4,096 x 512 by 527 rows 7.9 us, on pairs 8.7


@functools.lru_cache(maxsize=4096)
def pair_config(M: int, N: int, K: int, sms: int, gated: bool = False):
    """(tiles along the rows, K slices) of the product on pairs of SMs, or None where the kernel of one SM a tile stays: up to
    128 rows, short K, and where two row tiles of that kernel fill one wave of SMs better (10,304 x 2,048 by 256 rows 15.5 us, on
    pairs 17.6; 2,048 x 6,144 by 256 14.1 and 17.5, by 1,000 24.9 and 22.2).
    The two times come from models in `runtime.cpp`."""
    if M <= PAIR_M or K < PAIR_K:
        return None
    found = _pair_choice()(M, N, K, sms, *tc_config(M, N, K, sms, gated))
    return (found // 8, found % 8) if found else None


@functools.lru_cache(maxsize=1)
def _pair_choice():
    choose = build.load("runtime").hk_pair_config
    choose.argtypes, choose.restype = [ctypes.c_longlong] * 6, ctypes.c_longlong
    return choose


def run_pair(a, w, out, epilogue: int, ldo: int, tiles_m: int, slices: int, limit: float = 0.0, slope: float = 1.0) -> bool:
    """The product on pairs of SMs; `epilogue` and its numbers as `hk_gemm_pair` takes them.  False when the kernel refuses."""
    M, K = a.shape
    N = w.shape[0]
    lib = build.load("gemm_pair")
    partial = None
    if slices > 1:
        partial = torch.empty(int(lib.hk_gemm_pair_partial_floats(M, N, tiles_m, slices)), dtype=torch.float32, device=a.device)
    code = lib.hk_gemm_pair(_ptr(a), _ptr(w), _ptr(out), M, N, K, ldo, epilogue, tiles_m, slices, _sms(a.device) // 2,
                            _ptr(partial) if slices > 1 else 0, _ptr(status_flag(a.device)), limit,
                            slope, _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm (tcgen05, pairs)")
    return True


def _run_pair_where_chosen(a, w, out, choice: Optional[str], epilogue: int, ldo: int, limit: float = 0.0, slope: float = 1.0) -> bool:
    """The product on pairs where `pair_config` picks it; everywhere when it is pinned, nowhere when the other tcgen05 kernel is."""
    if choice == "tc" or _tc_bn or _tc_splits:
        return False
    chosen = pair_config(a.shape[0], w.shape[0], a.shape[1], _sms(a.device), epilogue in (2, 3, 4))
    if chosen is None and choice == "pair":
        chosen = (-(-a.shape[0] // 256), 1)
    return chosen is not None and run_pair(a, w, out, epilogue, ldo, *chosen, limit, slope)


def _tc_partial(lib, M: int, N: int, splits: int, device):
    """Scratch for the partial sums of `splits` K slices (None without slices)."""
    if splits <= 1:
        return None
    return torch.empty(int(lib.hk_gemm_tc_partial_floats(M, N, splits)), dtype=torch.float32, device=device)


def run(a, w, out, accumulate: bool, choice: Optional[str]) -> bool:
    """out (fp32) = a w^T (+ out).  Returns False when no tensor-core kernel takes the shape."""
    M, K = a.shape
    N = w.shape[0]
    if not _aligned(a, w):
        return False
    if choice == "stream" or (choice is None and stream_wanted(M, N, K)):
        if run_stream(a, w, out, 1 if accumulate else 0, N):
            return True
        if choice == "stream":
            return False
    if choice == "smallm" or (choice is None and M <= SMALL_M_AUTO):
        if M > SMALL_M:
            return False
        lib = build.load("gemm_smallm")
        code = lib.hk_gemm_smallm(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, 1 if accumulate else 0,
                                  row_tiles(M, N, a.device), _stream())
        if code == _UNSUPPORTED:
            return False
        ops._check(code, "gemm (small-M)")
        return True
    if _run_pair_where_chosen(a, w, out, choice, 1 if accumulate else 0, N):
        return True
    if choice == "pair":
        return False
    clusters = None if _tc_bn or _tc_splits else cluster_config(M, N, K, _sms(a.device))
    if clusters is not None and run_cluster(a, w, out, accumulate, *clusters):
        return True
    lib = build.load("gemm_tc")
    bn, splits = tc_config(M, N, K, _sms(a.device))
    partial = _tc_partial(lib, M, N, splits, a.device)
    code = lib.hk_gemm_tc(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, 1 if accumulate else 0, bn,
                          splits, _ptr(partial) if splits > 1 else 0, _ptr(status_flag(a.device)), _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm (tcgen05)")
    return True


def run_swiglu(a, w_gate_up, out, choice: Optional[str] = None, act: int = 0, limit: float = 0.0, slope: float = 1.0) -> bool:
    """out (bf16 [M, F]) = act(gate) * up of a w^T for w = [F gate rows | F up rows], in the epilogue of the
    streaming kernel (few rows) or of the tcgen05 kernel; act 0 is silu, 1 the tanh form of gelu, 2 the clamped form
    g sigmoid(slope g) (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit).  False when they refuse."""
    if act not in (0, 1, 2):
        return False
    epilogue = 2 + int(act)
    M, K = a.shape
    N = w_gate_up.shape[0]
    if not _aligned(a, w_gate_up) or N % 2:
        return False
    if choice == "stream" or (choice is None and stream_wanted(M, N, K)):
        if N % (16 * stream_row_warps(N, _sms(a.device))) == 0 and run_stream(a, w_gate_up, out, epilogue, out.shape[1], limit, slope):
            return True
        if choice == "stream":
            return False
    if choice is None and M <= SMALL_M_AUTO:
        return False             # few rows, small weights: the small-M product and the swiglu kernel
    if _run_pair_where_chosen(a, w_gate_up, out, choice, epilogue, out.shape[1], limit, slope):
        return True
    if choice == "pair":
        return False
    lib = build.load("gemm_tc")
    bn, splits = tc_config(M, N, K, _sms(a.device), swiglu=True)
    partial = _tc_partial(lib, M, N, splits, a.device)
    if epilogue == 4:
        code = lib.hk_gemm_tc_clamped(_ptr(a), _ptr(w_gate_up), _ptr(out), M, N, K, out.shape[1], bn, splits,
                                      _ptr(partial) if splits > 1 else 0, _ptr(status_flag(a.device)),
                                      limit, slope, _stream())
    else:
        code = lib.hk_gemm_tc(_ptr(a), _ptr(w_gate_up), _ptr(out), M, N, K, out.shape[1], epilogue, bn,
                              splits, _ptr(partial) if splits > 1 else 0, _ptr(status_flag(a.device)), _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm+swiglu (tcgen05)")
    return True


def run_squared_relu(a, w, out, factor: float, choice: Optional[str] = None) -> bool:
    """out (bf16 [M, N]) = factor * max(a w^T, 0)^2 in the epilogue of the product that `run` would take for the shape.
    False when no tensor-core kernel takes it."""
    M, K = a.shape
    N = w.shape[0]
    if not _aligned(a, w):
        return False
    if choice == "stream" or (choice is None and stream_wanted(M, N, K)):
        if run_stream(a, w, out, 5, N, slope=factor):
            return True
        if choice == "stream":
            return False
    if choice == "smallm" or (choice is None and M <= SMALL_M_AUTO):
        if M > SMALL_M:
            return False
        lib = build.load("gemm_smallm")
        code = lib.hk_gemm_smallm_sqrelu(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, row_tiles(M, N, a.device),
                                         factor, _stream())
        if code == _UNSUPPORTED:
            return False
        ops._check(code, "gemm+squared relu (small-M)")
        return True
    if _run_pair_where_chosen(a, w, out, choice, 5, N, slope=factor):
        return True
    if choice == "pair":
        return False
    lib = build.load("gemm_tc")
    bn, splits = tc_config(M, N, K, _sms(a.device))
    partial = _tc_partial(lib, M, N, splits, a.device)
    code = lib.hk_gemm_tc_sqrelu(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, bn, splits,
                                 _ptr(partial) if splits > 1 else 0, _ptr(status_flag(a.device)),
                                 factor, _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm+squared relu (tcgen05)")
    return True


def run_narrow(a, w, out, choice: Optional[str] = None) -> bool:
    """out (bf16 [M, N]) = a w^T on a tcgen05 kernel ('tc' and 'pair' pin one of them).  False when it refuses the shape."""
    M, K = a.shape
    N = w.shape[0]
    if not _aligned(a, w):
        return False
    if _run_pair_where_chosen(a, w, out, choice, 6, N):
        return True
    if choice == "pair":
        return False
    lib = build.load("gemm_tc")
    bn, splits = tc_config(M, N, K, _sms(a.device))
    partial = _tc_partial(lib, M, N, splits, a.device)
    code = lib.hk_gemm_tc_narrow(_ptr(a), _ptr(w), _ptr(out), M, N, K, N, bn, splits,
                                 _ptr(partial) if splits > 1 else 0, _ptr(status_flag(a.device)), _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "gemm, narrowed (tcgen05)")
    return True


def grouped_tile_rows(pairs: int, experts: int) -> int:
    """Rows of a tile of the grouped product for so many (row, choice) pairs: a tile's width follows its rows in steps of 32, but what
    it loads, and how deep its ring is, follows the most it may have.  Both products, us (8 experts, width 4,096; rows a tile 64 / 128 /
    256): 128 pairs 71.1 / 71.3 / 72.0, 600 87.0 / 77.5 / 78.4, 1,400 115 / 101 / 90, 4,096 263 / 196 / 187."""
    each = pairs / experts
    return 64 if each <= 32 else 128 if each <= 100 else 256


def grouped_takes(x, *weights) -> bool:
    """Whether the grouped product on the tensor cores takes rows x, as they lie, by each of the experts' weights [E, N, K]; what it does
    not take goes to the product by FMAs."""
    return x.shape[1] % 8 == 0 and x.data_ptr() % 16 == 0 and \
        all(w.data_ptr() % 16 == 0 and w.is_contiguous() and w.shape[0] * w.shape[1] < 2 ** 31 for w in weights)


def run_pair_grouped(a, w, out, tiles, offsets, tile_rows: int, gated: bool, act: int = 0, limit: float = 0.0, slope: float = 1.0) -> bool:
    """out[p] = a[p] w[group of p]^T for the rows p that `tiles` and `offsets` name (`hk_gemm_pair_grouped`); gated: act 0 (silu) or 2
    (the clamped form) of the two halves.  False when the kernel refuses."""
    if gated and act not in (0, 2):
        return False
    M, K = a.shape
    E, N = int(w.shape[0]), int(w.shape[1])
    if a.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or K % 8 or not _aligned(a, w) or not w.is_contiguous() or (gated and N % 2):
        return False
    code = build.load("gemm_pair").hk_gemm_pair_grouped(
        _ptr(a), _ptr(w), _ptr(out), M, N, K, out.shape[1], 2 + act if gated else 0, E, _ptr(tiles), tiles.shape[0], _ptr(offsets), tile_rows,
        _sms(a.device) // 2, _ptr(status_flag(a.device)), limit, slope, _stream())
    if code == _UNSUPPORTED:
        return False
    ops._check(code, "grouped gemm (tcgen05, pairs)")
    return True
