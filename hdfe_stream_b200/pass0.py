"""Pass 0 on the device: factorize the fixed-effect ids and sort the rows.

core/passes.py:285-294 codes every fixed effect by the rank of its level
among the sorted distinct levels, and :359-373 sorts the rows by the
streamed dimension's code, the other codes and then the variables (when the
fit keeps its intermediates; n_buckets = 1), the streamed code becoming the
dense group code.  Here the raw columns are already on the device and both
steps run on this library's own radix sort (csrc/sort.cu):

* each id column is factorized: integer ids of a range of at most 32 values
  an id through a bitmap of the range (`hdfe_factorize_range`), others by
  `hdfe_factorize` (a stable radix sort of the ids' order-preserving unsigned
  keys with their positions, run heads, a scan of the heads, the ranks
  scattered back; integers shifted by their minimum first, so only the bits
  their range needs are sorted);
* the codes are packed, most significant first, into one 64-bit key of
  ceil(log2(levels)) bits each (columns that do not fit go in further keys)
  and the rows ordered by a stable `hdfe_sort_pairs` of the keys with the
  row positions; with one key, the sorted codes are read back out of the
  sorted keys and one kernel gathers the rest (`hdfe_rows_from_order`);
* when two rows share every code, the variables break the tie: the order
  is rebuilt least significant key first (the last variable ... the first,
  then the code keys), each pass stable -- the same order as the host
  layout of these rows (`simulate.pass0_layout`, numpy's lexsort).
"""

from __future__ import annotations

import ctypes

from . import _lib
from .fit import DeviceRows

SIGN = -(2 ** 63)           # the int64 with only the top bit set


def _torch():
    import torch
    return torch


def _bits(n: int) -> int:
    """Bits that codes 0 .. n - 1 need (at least one)."""
    return max((int(n) - 1).bit_length(), 1)


def order_key(t):
    """int64 tensor whose bits, read as unsigned, order like t's values:
    integers by value; floats by value with -0.0 = 0.0 and NaN last."""
    torch = _torch()
    if t.dtype.is_floating_point:
        x = t.to(torch.float64) + 0.0                      # -0.0 -> +0.0
        b = x.view(torch.int64)
        k = torch.where(b < 0, ~b, b ^ SIGN)
        return torch.where(torch.isnan(x), torch.full_like(k, -1), k)
    return t.to(torch.int64) ^ SIGN


def _from_key(k, dtype):
    torch = _torch()
    if dtype.is_floating_point:
        b = torch.where(k < 0, k ^ SIGN, ~k)
        return b.view(torch.float64).to(dtype)
    return (k ^ SIGN).to(dtype)


def _workspace(n: int, device):
    torch = _torch()
    size = int(_lib.lib().hdfe_sort_workspace_bytes(int(n)))
    return torch.empty(size, dtype=torch.uint8, device=device), size


def sort_pairs(keys, vals=None, key_bits: int = 64):
    """(sorted keys, values) of a stable ascending sort of the int64 `keys`
    read as unsigned, by their low `key_bits` bits; vals int32 (None: the
    positions 0 .. n-1)."""
    torch = _torch()
    keys = keys.contiguous()
    n = keys.numel()
    if n > 2 ** 31 - 1:
        raise ValueError("sort_pairs: at most 2^31 - 1 items")
    if vals is not None:
        vals = vals.to(torch.int32).contiguous()
        if vals.numel() != n:
            raise ValueError("sort_pairs: keys and vals differ in length")
    k_out = torch.empty_like(keys)
    v_out = torch.empty(n, dtype=torch.int32, device=keys.device)
    if n == 0:
        return k_out, v_out
    ws, size = _workspace(n, keys.device)
    _lib.check(_lib.lib().hdfe_sort_pairs(keys.data_ptr(), _lib.ptr(vals), n, int(key_bits),
                                          k_out.data_ptr(), v_out.data_ptr(), ws.data_ptr(),
                                          size, _lib.stream_handle()))
    return k_out, v_out


# A range of ids up to this many values an id goes through the bitmap: its words
# then stay within 4 bytes an id, half of one radix pass's keys (16 with the words'
# counts and ranks, which leave the L2 from some 8M ids on).
RANGE_PER_ID = 32
RANGE_FREE = 1 << 20


def _ranges(cols):
    """(least, largest) of every integer column, one read for all; None for
    an empty or a float one."""
    torch = _torch()
    at = [i for i, c in enumerate(cols) if c.numel() and not c.dtype.is_floating_point]
    out = [None] * len(cols)
    if at:
        wide = [c if c.dtype in (torch.int32, torch.int64) else c.to(torch.int64)
                for c in (cols[i] for i in at)]
        got = torch.stack([torch.stack(torch.aminmax(c)).to(torch.int64) for c in wide])
        for i, (lo, hi) in zip(at, got.cpu().tolist()):
            out[i] = (lo, hi)
    return out


def _factorize_all(cols):
    """[(codes int32, levels)] of id columns (`factorize`), the sizes in two
    reads for all of them."""
    torch = _torch()
    lib = _lib.lib()
    work = []                               # codes, levels buffer, count, to levels
    for ids, ends in zip(cols, _ranges(cols)):
        n = ids.numel()
        if n == 0:
            work.append((torch.zeros(0, dtype=torch.int32, device=ids.device), ids.clone(), None,
                         None))
            continue
        if n > 2 ** 31 - 1:
            raise ValueError("factorize: at most 2^31 - 1 ids")
        codes = torch.empty(n, dtype=torch.int32, device=ids.device)
        count = torch.zeros(1, dtype=torch.int64, device=ids.device)
        span = None if ends is None else ends[1] - ends[0] + 1
        if span is not None and span <= RANGE_PER_ID * n + RANGE_FREE:
            x = ids if ids.dtype in (torch.int32, torch.int64) else ids.to(torch.int64)
            x = x.contiguous()
            levels = torch.empty(min(n, span), dtype=torch.int64, device=ids.device)
            size = int(lib.hdfe_factorize_range_workspace_bytes(span))
            ws = torch.empty(size, dtype=torch.uint8, device=ids.device)
            _lib.check(lib.hdfe_factorize_range(x.data_ptr(), x.element_size(), n, ends[0], span,
                                                codes.data_ptr(), levels.data_ptr(),
                                                count.data_ptr(), ws.data_ptr(), size,
                                                _lib.stream_handle()))
            work.append((codes, levels, count, lambda v, t=ids.dtype: v.to(t)))
            continue
        if span is None:
            keys, base, bits = order_key(ids), None, 64
        elif span <= 2 ** 63:
            keys, base, bits = ids.to(torch.int64) - ends[0], ends[0], max((span - 1).bit_length(), 1)
        else:                                   # the range needs the sign bit
            keys, base, bits = ids.to(torch.int64) ^ SIGN, None, 64
        keys = keys.contiguous()
        levels = torch.empty(n, dtype=torch.int64, device=ids.device)
        ws, size = _workspace(n, ids.device)
        _lib.check(lib.hdfe_factorize(keys.data_ptr(), n, bits, codes.data_ptr(),
                                      levels.data_ptr(), count.data_ptr(), ws.data_ptr(),
                                      size, _lib.stream_handle()))
        work.append((codes, levels, count,
                     (lambda v, t=ids.dtype, b=base: (v + b).to(t)) if base is not None
                     else (lambda v, t=ids.dtype: _from_key(v, t))))
    counts = [c for _, _, c, _ in work if c is not None]
    sizes = iter(torch.cat(counts).cpu().tolist() if counts else [])
    return [(codes, levels if count is None else back(levels[:next(sizes)]))
            for codes, levels, count, back in work]


def factorize(ids):
    """(codes int64, levels): the rank of each id among the sorted distinct
    ids, and those ids in order (ids' dtype)."""
    torch = _torch()
    (codes, levels), = _factorize_all([ids])
    return codes.to(torch.int64), levels


def _packed_keys(cols, sizes):
    """[(key, bits)] most significant first: consecutive code columns packed
    into 64-bit keys, each column `_bits(size)` wide."""
    torch = _torch()
    keys, cur, used = [], None, 0
    for c, n in zip(cols, sizes):
        b, c = _bits(n), c.to(torch.int64)
        if cur is None:
            cur, used = c, b
        elif used + b > 64:
            keys.append((cur, used))
            cur, used = c, b
        else:
            cur, used = (cur << b) | c, used + b
    keys.append((cur, used))
    return keys


def _chain(keys, n, device):
    """The stable order of n rows by keys [(key, bits)], most significant
    first: one sort per key, least significant first."""
    torch = _torch()
    order = None
    for k, b in reversed(keys):
        k = k if order is None else k[order.to(torch.int64)]
        _, order = sort_pairs(k, order, b)
    return order.to(torch.int64) if order is not None else torch.arange(n, device=device)


def pass0(streamed, fixed_effects, V, w=None, sort_only=()):
    """DeviceRows in pass 0's layout from raw device columns: `streamed` (N,)
    the streamed dimension's ids (the groups), `fixed_effects` a list of (N,)
    id columns (the codes, in order), V (N, m) float64 (outcome first), w (N,)
    or None, `sort_only` id columns that order the rows without being fixed
    effects.  Returns (rows, levels): levels per column, streamed first."""
    torch = _torch()
    N = streamed.numel()
    fixed_effects = list(fixed_effects)         # (any iterable, read once)
    ids = [streamed] + fixed_effects + list(sort_only)
    coded = _factorize_all(ids)
    sizes = [len(l) for _, l in coded]
    D = len(fixed_effects)
    levels = [l for _, l in coded[:1 + D]]
    rows = _rows_by_one_key(coded, sizes, D, V, w, N)
    if rows is not None:
        return rows, levels
    cols = [c.to(torch.int64) for c, _ in coded]
    g, fe = cols[0], cols[1:1 + D]
    code_keys = _packed_keys(cols, sizes)
    order = _chain(code_keys, N, g.device)
    # rows sharing every code: neighbours equal in every key after the sort
    same = torch.ones(max(N - 1, 0), dtype=torch.bool, device=g.device)
    for k, _ in code_keys:
        sk = k[order]
        same &= sk[1:] == sk[:-1]
    if bool(same.any()):
        var_keys = [(order_key(V[:, j]), 64) for j in range(V.shape[1])]
        order = _chain(code_keys + var_keys, N, g.device)
    codes = torch.stack([c[order] for c in fe], 1).to(torch.int32).contiguous()
    rows = DeviceRows(g[order].to(torch.int32).contiguous(), codes,
                      V[order].T.contiguous().to(torch.float64),
                      None if w is None else w[order].to(torch.float64).contiguous(),
                      sizes[1:1 + D])
    return rows, levels


def _rows_by_one_key(coded, sizes, D, V, w, N):
    """The rows when all codes pack into one key and no two rows share it:
    one sort, the codes out of the sorted keys, one gather.  None for every
    other form of the input (several keys, ties that the variables break, no
    rows, columns of different lengths or devices, inputs that record
    gradients or carry a forward derivative): those take the general path."""
    torch = _torch()
    lib = _lib.lib()
    bits = [_bits(n) for n in sizes]
    dev = coded[0][0].device
    if N == 0 or D == 0 or sum(bits) > 64 or max(bits) > 31 or len(bits) > 8:
        return None
    if any(c.numel() != N or c.device != dev for c, _ in coded) or V.dim() != 2 or \
            V.shape[0] != N or V.device != dev or V.requires_grad or V.is_complex() or \
            not _lib.is_plain(V):
        return None
    if w is not None and (w.dim() != 1 or w.numel() != N or w.device != dev or w.requires_grad
                          or w.is_complex() or not _lib.is_plain(w)):
        return None
    m = int(V.shape[1])
    cols = (ctypes.c_void_p * len(bits))(*[c.data_ptr() for c, _ in coded])
    width = (ctypes.c_int32 * len(bits))(*bits)
    keys = torch.empty(N, dtype=torch.int64, device=dev)
    _lib.check(lib.hdfe_pack_codes(cols, width, len(bits), N, keys.data_ptr(),
                                   _lib.stream_handle()))
    keys, order = sort_pairs(keys, None, sum(bits))
    V = V.to(torch.float64).contiguous()
    w = None if w is None else w.to(torch.float64).contiguous()
    gcode = torch.empty(N, dtype=torch.int32, device=dev)
    codes = torch.empty((N, D), dtype=torch.int32, device=dev)
    V_out = torch.empty((m, N), dtype=torch.float64, device=dev)
    w_out = None if w is None else torch.empty(N, dtype=torch.float64, device=dev)
    ties = torch.empty(1, dtype=torch.int32, device=dev)
    _lib.check(lib.hdfe_rows_from_order(
        width, len(bits), D, N, keys.data_ptr(), order.data_ptr(), V.data_ptr(), m, _lib.ptr(w),
        gcode.data_ptr(), codes.data_ptr(), V_out.data_ptr(), _lib.ptr(w_out), ties.data_ptr(),
        _lib.stream_handle()))
    if int(ties.item()):
        return None
    return DeviceRows(gcode, codes, V_out, w_out, sizes[1:1 + D])
