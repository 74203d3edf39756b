"""Decode-time ops: paged-KV attention and KV-cache append (CUDA kernels, PyTorch statement on CPU).

The reference decodes by running the whole context through the model again for every token
(llm-core/llm_core/model.py:187-236, no KV cache); these ops are what a cached decode step needs instead."""
from __future__ import annotations

import ctypes
import math

import torch

from . import native, torch_impl

_declared = False


def _lib():
    global _declared
    lib = native.load()
    if not _declared:
        P, I, L, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
        lib.b200_paged_decode.argtypes = [P, P, P, P, P, P, P, P, I, I, I, I, I, I, I, F, I, P, P]
        lib.b200_paged_decode.restype = I
        lib.b200_kv_append.argtypes = [P, P, P, P, L, I, L, P, P]
        lib.b200_kv_append.restype = I
        lib.b200_rope_kv_append.argtypes = [P, P, P, P, P, P, L, I, I, I, L, P, P]
        lib.b200_rope_kv_append.restype = I
        lib.b200_gemm_bf16_append.argtypes = [P, P, P, I, I, L, L, L, I, P, P, P]
        lib.b200_gemm_bf16_append.restype = I
        lib.b200_lm_layers.argtypes = [P, P]
        lib.b200_lm_layers.restype = I
        _declared = True
    return lib


def kv_append(k_cache, v_cache, qkv, slot_mapping):
    """Write the K and V thirds of qkv (R, 3d) into cache slots ``page * page_size + offset`` (int64, -1 skips)."""
    if not qkv.is_cuda:
        keep = slot_mapping >= 0
        return torch_impl.kv_append(k_cache, v_cache, qkv[keep], slot_mapping[keep])
    lib = _lib()
    d = qkv.shape[1] // 3
    native._req(qkv.dtype == torch.bfloat16 and qkv.is_contiguous() and k_cache.is_contiguous(), "bad kv_append inputs")
    native._req(slot_mapping.dtype == torch.int64 and slot_mapping.numel() == qkv.shape[0], "bad slot mapping")
    native._req(k_cache.shape == v_cache.shape and k_cache.shape[-1] == d, "cache shape does not match qkv")
    num_slots = k_cache.shape[0] * k_cache.shape[1]
    native._check(lib.b200_kv_append(qkv.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), slot_mapping.data_ptr(),
                                     qkv.shape[0], d, num_slots, native.status_word(qkv.device).data_ptr(),
                                     native._stream()), "kv_append")


def rope_kv_append(qkv, cos_sin, positions, k_cache, v_cache, slot_mapping, n_heads: int):
    """Rotate the Q and K thirds of qkv (R, 3d) in place by the angle of ``positions`` and write the rotated K row and
    the V row into cache slot ``slot_mapping`` (-1: rotate only).  One kernel on the GPU; the two separate ops elsewhere."""
    if not qkv.is_cuda:
        from . import rope_ as _rope
        _rope(qkv, cos_sin, positions, n_heads, False, None)
        return kv_append(k_cache, v_cache, qkv, slot_mapping)
    lib = _lib()
    d = qkv.shape[1] // 3
    dh = d // n_heads
    native._req(qkv.dtype == torch.bfloat16 and qkv.is_contiguous() and k_cache.is_contiguous() and v_cache.is_contiguous(),
                "bad rope_kv_append inputs")
    native._req(slot_mapping.dtype == torch.int64 and slot_mapping.numel() == qkv.shape[0], "bad slot mapping")
    native._req(positions.dtype == torch.int32 and positions.numel() == qkv.shape[0] and positions.is_contiguous(),
                "positions must be int32 (R,)")
    native._req(k_cache.shape == v_cache.shape and k_cache.shape[-1] == d, "cache shape does not match qkv")
    native._req(cos_sin.dtype == torch.float32 and cos_sin.is_contiguous() and cos_sin.shape[0] == 2
                and cos_sin.shape[2] == dh // 2 and dh % 8 == 0, "bad rope cache")
    num_slots = k_cache.shape[0] * k_cache.shape[1]
    native._check(lib.b200_rope_kv_append(qkv.data_ptr(), cos_sin.data_ptr(), positions.data_ptr(), k_cache.data_ptr(),
                                          v_cache.data_ptr(), slot_mapping.data_ptr(), qkv.shape[0], d, dh,
                                          cos_sin.shape[1], num_slots, native.status_word(qkv.device).data_ptr(),
                                          native._stream()), "rope_kv_append")


class QkvAppend(ctypes.Structure):
    """csrc/gemm_common.cuh: QkvAppend."""
    _fields_ = [("cs", ctypes.c_void_p), ("positions", ctypes.c_void_p), ("slots", ctypes.c_void_p), ("k_cache", ctypes.c_void_p),
                ("v_cache", ctypes.c_void_p), ("num_slots", ctypes.c_longlong), ("d", ctypes.c_int), ("dh", ctypes.c_int), ("ctx", ctypes.c_int)]


# Rows x width x width up to which a layer takes the device less time than its launches take the host (about 100 us): there a launch less is
# worth more than the time that rotating and appending takes a product's epilogue, whose rows lie scattered (rows x width, us a launch, fused and as
# three launches: 256 x 768 7.5, 8.6; 512 x 2048 27.7, 20.3; 2048 x 1024 25.0, 22.4).  Whole prompts, us, three launches -> fused: 256 x 2048
# 2831 -> 2693, 1536 x 1024 1686 -> 1619, 4096 x 512 963 -> 937; beyond the limit 512 x 2048 3163 -> 3278, 4096 x 768 2002 -> 2138,
# 8192 x 2048 18230 -> 20200.  Captured decode steps, all within the limit: 16 x 2048 1833 -> 1765, 128 x 768 869 -> 860, 256 x 2048 4739 -> 4746.
APPEND_MAX_WORK = 1.6e9


def _appends_in_product(r: int, k: int, d: int, dh: int) -> bool:
    sliced = native.USE_SPLITK and r <= native.SPLITK_MAX_M and k >= native.SPLITK_MIN_K
    return r * k * d <= APPEND_MAX_WORK and dh % 32 == 0 and d % 64 == 0 and not sliced


def qkv_rope_append(h, wqkv, cos_sin, positions, k_cache, v_cache, slot_mapping, n_heads: int):
    """qkv = h (R, d) @ wqkv (3 d, d)^T, then what ``rope_kv_append`` does with it, in the product's epilogue where the step is short
    (``APPEND_MAX_WORK``), the heads are made of its chunks of columns and its contraction is not cut in slices.  The same values either way."""
    r, k = h.shape
    d = wqkv.shape[0] // 3
    dh = d // n_heads
    if h.is_cuda and _appends_in_product(r, k, d, dh):
        native._req(h.dtype == torch.bfloat16 and wqkv.dtype == torch.bfloat16 and h.stride(1) == 1 and wqkv.stride(1) == 1
                    and wqkv.shape[1] == k and dh * n_heads == d, "bad projection")
        native._req(slot_mapping.dtype == torch.int64 and slot_mapping.numel() == r and slot_mapping.is_contiguous()
                    and positions.dtype == torch.int32 and positions.numel() == r and positions.is_contiguous(), "bad slot mapping or positions")
        native._req(k_cache.shape == v_cache.shape and k_cache.shape[-1] == d and k_cache.is_contiguous() and v_cache.is_contiguous()
                    and k_cache.dtype == v_cache.dtype == torch.bfloat16, "cache shape does not match")
        native._req(cos_sin.dtype == torch.float32 and cos_sin.is_contiguous() and cos_sin.shape[0] == 2 and cos_sin.shape[2] == dh // 2
                    and dh % 8 == 0, "bad rope cache")
        out = torch.empty((r, 3 * d), dtype=torch.bfloat16, device=h.device)
        what = QkvAppend(cos_sin.data_ptr(), positions.data_ptr(), slot_mapping.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(),
                         k_cache.shape[0] * k_cache.shape[1], d, dh, cos_sin.shape[1])
        rc = _lib().b200_gemm_bf16_append(h.data_ptr(), wqkv.data_ptr(), out.data_ptr(), r, k, h.stride(0), wqkv.stride(0), 3 * d,
                                          native.EPI_B_STABLE, ctypes.byref(what), native.status_word(h.device).data_ptr(), native._stream())
        native._check(rc, "gemm_bf16_append")
        return out
    from . import gemm
    qkv = gemm(h, wqkv, "nt", b_stable=True)
    rope_kv_append(qkv, cos_sin, positions, k_cache, v_cache, slot_mapping, n_heads)
    return qkv


def choose_splits(rows: int, heads: int, max_context: int, sms: int = 148, head_dim: int = 128) -> int:
    """Context splits per request for the decode kernel (one CTA per (request, split)).

    The CTAs of a launch run in waves of ``sms * resident`` (a CTA has heads * head_dim / 8 threads of 128 registers,
    so two fit on an SM for a 2048-wide model), and a last wave that is mostly empty costs as much as a full one:
    at batch 128 five splits are 2.2 waves (5.6 TB/s measured) where eight are 3.5 (6.1 TB/s).  Among the split
    counts that leave at least 256 tokens per split at full context, take the one whose CTAs fill their waves best;
    ties go to more splits (shorter CTAs, a shorter tail)."""
    threads = max(32, -(-heads * head_dim // 8 // 32) * 32)
    resident = sms * max(1, min(32, 65536 // (128 * threads)))
    best, best_fill = 1, -1.0
    for s in range(1, max(1, min(32, max_context // 256)) + 1):
        ctas = rows * s
        fill = ctas / (-(-ctas // resident) * resident)
        if fill >= best_fill - 1e-9:
            best, best_fill = s, max(fill, best_fill)
    return best


def paged_decode_attention(qkv, k_cache, v_cache, block_tables, context_lens, n_heads: int, splits: int = 0,
                           scratch=None):
    """One query token per request against its paged KV history.

    qkv: (R, 3d) packed (only the query third is read) or (R, d); caches: (num_pages, page_size, d);
    block_tables: (R, max_pages) int32; context_lens: (R,) int32, number of cached tokens to attend to.
    Returns (R, d).  The values inside the tables are checked on the device: a length beyond ``max_pages * page`` or
    a page id beyond the cache is skipped and recorded in the status word (``native.check_status`` raises).
    """
    r, width = qkv.shape
    d = k_cache.shape[-1]
    dh = d // n_heads
    if not qkv.is_cuda:
        return torch_impl.paged_decode_attention(qkv[:, :d], k_cache, v_cache, block_tables, context_lens, n_heads)
    lib = _lib()
    native._req(qkv.dtype == torch.bfloat16 and qkv.stride(1) == 1, "qkv must be bf16 with unit inner stride")
    native._req(block_tables.dtype == torch.int32 and context_lens.dtype == torch.int32, "tables must be int32")
    native._req(block_tables.dim() == 2 and block_tables.is_contiguous() and block_tables.shape[0] >= r
                and context_lens.is_contiguous() and context_lens.numel() >= r, "one table row and one length per request")
    native._req(k_cache.is_contiguous() and v_cache.is_contiguous() and k_cache.shape == v_cache.shape and
                width in (d, 3 * d) and dh * n_heads == d, "cache / query shapes do not match")
    page = k_cache.shape[1]
    max_pages = block_tables.shape[1]
    if splits <= 0:
        splits = choose_splits(r, n_heads, max_pages * page, head_dim=dh)
    out = torch.empty((r, d), dtype=torch.bfloat16, device=qkv.device)
    if scratch is None:
        scratch = torch.empty(r * n_heads * splits * (dh + 2), dtype=torch.float32, device=qkv.device)
    part_o = scratch[:r * n_heads * splits * dh]
    part_ml = scratch[r * n_heads * splits * dh:]
    native._check(lib.b200_paged_decode(qkv.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), block_tables.data_ptr(),
                                        context_lens.data_ptr(), out.data_ptr(), part_o.data_ptr(), part_ml.data_ptr(),
                                        r, qkv.stride(0), n_heads, dh, page, max_pages, splits, 1.0 / math.sqrt(dh),
                                        k_cache.shape[0], native.status_word(qkv.device).data_ptr(), native._stream()),
                  "paged_decode")
    return out


# ------------------------------------------------------------------------------------------------------- all layers of a step
class LmProduct(ctypes.Structure):
    """csrc/lm_layers.cu: LmProduct."""
    _fields_ = [("kind", ctypes.c_int), ("slices", ctypes.c_int)]


class LmLayer(ctypes.Structure):
    """csrc/lm_layers.cu: LmLayer."""
    _fields_ = [(n, ctypes.c_void_p) for n in ("wqkv", "wo", "wgu", "wdown", "n1", "n2", "k", "v")]


class LmStep(ctypes.Structure):
    """csrc/lm_layers.cu: LmStep."""
    _fields_ = [(n, ctypes.c_void_p) for n in ("layers", "x", "y", "h", "qkv", "o", "gu", "act", "rstd", "cos_sin", "positions", "slots", "cu",
                                               "tables", "ctx_lens", "part_o", "part_ml", "ws", "counters", "status")] + \
               [(n, ctypes.c_longlong) for n in ("num_slots", "ws_floats")] + \
               [(n, ctypes.c_int) for n in ("n_layers", "rows", "d", "heads", "ff", "rope_ctx", "batch", "max_seq", "page_size", "max_pages",
                                            "splits", "num_pages", "n_counters", "append", "glu")] + \
               [("eps", ctypes.c_float), ("scale", ctypes.c_float)] + [(n, LmProduct) for n in ("pqkv", "po", "pgu", "pdown")]


_PAIR, _GROUPED, _ROUNDED = 0, 1, 2          # csrc/lm_layers.cu: LmGlu


def transformer_layers(x, layers, n_heads: int, d_ff: int, eps: float, cos_sin, positions, slots, k_cache, v_cache, fused: bool, cu=None,
                       max_seq: int = 0, tables=None, context_lens=None, splits: int = 0):
    """All layers of a serving step over the residual stream x (R, d), from one call into the kernel library: what the ops make of it one by one,
    launch by launch.  ``layers``: ``models.engine.BlockWeights``; caches (layers, pages, page size, d).  Attention among the step's rows
    (``cu``, ``max_seq``) or through the cache (``tables``, ``context_lens``).  ``fused``: gate and up are multiplied unrounded.
    Returns x, which then holds the result, or None for what only the single ops take (widths and heads that they pad)."""
    rows, d = x.shape
    dh = d // n_heads
    bf16, dev = torch.bfloat16, x.device
    if rows == 0 or not layers or d % 8 or d_ff % 8 or dh not in ((32, 64, 128) if cu is not None else (64, 128)) or d > 4096 and cu is None:
        return None
    req = native._req
    req(x.dtype == bf16 and x.is_contiguous() and dh * n_heads == d, "the residual stream must be contiguous bf16")
    req(positions.dtype == torch.int32 and positions.numel() == rows and positions.is_contiguous()
        and slots.dtype == torch.int64 and slots.numel() == rows and slots.is_contiguous(), "bad slot mapping or positions")
    req(k_cache.dtype == bf16 and v_cache.dtype == bf16 and k_cache.is_contiguous() and v_cache.is_contiguous() and k_cache.shape == v_cache.shape
        and k_cache.dim() == 4 and k_cache.shape[0] == len(layers) and k_cache.shape[3] == d, "cache shape does not match")
    req(cos_sin.dtype == torch.float32 and cos_sin.is_contiguous() and cos_sin.shape[0] == 2 and cos_sin.shape[2] == dh // 2, "bad rope cache")
    shapes = ((3 * d, d), (d, d), (2 * d_ff, d), (d, d_ff), (d,), (d,))
    table, step = (LmLayer * len(layers))(), k_cache.stride(0) * 2
    kp, vp = k_cache.data_ptr(), v_cache.data_ptr()
    for i, w in enumerate(layers):
        for t, shape in zip(w, shapes):
            req(t.shape == shape and t.dtype == bf16 and t.is_contiguous() and t.device == dev, "layer weights must be contiguous bf16")
        table[i] = LmLayer(*[t.data_ptr() for t in w], kp + i * step, vp + i * step)
    new = lambda *shape, dtype=bf16: torch.empty(shape, dtype=dtype, device=dev)
    s = LmStep(layers=ctypes.addressof(table), n_layers=len(layers), rows=rows, d=d, heads=n_heads, ff=d_ff, rope_ctx=cos_sin.shape[1], eps=eps,
               scale=1.0 / math.sqrt(dh), cos_sin=cos_sin.data_ptr(), positions=positions.data_ptr(), slots=slots.data_ptr(),
               num_slots=k_cache.shape[1] * k_cache.shape[2], page_size=k_cache.shape[2], num_pages=k_cache.shape[1],
               status=native.status_word(dev).data_ptr())
    held = [new(rows, d), new(rows, d), new(rows, 3 * d), new(rows, d), new(rows, d_ff), new(rows, dtype=torch.float32)]
    s.x = x.data_ptr()
    s.y, s.h, s.qkv, s.o, s.act, s.rstd = (t.data_ptr() for t in held)
    if cu is not None:
        req(cu.dtype == torch.int32 and cu.is_cuda and cu.is_contiguous(), "cu_seqlens must be int32 on the device")
        s.cu, s.batch, s.max_seq = cu.data_ptr(), cu.numel() - 1, max_seq
    else:
        req(tables.dtype == torch.int32 and context_lens.dtype == torch.int32 and tables.dim() == 2 and tables.is_contiguous()
            and tables.shape[0] >= rows and context_lens.is_contiguous() and context_lens.numel() >= rows, "one table row and one length per request")
        s.tables, s.ctx_lens, s.max_pages = tables.data_ptr(), context_lens.data_ptr(), tables.shape[1]
        s.splits = splits if splits > 0 else choose_splits(rows, n_heads, s.max_pages * s.page_size, head_dim=dh)
        held.append(new(rows * n_heads * s.splits * (dh + 2), dtype=torch.float32))
        s.part_o = held[-1].data_ptr()
        s.part_ml = s.part_o + rows * n_heads * s.splits * dh * 4
    route = lambda n, k: LmProduct(*native.nt_route(rows, n, k, dev))
    s.append = int(_appends_in_product(rows, d, d, dh))
    s.pqkv, s.po, s.pdown = route(3 * d, d), route(d, d), route(d, d_ff)
    if fused:
        s.glu = _PAIR if native.USE_PAIR and rows >= native.PAIR_MIN_M and d_ff % 64 == 0 else _GROUPED
    else:
        s.glu, s.pgu = _ROUNDED, route(2 * d_ff, d)
        held.append(new(rows, 2 * d_ff))
        s.gu = held[-1].data_ptr()
    scratch = native._splitk_scratch(dev) if 2 in (s.pqkv.kind, s.po.kind, s.pgu.kind, s.pdown.kind) else None
    if scratch is not None:
        ws, counters = scratch
        s.ws, s.ws_floats, s.counters, s.n_counters = ws.data_ptr(), ws.numel(), counters.data_ptr(), counters.numel()
    launches = _lib().b200_lm_layers(ctypes.byref(s), native._stream())
    native._check(min(launches, 0), "lm_layers")
    native.count_launches(launches - 1)
    return x
