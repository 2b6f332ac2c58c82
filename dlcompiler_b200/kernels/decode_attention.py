"""decode_attention_fwd with the signature of python/dlBLAS/dlblas/kernels/decode_attention.py:559."""
from __future__ import annotations

import torch

from .. import _lib
from .paged_attention import _pick_chunk


def decode_attention_fwd(
    q,
    k_buffer,
    v_buffer,
    o,
    req_to_token,
    b_req_idx,
    b_start_loc,
    b_seq_len,
    attn_logits,
    max_len_in_batch,
    sm_scale,
    logit_cap=0.0,
):
    """Token-granular decode attention: request `b_req_idx[i]` reads its keys and values from rows
    `req_to_token[b_req_idx[i], :b_seq_len[i]]` of `k_buffer` / `v_buffer` ([tokens, Hkv, D]).

    The reference runs two stages through a materialised `attn_logits` buffer
    (decode_attention.py:559-620); here the same math is one split-KV pass of the paged decode
    kernel with a page size of one token, so `attn_logits` and `b_start_loc` are accepted for
    signature compatibility and not touched.  `logit_cap > 0` applies cap * tanh(qk / cap).

    A `b_req_idx[i]` outside `req_to_token` is an error: the request gets zeros and `check_device_status()` raises.
    """
    dev = _lib.require_cuda(q, k_buffer, v_buffer, o, req_to_token, b_req_idx, b_seq_len)
    assert q.dim() == 3 and k_buffer.dim() == 3 and v_buffer.dim() == 3
    batch, head, D = q.shape
    Dv = v_buffer.shape[-1]
    assert k_buffer.shape[-1] == D and o.shape[-1] == Dv, "k must have the query's head size, o the value's"
    assert D % 8 == 0 and Dv % 8 == 0 and D <= 128 and Dv <= 128, "head sizes: multiples of 8 up to 128"
    assert q.stride(-1) == 1 and o.stride(-1) == 1 and k_buffer.stride(-1) == 1 and v_buffer.stride(-1) == 1
    hkv = k_buffer.shape[1]
    rows = b_req_idx if b_req_idx.dtype in (torch.int32, torch.int64) else b_req_idx.to(torch.int64)
    assert rows.dim() <= 1, "b_req_idx is one-dimensional"
    rows = rows.reshape(-1).contiguous()
    assert rows.size(0) >= batch, "b_req_idx: one table row per request"
    assert req_to_token.size(1) >= 1, "req_to_token has no columns"
    max_ctx = max(min(int(max_len_in_batch), req_to_token.size(1)) if max_len_in_batch else req_to_token.size(1), 1)
    if req_to_token.dtype in (torch.int32, torch.int64) and req_to_token.stride(1) == 1:
        # the kernel looks its row up itself: gathering the rows of 16 requests of up to 32768 tokens first took 17 us of 234
        table, gathered = req_to_token, 0
    else:
        # a table that it cannot read in place: only the rows and columns in use are copied, not the whole pool (int16,
        # 4096 x 32768, 16 requests of 2048 tokens: 423 us for the pool, 74 so); the kernel still says which rows exist
        table = req_to_token[:, :max_ctx].index_select(0, rows.clamp(0, req_to_token.size(0) - 1))
        if table.dtype not in (torch.int32, torch.int64):
            table = table.to(torch.int32 if table.element_size() < 4 and not table.is_floating_point() else torch.int64)
        gathered = 2
    lens = b_seq_len if b_seq_len.dtype in (torch.int32, torch.int64) else b_seq_len.to(torch.int64)
    lens = lens.contiguous()
    chunk = _pick_chunk(batch, hkv, max_ctx, 1)
    max_splits = (max_ctx + chunk - 1) // chunk
    lib = _lib.load()
    nfloats = lib.dlb_paged_decode_workspace_floats(batch, head, max(D, Dv), max_splits)
    partial = torch.empty(max(nfloats, 1), dtype=torch.float32, device=dev)
    status = _lib.status_word(dev)
    with _lib.on_device(dev):
        rc = lib.dlb_paged_decode_rows(
            q.data_ptr(), k_buffer.data_ptr(), v_buffer.data_ptr(), o.data_ptr(), table.data_ptr(), rows.data_ptr(),
            req_to_token.size(0), int(rows.dtype == torch.int64) + gathered, lens.data_ptr(),
            partial.data_ptr(), batch, head, hkv, D, Dv, 1, k_buffer.size(0), max_ctx,
            q.stride(0), q.stride(1), o.stride(0), o.stride(1),
            k_buffer.stride(0), k_buffer.stride(0), k_buffer.stride(1),
            v_buffer.stride(0), v_buffer.stride(0), v_buffer.stride(1),
            table.stride(0), int(table.dtype == torch.int64), int(lens.dtype == torch.int64),
            chunk, max_splits, -1, float(sm_scale), float(logit_cap) if logit_cap and logit_cap > 0 else -1.0,
            _lib.dtype_code(q), status.data_ptr(), _lib.stream_ptr(dev))
    _lib.check(rc, "decode_attention_fwd")
    return o
