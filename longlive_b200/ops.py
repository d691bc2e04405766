"""torch.Tensor-level wrappers around the C-ABI entry points (device pointers in, nothing
allocated by the library).  Argument checks, output allocation and the call itself live in the compiled
binding (``csrc/binding.cpp``); the forms that only a multi-GPU group uses go through ctypes here."""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib

DEQ_FUSED, DEQ_PYTORCH, DEQ_TRITON = 0, 1, 2


def _stream(t: torch.Tensor) -> int:
    _lib.init_device(t.device.index if t.device.index is not None else torch.cuda.current_device())
    return torch.cuda.current_stream(t.device).cuda_stream


class DeviceTimeout(RuntimeError):
    """A bounded device-side wait gave up (``LLNV_E_TIMEOUT``): results of the affected step are invalid."""


def check_status(device=None) -> None:
    """Synchronise the current stream of ``device`` and raise ``DeviceTimeout`` if a kernel's bounded wait
    (an mbarrier wait, a peer barrier) gave up since the last check (``llnv_check_status``; clears the flag)."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    with torch.cuda.device(dev):
        rc = _lib.lib().llnv_check_status(torch.cuda.current_stream(dev).cuda_stream)
    if rc == -3:
        raise DeviceTimeout(_lib.lib().llnv_last_error().decode("utf-8", "replace"))
    _check(rc)


def _require_cuda(t: torch.Tensor, name: str) -> None:
    if not isinstance(t, torch.Tensor) or t.device.type != "cuda":
        raise ValueError(f"{name} must be a CUDA tensor (the NVFP4 path has no CPU implementation)")


def _check(rc: int) -> None:
    if rc != 0:
        msg = _lib.lib().llnv_last_error().decode("utf-8", "replace")
        raise RuntimeError(f"llnvfp4 error {rc}: {msg}")


def _seq(x):
    """The binding takes lists and tuples; any other iterable (a dictionary's values, a stacked tensor) is listed first."""
    return x if x is None or type(x) in (list, tuple) else list(x)


def _opt_int(x):
    return None if x is None else int(x)


def padded_rows(m: int) -> int:
    return (m + 127) // 128 * 128


def amax_bf16(x: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    _require_cuda(x, "x")
    assert x.dim() == 2 and x.dtype == torch.bfloat16 and x.stride(1) == 1
    if out is None:
        out = torch.empty(1, dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _check(_lib.lib().llnv_amax_bf16(x.data_ptr(), x.shape[0], x.shape[1], x.stride(0), out.data_ptr(), _stream(x)))
    return out


def _group_args(group):
    """(slot pointer table, signal pointer table, rank, world, epoch pointer) of a peer arena (``sp.PeerArena``)."""
    return (_ptr_table([b + group.SIGNAL_BYTES for b in group.base]), _ptr_table(group.base), group.rank, group.world,
            group.epoch.data_ptr())


def quantize_nvfp4(x: torch.Tensor, rule_id: int, amax: torch.Tensor | None = None, codes=None, sf=None,
                   amax_given: bool | None = None, group=None):
    """bf16 [M, K] (K % 64 == 0, unit column stride) -> (codes [Mp, K/2] u8, sf [Mp*K/16] e4m3, amax [1] f32).

    A contiguous 3-D ``x`` [shards, M, K / shards] is read as the column-sharded form of the [M, K]
    matrix (``llnv_quantize_nvfp4_ex``).

    ``amax`` is the fp32 tensor-scale buffer.  With ``amax_given`` (default: true when a buffer is
    passed) it is read as the scale; otherwise it is computed on the device into that buffer (or a
    new one).  ``codes`` / ``sf`` may be preallocated slot buffers (KV cache) written in place.
    ``group`` (a ``sp.PeerArena``): ``amax`` holds this rank's amax of its shard; the quantize kernel MAX-reduces it over
    the group before its first block and leaves the group maximum in ``amax`` (``llnv_quantize_nvfp4_group``).
    """
    if group is None:
        return _lib.native().quantize(x, rule_id, amax, codes, sf, amax_given)
    _require_cuda(x, "x")
    shards = 1
    if x.dim() == 3 and x.dtype == torch.bfloat16 and x.is_contiguous():
        shards, m, ks = x.shape
        k, ldx = shards * ks, ks
    elif x.dim() != 2 or x.dtype not in (torch.bfloat16, torch.float16):
        raise RuntimeError("quantize_nvfp4 expects a 2-D bfloat16 or float16 tensor (or a contiguous bfloat16 [shards, M, K/shards] one)")
    else:
        if x.stride(1) != 1:
            x = x.contiguous()
        m, k = x.shape
        ldx = x.stride(0)
    if x.dtype == torch.float16:
        raise ValueError("the group form takes bfloat16 input")
    if amax is None or amax_given is False:
        raise ValueError("the group form needs this rank's amax in `amax`")
    codes, sf, amax = _quant_outputs(x, m, k, codes, sf, amax)
    with torch.cuda.device(x.device):
        _check(_lib.lib().llnv_quantize_nvfp4_group(x.data_ptr(), m, k, ldx, rule_id, codes.data_ptr(), sf.data_ptr(),
                                                    amax.data_ptr(), shards, *_group_args(group), _stream(x)))
    return codes, sf, amax


def _quant_outputs(x, m, c, codes, sf, amax):
    mp = padded_rows(m)
    if codes is None:
        codes = torch.empty((mp, c // 2), dtype=torch.uint8, device=x.device)
    if sf is None:
        sf = torch.empty(mp * c // 16, dtype=torch.float8_e4m3fn, device=x.device)
    if amax is None:
        amax = torch.empty(1, dtype=torch.float32, device=x.device)
    return codes, sf, amax


def adaln_quantize_nvfp4(x, scale, shift, frame_rows, rule_id, eps=1e-6, add_one=True, *, want_y=False, codes=None,
                         sf=None, amax=None, row_stats=None, row_offset=0, phase=0, y_only=False, group=None):
    """LayerNorm(no affine) -> (1 + scale[f]) * x + shift[f] (bf16 rounding points of the reference)
    fused with the NVFP4 quantize of the result.  x: bf16 [M, C]; scale/shift: bf16 [F, C] views
    (row stride free).  Returns (codes, sf, amax, y or None); with ``y_only`` nothing is quantized
    (codes and sf are None) and only y is produced.  ``group`` (a ``sp.PeerArena``): the tensor amax is MAX-reduced
    over the group inside the quantize kernel (``llnv_adaln_quantize_nvfp4_group``)."""
    if group is None:
        return _lib.native().adaln_quantize(x, scale, shift, int(frame_rows), rule_id, eps, add_one, want_y, codes, sf, amax, row_stats,
                                            int(row_offset), int(phase), y_only)
    _require_cuda(x, "x")
    if x.dim() != 2 or x.dtype != torch.bfloat16 or x.stride(1) != 1:
        raise RuntimeError("adaln_quantize_nvfp4 expects a 2-D bfloat16 tensor with unit column stride")
    if scale.dim() != 2 or shift.dim() != 2 or scale.stride(1) != 1 or shift.stride(1) != 1 or scale.stride(0) != shift.stride(0):
        raise RuntimeError("scale and shift must be [frames, C] views with the same row stride")
    if want_y or y_only or phase != 0:
        raise ValueError("the group form runs both passes and produces no y")
    m, c = x.shape
    codes, sf, amax = _quant_outputs(x, m, c, codes, sf, amax)
    if row_stats is None:
        row_stats = torch.empty(2 * max(m, 1), dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _check(_lib.lib().llnv_adaln_quantize_nvfp4_group(
            x.data_ptr(), m, c, x.stride(0), scale.data_ptr(), shift.data_ptr(), scale.stride(0), int(frame_rows), float(eps),
            1 if add_one else 0, rule_id, codes.data_ptr(), sf.data_ptr(), amax.data_ptr(), row_stats.data_ptr(), int(row_offset),
            *_group_args(group), _stream(x)))
    return codes, sf, amax, None


def layernorm_quantize_nvfp4(x, weight, bias, rule_id, eps=1e-6, *, want_y=False, codes=None, sf=None, amax=None,
                             row_stats=None, phase=0, group=None):
    """Affine LayerNorm fused with the NVFP4 quantize of its output.  Returns (codes, sf, amax, y or None).
    ``group`` (a ``sp.PeerArena``): the tensor amax is MAX-reduced over the group inside the quantize kernel."""
    if group is None:
        return _lib.native().layernorm_quantize(x, weight, bias, rule_id, eps, want_y, codes, sf, amax, row_stats, int(phase))
    _require_cuda(x, "x")
    if x.dim() != 2 or x.dtype != torch.bfloat16 or x.stride(1) != 1:
        raise RuntimeError("layernorm_quantize_nvfp4 expects a 2-D bfloat16 tensor with unit column stride")
    if want_y or phase != 0:
        raise ValueError("the group form runs both passes and produces no y")
    m, c = x.shape
    codes, sf, amax = _quant_outputs(x, m, c, codes, sf, amax)
    if row_stats is None:
        row_stats = torch.empty(2 * max(m, 1), dtype=torch.float32, device=x.device)
    with torch.cuda.device(x.device):
        _check(_lib.lib().llnv_layernorm_quantize_nvfp4_group(
            x.data_ptr(), m, c, x.stride(0), weight.data_ptr(), bias.data_ptr(), float(eps), rule_id, codes.data_ptr(),
            sf.data_ptr(), amax.data_ptr(), row_stats.data_ptr(), *_group_args(group), _stream(x)))
    return codes, sf, amax, None


def rmsnorm_rope(x, weight=None, cos=None, sin=None, eps=1e-6, *, out=None, out_smooth=None, want_smooth=False,
                 amax_out=None, want_amax=False, shards=1):
    """RMSNorm (if ``weight``) -> per-head RoPE (if ``cos``/``sin``, fp32 [S, 64]) on bf16 [S, C];
    optionally the k_smooth copy and max|out|.  Returns (out, out_smooth or None, amax or None).
    With ``shards`` > 1 the outputs are contiguous [shards, S, C / shards] tensors (head-sharded)."""
    return _lib.native().rmsnorm_rope(x, weight, cos, sin, eps, out, out_smooth, want_smooth, amax_out, want_amax, shards)


def quantize_nvfp4_pair(x0, x1, rule_id, q0, q1, amax_given=True):
    """Quantize two bf16 [M, K] tensors of the same shape in one launch into the preallocated
    QuantizedTensor-like targets q0 / q1 (``values``, ``scale_factors``, ``amax``)."""
    _lib.native().quantize_pair(x0, x1, rule_id, q0.values, q0.scale_factors, q0.amax, q1.values, q1.scale_factors, q1.amax, amax_given)


def _ptr_table(ptrs):
    arr = (C.c_void_p * len(ptrs))(*[int(p) for p in ptrs])
    return arr


def rmsnorm_rope_scatter(x, weight, cos, sin, eps, out_ptrs, ldo, smooth_ptrs=None, lds=0, amax_out=None):
    """``rmsnorm_rope`` whose head shard r is stored at ``out_ptrs[r]`` (and ``smooth_ptrs[r]``): raw
    device addresses, possibly on other GPUs of the node.  See ``llnv_rmsnorm_rope_scatter``."""
    _require_cuda(x, "x")
    s, c = x.shape
    shards = len(out_ptrs)
    with torch.cuda.device(x.device):
        _check(_lib.lib().llnv_rmsnorm_rope_scatter(
            x.data_ptr(), s, c, x.stride(0), weight.data_ptr() if weight is not None else None, float(eps),
            cos.data_ptr() if cos is not None else None, sin.data_ptr() if sin is not None else None,
            _ptr_table(out_ptrs), ldo, _ptr_table(smooth_ptrs) if smooth_ptrs is not None else None, lds,
            amax_out.data_ptr() if amax_out is not None else None, shards, _stream(x)))


def rmsnorm_rope_qk(xq, wq, q_ptrs, ldq, xk, wk, k_ptrs, ldk, k_smooth_ptrs, lds, k_amax, cos, sin, eps):
    """The q and the k prologue of a block in one launch (``llnv_rmsnorm_rope_qk``); outputs are raw
    device addresses, one per head shard."""
    _lib.native().rmsnorm_rope_qk(xq, wq, _seq(q_ptrs), ldq, xk, wk, _seq(k_ptrs), ldk, _seq(k_smooth_ptrs), lds, k_amax, cos, sin, eps)


def scatter_2d(src, src_shard_bytes, dst_ptrs, dst_pitch, rows, row_bytes):
    """Push ``rows`` x ``row_bytes`` blocks of the 2-D tensor ``src`` (block r starts r * src_shard_bytes
    bytes in) to the raw device addresses ``dst_ptrs`` (possibly peer memory).  See ``llnv_scatter_2d``."""
    _require_cuda(src, "src")
    with torch.cuda.device(src.device):
        _check(_lib.lib().llnv_scatter_2d(src.data_ptr(), src_shard_bytes, src.stride(0) * src.element_size(), _ptr_table(dst_ptrs),
                                          dst_pitch, rows, row_bytes, len(dst_ptrs), _stream(src)))


_LINEAR_ACT = {None: 0, "none": 0, "gelu_tanh": 1, "silu": 2}


def linear_bf16(x, w, bias=None, act=None, out=None):
    """``act(x @ w.T + bias)`` for bf16 ``x`` [M, K], ``w`` [N, K], ``bias`` [N] on the tcgen05 bf16 kernel
    (``llnv_linear_bf16``): the Linear of the layers the reference keeps in bf16.  ``act``: None,
    "gelu_tanh" or "silu".  Unit column strides; K, N and the row strides multiples of 8."""
    if act not in _LINEAR_ACT:
        _require_cuda(x, "x")
        raise ValueError(f"act must be one of {sorted(k for k in _LINEAR_ACT if k)} or None")
    return _lib.native().linear_bf16(x, w, bias, _LINEAR_ACT[act], out)


def patchify(latent, channels_first=True, out=None):
    """bf16 latent [C, F, H, W] (or [F, C, H, W] with ``channels_first=False``) -> tokens [F*H/2*W/2, 4*C],
    features ordered (c, kh, kw): the input of the patch embedding (``llnv_patchify``)."""
    return _lib.native().patchify(latent, channels_first, out)


def unpatchify(tokens, out, channels_first=True):
    """Tokens [F*h*w, 4*C] (features (c, kh, kw)) -> the bf16 latent ``out`` [C, F, 2h, 2w] (or [F, C, 2h, 2w]);
    the inverse of ``patchify`` (``llnv_unpatchify``)."""
    return _lib.native().unpatchify(tokens, out, channels_first)


def peer_barrier(signal_ptrs, rank, epoch):
    """Stream-ordered barrier over the GPUs whose signal areas are ``signal_ptrs`` (``llnv_peer_barrier``)."""
    with torch.cuda.device(epoch.device):
        _check(_lib.lib().llnv_peer_barrier(_ptr_table(signal_ptrs), rank, len(signal_ptrs), epoch.data_ptr(), _stream(epoch)))


def peer_allreduce_max(vals, slot_ptrs, signal_ptrs, rank, epoch):
    """In-place MAX all-reduce of a small fp32 tensor over the GPUs of a peer arena (``llnv_peer_allreduce_max``)."""
    with torch.cuda.device(vals.device):
        _check(_lib.lib().llnv_peer_allreduce_max(vals.data_ptr(), vals.numel(), _ptr_table(slot_ptrs), _ptr_table(signal_ptrs), rank,
                                                  len(signal_ptrs), epoch.data_ptr(), _stream(vals)))


SPLIT_TAIL = -1          # LLNV_ATTN_SPLIT_TAIL: cut the tiles of the last partial wave once (see include/llnvfp4.h)


def attention_workspace_bytes(lq, lk, heads, key_splits=None):
    """Bytes of workspace ``attention_bf16`` uses, and ``attention_nvfp4kv`` needs, for this shape (0 when the call is not split);
    ``key_splits`` None = what the library proposes for the current device."""
    lib = _lib.lib()
    if key_splits is None:
        key_splits = lib.llnv_attention_key_splits(lq, lk, heads)
    return int(lib.llnv_attention_workspace_bytes(lq, heads, key_splits)) if (key_splits > 1 or key_splits == SPLIT_TAIL) else 0


def attention_nvfp4kv_workspace_bytes(lq, blocks, block_tokens, l_cur, heads, key_splits=None):
    """Bytes of workspace ``attention_nvfp4kv`` uses for ``blocks`` cached blocks and a current chunk of ``l_cur`` tokens
    (``llnv_attention_nvfp4kv_workspace_bytes``)."""
    lib = _lib.lib()
    if key_splits is None:
        key_splits = lib.llnv_attention_key_splits(lq, blocks * block_tokens + l_cur, heads)
    return int(lib.llnv_attention_nvfp4kv_workspace_bytes(lq, heads, key_splits, blocks, block_tokens))


def attention_bf16(q, k, v, heads, scale=None, out=None, key_splits=None, out_amax=None, workspace=None):
    """softmax(q k^T * scale) v per head, non-causal.  q: bf16 [Lq, heads*128]; k, v: bf16 [Lk, heads*128]
    (row strides free, unit column stride).  Returns bf16 [Lq, heads*128].  ``key_splits`` > 1 splits
    the key window over several CTAs per query tile (default: what the library proposes for the
    device, 1 unless the tiles alone leave most SMs idle).  ``out_amax`` (fp32 [1]) receives max |out|.
    ``workspace``: a uint8 tensor for the partial results of a split call (``attention_workspace_bytes``); allocated
    per call when omitted."""
    return _lib.native().attention_bf16(q, k, v, heads, scale, out, _opt_int(key_splits), out_amax, workspace)


def attention_nvfp4kv(q, k_blocks, v_blocks, block_tokens, k_cur, v_cur, heads, scale=None, out=None, key_splits=None,
                      out_amax=None, e2m1_max=6.0, e4m3_max=256.0, workspace=None):
    """Chunk attention over [cached NVFP4 blocks ... | current chunk (bf16)] (``llnv_attention_nvfp4kv``): the cached part is
    expanded to bf16 in the workspace and attended from there, the current chunk is read in place.  ``k_blocks`` / ``v_blocks``:
    cache blocks oldest first, each with ``values`` (uint8 [rows_padded, 64]), ``scale_factors`` and ``amax`` (a
    ``QuantizedTensor`` of ``block_tokens * heads`` rows of 128 channels, token-major / head-minor).  ``k_cur`` / ``v_cur``: bf16
    [L_cur, heads*128] (or None when the window is the cache alone).  Result: bf16 [Lq, heads*128], equal bit
    for bit to dequantizing the blocks into a window and calling ``attention_bf16`` on it.
    ``workspace``: a uint8 tensor of ``attention_nvfp4kv_workspace_bytes``, allocated per call when omitted; one that holds the
    partial results of a split call alone (``attention_workspace_bytes``, any size for an unsplit one) has the blocks decoded inside
    the attention kernel, which is slower on long windows and takes no memory for them."""
    return _lib.native().attention_nvfp4kv(q, _seq(k_blocks), _seq(v_blocks), int(block_tokens), k_cur, v_cur, heads, scale, out,
                                           _opt_int(key_splits), out_amax, e2m1_max, e4m3_max, workspace)


def dequantize_nvfp4(codes, sf, amax, rows, cols, cols_padded, dtype, e2m1_max, e4m3_max, rounding=DEQ_PYTORCH):
    return _lib.native().dequantize(codes, sf, amax, rows, cols, cols_padded, dtype, e2m1_max, e4m3_max, rounding)


def kv_dequant(values, scale_factors, amax, num_heads, block_token_size, dtype, e2m1_max, e4m3_max,
               rounding=DEQ_FUSED, out=None):
    if not isinstance(dtype, torch.dtype):
        raise ValueError(f"Unsupported fused KV dequant dtype: {dtype}")
    return _lib.native().kv_dequant(_seq(values), _seq(scale_factors), _seq(amax), num_heads, block_token_size, dtype, e2m1_max, e4m3_max, rounding, out)


def gemm_nvfp4(a_codes, a_sf, a_amax, a_rule, b_codes, b_sf, b_amax, b_rule, m, n, k, *, out=None, alpha=None,
               bias=None, act=0, residual=None, gate=None, frame_rows=0, out_amax=None, row_offset=0, tile=0,
               requant=None, requant_amax=None, store_out=True):
    """``epilogue(alpha * A @ B^T)`` -> bf16 [m, n]; see ``llnv_gemm_nvfp4`` in include/llnvfp4.h.
    ``tile``: 0 = tiling chosen by shape, 128 / 192 / 256 = that tile width, 2 = CTA-pair kernel.
    ``requant`` = (codes, sf) buffers: the epilogue also writes the NVFP4 form of the result (4-over-6 MSE rule)
    under the tensor amax ``requant_amax`` (fp32 [1], known before the call); with ``store_out=False`` the bf16
    result itself is not written and None is returned."""
    q_codes, q_sf = requant if requant is not None else (None, None)
    frame_rows, row_offset = (int(frame_rows), int(row_offset)) if gate is not None else (0, 0)        # read with a gate only
    return _lib.native().gemm(a_codes, a_sf, a_amax, a_rule, b_codes, b_sf, b_amax, b_rule, m, n, k, out, alpha, bias, int(act), residual, gate,
                              frame_rows, out_amax, row_offset, int(tile), q_codes, q_sf, requant_amax if requant is not None else None, store_out)


def gemm_nvfp4_grouped(a_codes, a_sf, a_amax, a_rule, b_codes, b_sf, b_amax, b_rule, m, n_each, k, outs, *, bias=None, act=0,
                       out_amax=None):
    """Two or three Linears sharing their input in one launch (``llnv_gemm_nvfp4_grouped``): ``b_codes`` /
    ``b_sf`` are the weights concatenated along N, ``b_amax`` an fp32 tensor with one amax per weight,
    ``outs`` the output tensors (bf16 [m, n_each], any row stride), ``out_amax`` a list of fp32 [1]
    tensors or None per output."""
    _lib.native().gemm_grouped(a_codes, a_sf, a_amax, a_rule, b_codes, b_sf, b_amax, b_rule, m, n_each, k, _seq(outs), bias, int(act), _seq(out_amax))
    return outs
