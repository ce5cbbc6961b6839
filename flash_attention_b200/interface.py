"""Python call surface of the NVFP4 attention forward.

Mirrors ``flash_attn.cute.flash_attn_func`` of the reference
(flash_attn/cute/interface.py:1753-1792 -> FlashAttnFunc.forward :1576-1633 -> _flash_attn_fwd
:279-813): same positional surface, same tensor conventions ((batch, seqlen, heads, head_dim),
GQA map ``h_kv = h // (Hq // Hkv)``, ``softmax_scale=None -> 1/sqrt(D)``, bottom-right aligned
``causal``, returns ``(out, lse)`` with ``lse`` fp32 ``(B, Hq, Sq)`` or ``None``), same error
behaviour (``AssertionError`` for malformed tensors, ``NotImplementedError`` for features that are
not built), launch on the current CUDA stream with no host synchronisation.  The checks and the
launch itself are native (csrc/host.cpp): in Python they cost more than a decode step.

The reference asserts fp16/bf16 inputs (interface.py:370); this module is the branch an NVFP4
overload takes before that assert.  Operands arrive either as :class:`NVFP4Tensor` triples through
:func:`flash_attn_func`, or as raw tensors through :func:`flash_attn_fp4_func` whose scale
arguments follow the descale convention of the reference's FP8 path
(hopper/flash_attn_interface.py:81-83).  Output is bf16, as for the reference's quantised inputs
(hopper/flash_api.cpp:859-863).
"""
from __future__ import annotations

from typing import Callable, Optional, Tuple

import torch

from . import _lib
from .quant import NVFP4Tensor

VARIANT_AUTO, VARIANT_WS, VARIANT_WS64, VARIANT_DECODE = 0, 2, 3, 4


class DeviceStatus:
    """One device word per CUDA device that the kernels report bounded-wait expiry into.

    The word is checked lazily: :func:`check_status` reads it back (one small copy, which
    synchronises) and raises if a kernel gave up; the attention call itself never synchronises.
    A launch whose wait ran out leaves its outputs unwritten and returns normally, like any
    asynchronous CUDA failure: call :func:`check_status` wherever results are consumed on the host.
    The word keeps the first failure until it is read, but only the launch that recorded it stops
    early (the kernels compare a per-launch epoch), so later calls are not affected by a stale word.
    """
    _words = {}

    @classmethod
    def word(cls, device: torch.device) -> torch.Tensor:
        idx = device.index if device.index is not None else torch.cuda.current_device()
        w = cls._words.get(idx)
        if w is None:
            # one word per device also when several threads make their first call at once: its address is kept
            w = cls._words.setdefault(idx, torch.zeros(1, dtype=torch.int32, device=torch.device("cuda", idx)))
        return w


def check_status(device=None) -> None:
    """Raise ``RuntimeError`` if a kernel on ``device`` recorded a failure since the last check."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    w = DeviceStatus.word(device)
    v = int(w.item()) & 0xFFFFFFFF
    if v != 0:
        w.zero_()
        code, site, epoch, blk = v >> 24, (v >> 16) & 0xFF, (v >> 8) & 0xFF, v & 0xFF
        raise RuntimeError(f"fa4_nvfp4 kernel failure: code {code} (1 = bounded wait expired), "
                           f"wait site {site}, launch epoch {epoch}, block {blk} (mod 256)")


def flash_attn_fp4_func(
    q: torch.Tensor, k: torch.Tensor, v: torch.Tensor,
    q_sf: torch.Tensor, k_sf: torch.Tensor, v_sf: torch.Tensor,
    q_scale, k_scale, v_scale,
    softmax_scale: Optional[float] = None,
    causal: bool = False,
    return_lse: bool = False,
    out: Optional[torch.Tensor] = None,
    lse: Optional[torch.Tensor] = None,
    sf_layout: str = "linear",
    variant: int = VARIANT_AUTO,
    num_splits: int = 1,
    window_size: Tuple[Optional[int], Optional[int]] = (None, None),
    learnable_sink: Optional[torch.Tensor] = None,
    softcap: float = 0.0,
    seqused_k: Optional[torch.Tensor] = None,
    page_table: Optional[torch.Tensor] = None,
) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """NVFP4 attention forward.

    q (B,Sq,Hq,D/2), k (B,Sk,Hkv,D/2), v (B,Hkv,Dv,Skp/2): packed e2m1 bytes (V key-contiguous, its
    key axis padded with zeros to Skp = Sk rounded up to a multiple of 32; the quantisers do that).
    *_sf: e4m3 block scales, ``sf_layout="linear"``: (B,S,H,D/16) / (B,Hkv,Dv,Skp/16), converted
    to the tiled layout by a small kernel; ``"tiled"``: already (B,H,ceil(rows/128),column tiles,512), see ``sf_to_tiled``.
    *_scale: fp32 per-tensor scales.  Returns ``(out bf16 (B,Sq,Hq,Dv), lse fp32 (B,Hq,Sq) | None)``.

    ``num_splits``: 1 = one pass over K/V per query tile; k > 1 = split-KV with a combine kernel
    (the reference's ``num_splits``, interface.py:494-510), for short Sq against long Sk;
    0 = choose (split only when the query tiles alone leave most SMs idle).  Decode and append
    shapes (D = Dv = 128, Sq * Hq / Hkv <= 32, no window / sink / softcap) run the transposed
    decode kernel (``VARIANT_DECODE``: keys on the tile's lanes, grid = splits x Hkv x B); there
    ``num_splits=0`` is what a serving loop wants (about two CTAs per SM; with ``seqused_k`` over
    many keys the CTAs are then dealt by the lengths of the entries, in which an entry's bits depend on
    the other entries' lengths too).  A chosen count gives the bits of the entry computed alone.

    ``window_size=(left, right)``: local attention, query row i sees keys
    ``i + Sk - Sq - left <= j <= i + Sk - Sq + right`` (``None`` = unlimited; ``causal`` is
    ``right = 0``), the reference's semantics (flash_attn/cute/interface.py:256-276).

    ``learnable_sink``: (Hq,) logits that join every row's softmax normalisation (and the LSE)
    without contributing a value, the reference's argument of the same name (testing.py:406-416).

    ``softcap`` > 0: the scaled scores become ``softcap * tanh(scores / softcap)`` before masking
    (the reference's ``softcap``, interface.py:528-530 / testing.py:373-374), with the hardware
    ``tanh.approx`` as in the reference's kernel; one more transcendental per score.

    KV cache, the reference's ``seqused_k`` / ``page_table`` (interface.py:296-300, paged_kv.py):
    ``seqused_k`` (B,) int32: batch entry b attends to its first ``seqused_k[b]`` keys only (any
    value in 0..Sk; causal and window limits align to it).  ``page_table`` (B, pages_per_seq)
    int32: k, v and their scales are then a POOL of pages, k (num_pages, page_size, Hkv, D/2),
    v (num_pages, Hkv, Dv, page_size/2), scales per page in either layout, page_size a multiple
    of 128; the logical key length is ``pages_per_seq * page_size``.  Scale bytes of unused
    cache slots must not be NaN encodings (a zero-filled cache is fine).

    Built so far: D = Dv = 128 or 64, or (D, Dv) = (192, 128) (every feature but split-KV and the
    decode kernel); any Sq and Sk, as in the reference (partial last tiles are handled by
    zero-filled loads, a key-length mask and unstored rows).  Anything else raises ``NotImplementedError``
    before a launch.
    """
    win_left, win_right = window_size
    return _lib.host().fwd(q, k, v, q_sf, k_sf, v_sf, q_scale, k_scale, v_scale, softmax_scale, causal, return_lse,
                           out, lse, sf_layout, variant, num_splits, win_left, win_right, learnable_sink, softcap,
                           seqused_k, page_table)


def choose_decode_splits(B: int, Hkv: int, Sk: int, device=None) -> int:
    """Key splits of the decode kernel (grid = splits x Hkv x B; three CTAs fit an SM).

    The kernel streams K and V at the pace of HBM once about two CTAs per SM pull on it, so the
    count aims at 2 x SMs CTAs (more splits only add partials for the combine kernel), with at
    least two 128-key blocks per split.  When B x Hkv alone exceeds the 3 x SMs resident CTAs the
    grid runs in waves anyway: then the count (up to 4) that minimises waves x (blocks per split + 4
    blocks of fixed cost per CTA) evens out the last wave.  Measured on B200 (Hq 32, Hkv 8, us per
    call): B=4, Sk=32768: 9 or 13 splits 46, 18 splits 54; B=1, Sk=131072: 37 splits 50, 55 splits
    54; B=64, Sk=4096: 1 split 89, 2 splits 79."""
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    return _lib.host().choose_decode_splits(B, Hkv, Sk, sms)


def resolve_window(causal: bool, window_size) -> Tuple[bool, Optional[int], Optional[int]]:
    """(causal, left, right) after the reference's rules (flash_attn/cute/interface.py:256-276):
    causal sets right = 0; a window whose two limits sum to less than zero means no window;
    (None, 0) is plain causal.  One difference: the reference keeps a negative limit whose partner
    outweighs it (a band shifted off the diagonal, e.g. (-2, 5)); the C ABI encodes "no limit" as
    -1, so such windows raise ``NotImplementedError`` here instead."""
    return _lib.host().resolve_window(causal, *window_size)


def choose_num_splits(B: int, Sq: int, Sk: int, Hq: int, causal: bool, device) -> int:
    """Split count for ``num_splits=0``.

    1 unless the query tiles alone would leave more than half of the SMs idle.  Otherwise the
    count that minimises (waves of work items over the SMs) x (K/V blocks per item + 2 blocks of
    fixed cost per item), at least four blocks per split -- the efficiency search of the
    reference's heuristic (flash_attn/cute/interface.py:494-510) on this kernel's cost model.
    """
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    return _lib.host().choose_num_splits(B, Sq, Sk, Hq, sms)


def flash_attn_func(
    q, k, v,
    softmax_scale: Optional[float] = None,
    causal: bool = False,
    window_size: Tuple[Optional[int], Optional[int]] = (None, None),
    learnable_sink: Optional[torch.Tensor] = None,
    softcap: float = 0.0,
    num_splits: int = 1,
    pack_gqa: Optional[bool] = None,
    deterministic: bool = False,
    mask_mod: Optional[Callable] = None,
    full_block_cnt: Optional[torch.Tensor] = None,
    full_block_idx: Optional[torch.Tensor] = None,
    mask_block_cnt: Optional[torch.Tensor] = None,
    mask_block_idx: Optional[torch.Tensor] = None,
    block_size: Optional[Tuple[int, int]] = None,
    return_lse: bool = False,
):
    """Same signature as the reference's ``flash_attn_func`` (interface.py:1753-1772); q, k, v are
    :class:`NVFP4Tensor`.  Keyword arguments of features that are not built raise
    ``NotImplementedError``; ``pack_gqa`` and ``deterministic`` are accepted and ignored (the
    forward is deterministic, and query heads of a kv head share K/V through L2 instead of being
    packed into one tile)."""
    if not all(isinstance(t, NVFP4Tensor) for t in (q, k, v)):
        raise TypeError("flash_attn_func of this package takes NVFP4Tensor operands; "
                        "see quantize_qkv()")
    if mask_mod is not None or any(t is not None for t in (full_block_cnt, full_block_idx,
                                                           mask_block_cnt, mask_block_idx)):
        raise NotImplementedError("mask_mod / block sparsity is not built")
    if q.tiled or k.tiled or v.tiled or q.sf_tiled is not None or k.sf_tiled is not None or v.sf_tiled is not None:
        layout, q_sf, k_sf, v_sf = "tiled", q.tiled_sf(), k.tiled_sf(), v.tiled_sf()
    else:
        layout, q_sf, k_sf, v_sf = "linear", q.sf, k.sf, v.sf
    win_left, win_right = window_size
    # (_scale: a scale the quantiser has not delivered to the host yet is used where it is, on the device)
    return _lib.host().fwd(q.data, k.data, v.data, q_sf, k_sf, v_sf, q._scale, k._scale, v._scale, softmax_scale, causal,
                           return_lse, None, None, layout, VARIANT_AUTO, num_splits, win_left, win_right,
                           learnable_sink, softcap, None, None)


def measure_fp4_mma_rate(iters: int = 1 << 16, device=None, repeats: int = 3) -> dict:
    """Dense block-scaled e2m1 tensor-pipe rate of this GPU, measured.

    Launches one CTA per SM that issues ``iters`` 128x128x64 MMAs back to back from shared memory
    (``fa4_nvfp4_debug_mma_rate``) and times the launch with CUDA events.  Returns the best of
    ``repeats``: ``{"tflops", "clk_per_mma" (median over CTAs, in-kernel clocks), "ms", "sms"}``.
    The benchmark reports it beside the nominal dense-FP4 figure.
    """
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    clocks = torch.zeros(sms, dtype=torch.int64, device=device)
    status = DeviceStatus.word(device)
    stream = torch.cuda.current_stream(device)
    best = None
    for _ in range(repeats + 1):          # the first launch is the warm-up
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        _lib.check(_lib.lib().fa4_nvfp4_debug_mma_rate(iters, sms, clocks.data_ptr(), status.data_ptr(),
                                                      stream.cuda_stream), "fa4_nvfp4_debug_mma_rate")
        e1.record(stream)
        e1.synchronize()
        ms = e0.elapsed_time(e1)
        if best is None or ms < best:
            best = ms
    check_status(device)
    flops = sms * iters * 2.0 * 128 * 128 * 64
    return {"tflops": flops / (best * 1e-3) / 1e12, "ms": best, "sms": sms,
            "clk_per_mma": float(clocks.double().median().item()) / iters}


def measure_ex2_rate(iters: int = 1 << 12, device=None) -> dict:
    """Rate of the exponential unit of this GPU, measured (``fa4_nvfp4_debug_ex2_rate``): one CTA of
    16 warps per SM, 16 independent ``ex2.approx`` per thread and round.  Returns
    ``{"per_clk_per_sm" (median over CTAs), "sms"}``; the benchmark's exponential roofline uses it."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    clocks = torch.zeros(sms, dtype=torch.int64, device=device)
    scratch = torch.zeros(1, dtype=torch.float32, device=device)
    stream = torch.cuda.current_stream(device)
    for _ in range(2):                    # the first launch is the warm-up
        _lib.check(_lib.lib().fa4_nvfp4_debug_ex2_rate(iters, sms, clocks.data_ptr(), scratch.data_ptr(),
                                                      stream.cuda_stream), "fa4_nvfp4_debug_ex2_rate")
    torch.cuda.synchronize(device)
    clk = float(clocks.double().median().item())
    return {"per_clk_per_sm": 512.0 * iters * 16 / clk, "sms": sms}
