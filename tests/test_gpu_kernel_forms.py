"""The branches of the dispatch and of the host path at the sizes where they can go wrong: the edge between
the narrow and the wide window form, more tiles than CTAs with tiles that have no rows between them, tile
lists longer than a CTA's table, the decode kernel's ring depths and the two ways its splits are merged, and
the quantiser's small, unaligned and strided inputs."""
import ctypes
import math

import numpy as np
import pytest
import torch

import flash_attention_b200 as fa
from flash_attention_b200 import _lib
from flash_attention_b200.interface import DeviceStatus
from oracle import nvfp4_oracle as orc
from tests.helpers import assert_parity, make_qkv, oracles
from tests.test_zz_no_alloc import _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128, 192])
@pytest.mark.parametrize("window", [(256, 0), (257, 0), (128, 128), (0, 0), (1, 300)])
def test_window_forms_over_several_tiles_per_cta(cuda_device, window, D):
    q, k, v = make_qkv(2, 430, 430, 24, 2, D, seed=3, device=cuda_device)
    if D == 192:
        v = v[..., :128].contiguous()
    Q, K, V = fa.quantize_qkv(q, k, v)
    out, lse = fa.flash_attn_func(Q, K, V, window_size=window, return_lse=True)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert_parity(out, lse, *oracles(Q, K, V, False, window=window))


@pytest.mark.parametrize("Sk", [900, 500])       # 500: the first tiles see nothing and take no accumulator
@pytest.mark.parametrize("window", [(0, 0), (127, 0), (255, 1)])
def test_two_accumulators_in_turn(cuda_device, window, Sk):
    """Head dim 64, narrow windows, more than three tiles of one to eight steps per CTA; windows whose limits cut a warp's
    halves of 32 keys and others that leave them whole."""
    q, k, v = make_qkv(1, 900, Sk, 64, 4, 64, seed=6, device=cuda_device)
    Q, K, V = fa.quantize_qkv(q, k, v)
    out, lse = fa.flash_attn_func(Q, K, V, window_size=window, return_lse=True)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert_parity(out, lse, *oracles(Q, K, V, False, window=window))


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("lens", [[700, 1, 130, 390, 5, 700, 64, 257, 129, 31],      # a slot per row block of the longest
                                  [1025, 1, 130, 1300, 5, 128, 64, 257, 129, 31, 0, 897],   # only the tiles that exist
                                  [2000] + [17] * 200], ids=["slots", "existing", "many"])
def test_packed_batch_of_unequal_lengths(cuda_device, lens, causal):
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=cuda_device)
    q, k, v = (t[0] for t in make_qkv(1, sum(lens), sum(lens), 8, 2, 128, seed=4, device=cuda_device))
    Q, K, V, cu_v = fa.quantize_varlen_qkv(q, k, v, cu)
    out, lse = fa.flash_attn_varlen_fp4_func(Q.data[0], K.data[0], V.data[0], Q.sf[0], K.sf[0], V.sf[0], Q.scale, K.scale,
                                             V.scale, cu, cu, cu_seqlens_v=cu_v, max_seqlen_q=max(lens),
                                             max_seqlen_k=max(lens),
                                             causal=causal, return_lse=True)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    for i, n in list(enumerate(lens))[:14]:
        if n == 0:
            continue
        a, b, s0 = int(cu[i]), int(cu[i + 1]), int(cu_v[i])
        s1 = s0 + (n + 31) // 32 * 32
        o, l = fa.flash_attn_fp4_func(
            Q.data[:, a:b], K.data[:, a:b], V.data[..., s0 // 2:s1 // 2].contiguous(), Q.sf[:, a:b].contiguous(),
            K.sf[:, a:b].contiguous(), V.sf[..., s0 // 16:s1 // 16].contiguous(), Q.scale, K.scale, V.scale, causal=causal,
            return_lse=True, variant=fa.VARIANT_WS64)
        assert torch.equal(out[a:b], o[0]) and torch.equal(lse[:, a:b], l[0]), i


def test_tile_list_longer_than_the_table_of_a_cta(cuda_device):
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    Hq, Sq = 256, 16
    B = 768 * sms // Hq + 20                      # a second launch with a partial round
    g = torch.Generator(device=cuda_device).manual_seed(5)
    q, k, v = (torch.randn(B, S, H, 64, generator=g, device=cuda_device, dtype=torch.bfloat16)
               for S, H in ((Sq, Hq), (96, 8), (96, 8)))
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    out, _ = fa.flash_attn_func(Q, K, V, causal=True)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    for b in (0, B // 2, B - 3, B - 1):
        part = [fa.NVFP4Tensor(t.data[b:b + 1], t.sf[b:b + 1], t.scale, is_v=t.is_v) for t in (Q, K, V)]
        assert torch.equal(out[b:b + 1], fa.flash_attn_func(*part, causal=True)[0]), b


@pytest.mark.parametrize("B,S,H,D,offset", [(1, 1, 1, 64, 0), (1, 333, 4, 128, 0), (2, 129, 3, 192, 0),
                                            (3, 700, 16, 128, 0), (1, 200, 4, 64, 8)])
def test_quantiser_against_the_oracle(cuda_device, B, S, H, D, offset):
    """Small tensors (one row per work item), large ones (four), and views whose 32-byte pieces are only
    16-byte aligned; the scale is fetched from the device when it is read."""
    g = torch.Generator().manual_seed(6)
    base = torch.randn(B, S, H + 1, D + 8, generator=g).bfloat16().to(cuda_device)
    x = base[:, :, :H, offset:offset + D]
    Q, K, V = fa.quantize_qkv_fused(x, x, x)
    want = orc.quantize_nvfp4(x.float().cpu().numpy())
    for t in (Q, K):
        assert t.scale == want.scale
        assert np.array_equal(t.data.cpu().numpy(), want.data) and np.array_equal(t.sf.cpu().numpy(), want.sf)
        lin = np.transpose(want.sf, (0, 2, 1, 3))
        assert np.array_equal(t.sf_tiled.cpu().numpy(), orc.sf_linear_to_tiled(lin, 1))
    padded = torch.nn.functional.pad(x.float().cpu(), (0, 0, 0, 0, 0, -S % 32)).permute(0, 2, 3, 1).numpy()
    want_v = orc.quantize_nvfp4(padded)
    assert np.array_equal(V.data.cpu().numpy(), want_v.data) and np.array_equal(V.sf.cpu().numpy(), want_v.sf)
    assert np.array_equal(V.sf_tiled.cpu().numpy(), orc.sf_linear_to_tiled(want_v.sf, 2))


def test_scales_on_the_device_give_the_bits_of_scales_on_the_host(cuda_device):
    q, k, v = make_qkv(1, 200, 300, 4, 2, 128, seed=7, device=cuda_device)
    for kw in ({"causal": True}, {"softcap": 5.0}, {"num_splits": 2}):
        lazy = fa.flash_attn_func(*fa.quantize_qkv_fused(q, k, v), return_lse=True, **kw)
        ops = fa.quantize_qkv_fused(q, k, v)
        assert all(isinstance(t.scale, float) for t in ops)
        known = fa.flash_attn_func(*ops, return_lse=True, **kw)
        assert torch.equal(lazy[0], known[0]) and torch.equal(lazy[1], known[1]), kw


@pytest.mark.parametrize("layout", ["linear", "tiled"])
@pytest.mark.parametrize("Sq", [1, 2, 4, 8])
@pytest.mark.parametrize("B,splits", [(8, 1), (8, 2), (8, 8), (8, 9), (8, 19), (120, 2)],
                         ids=["deep", "deep2", "deep8", "deep9combined", "shallow19", "clusters_do_not_fit"])
def test_decode_ring_depths_and_merges(cuda_device, B, splits, Sq, layout):
    """Ragged entries with none, one, and odd and even numbers of key blocks (the two or four softmax warpgroups take
    them in turn), in the deep ring (at least four entries, up to two CTAs an SM) and the shallow one, merged
    inside a cluster (up to eight splits that fit at once) or by the combine kernel, with 4, 8, 16 and 32 rows, from
    scales that the kernel tiles itself and from tiled ones: the bits of the entry alone, which runs the shallow
    ring, and the oracle's values."""
    lens = [0, 1, 128, 129, 300, 640, 641, 1500] * (B // 8)
    q, k, v = make_qkv(B, Sq, 1536, 8, 2, 128, seed=8, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    sf = [t.tiled_sf() if layout == "tiled" else t.sf for t in (Q, K, V)]

    def run(b0, b1):
        return fa.flash_attn_fp4_func(*(t.data[b0:b1] for t in (Q, K, V)), *(t[b0:b1] for t in sf), Q.scale,
                                      K.scale, V.scale, causal=True, return_lse=True, seqused_k=used[b0:b1],
                                      num_splits=splits, sf_layout=layout)

    out, lse = run(0, B)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    for b in list(range(8)) + [B - 1]:
        o, l = run(b, b + 1)
        assert torch.equal(out[b:b + 1], o) and torch.equal(lse[b:b + 1], l), lens[b]
    n = lens[7]
    ops = [fa.NVFP4Tensor(Q.data[7:8], Q.sf[7:8], Q.scale), fa.NVFP4Tensor(K.data[7:8, :n], K.sf[7:8, :n], K.scale),
           fa.NVFP4Tensor(V.data[7:8, ..., :(n + 31) // 32 * 16], V.sf[7:8, ..., :(n + 31) // 32 * 2], V.scale, is_v=True)]
    assert_parity(out[7:8], lse[7:8], *oracles(*ops, True, num_splits=splits, variant=fa.VARIANT_DECODE))


@pytest.mark.parametrize("Sq", [1, 2, 4, 8])
@pytest.mark.parametrize("splits", [0, 1, 3, 9], ids=["chosen", "one", "cluster", "combine"])
def test_decode_of_a_paged_batch_with_tiled_scales(cuda_device, splits, Sq):
    """A serving cache: five entries of unequal lengths in a shuffled pool whose scales are kept tiled, 4 to 32 rows: the
    bits of a contiguous cache, and every entry against the oracle on its own keys."""
    lens, page, Sk = [700, 1, 1536, 129, 900], 256, 1536
    B, pages = len(lens), Sk // 256
    q, k, v = make_qkv(B, Sq, Sk, 8, 2, 128, seed=17, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    g = torch.Generator().manual_seed(18)
    table = torch.randperm(B * pages + 2, generator=g)[:B * pages].reshape(B, pages)
    pool = [torch.full((B * pages + 2, *shape), fill, dtype=torch.uint8, device=cuda_device)
            for shape, fill in (((page, 2, 64), 0x77), ((2, 128, page // 2), 0x77), ((2, page // 128, 2, 512), 0x7f),
                                ((2, 1, 2 * (page // 128), 512), 0x7f))]
    for b in range(B):
        for j in range(pages):
            at, k0, t0 = int(table[b, j]), j * page, j * (page // 128)
            pool[0][at] = K.data[b, k0:k0 + page]
            pool[1][at] = V.data[b, ..., k0 // 2:(k0 + page) // 2]
            pool[2][at] = K.tiled_sf()[b, :, t0:t0 + page // 128]
            pool[3][at] = V.tiled_sf()[b, :, :, 2 * t0:2 * (t0 + page // 128)]
    kw = {"causal": True, "return_lse": True, "seqused_k": used, "num_splits": splits, "sf_layout": "tiled"}
    scales = (Q.scale, K.scale, V.scale)
    out, lse = fa.flash_attn_fp4_func(Q.data, pool[0], pool[1], Q.tiled_sf(), pool[2], pool[3], *scales,
                                      page_table=table.to(torch.int32).to(cuda_device), **kw)
    flat = fa.flash_attn_fp4_func(Q.data, K.data, V.data, Q.tiled_sf(), K.tiled_sf(), V.tiled_sf(), *scales, **kw)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert torch.equal(out, flat[0]) and torch.equal(lse, flat[1])
    n_splits = splits or fa.interface.choose_decode_splits(B, 2, Sk, cuda_device)
    for b, n in enumerate(lens):
        ops = [fa.NVFP4Tensor(Q.data[b:b + 1], Q.sf[b:b + 1], Q.scale), fa.NVFP4Tensor(K.data[b:b + 1, :n], K.sf[b:b + 1, :n], K.scale),
               fa.NVFP4Tensor(V.data[b:b + 1, ..., :(n + 31) // 32 * 16], V.sf[b:b + 1, ..., :(n + 31) // 32 * 2], V.scale, is_v=True)]
        assert_parity(out[b:b + 1], lse[b:b + 1], *oracles(*ops, True, num_splits=n_splits, variant=fa.VARIANT_DECODE))


@pytest.mark.parametrize("Sq,Sk,splits", [(1, 2048, 4), (1, 2048, 9), (100, 2048, 4), (100, 4096, 9)],
                         ids=["decode_cluster", "decode_combine", "prefill_cluster", "prefill_combine"])
def test_split_calls_replay_from_a_cuda_graph(cuda_device, Sq, Sk, splits):
    q, k, v = make_qkv(2, Sq, Sk, 8, 2, 128, seed=9, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    call = lambda: fa.flash_attn_fp4_func(Q.data, K.data, V.data, Q.sf, K.sf, V.sf, Q.scale, K.scale, V.scale, causal=True,
                                          return_lse=True, num_splits=splits)
    first = [t.clone() for t in call()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out, lse = call()
    Q.data.bitwise_xor_(0x88)                       # other operands in the same buffers: every sign of q
    second = call()
    assert not torch.equal(first[0], second[0])
    graph.replay()
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert torch.equal(out, second[0]) and torch.equal(lse, second[1])


def _attend(Q, K, V, **kw):
    out, lse = fa.flash_attn_fp4_func(Q.data, K.data, V.data, Q.sf, K.sf, V.sf, Q.scale, K.scale, V.scale, return_lse=True, **kw)
    torch.cuda.synchronize()
    fa.check_status(Q.data.device)
    return out, lse


@pytest.mark.parametrize("D", [64, 128, 192])
@pytest.mark.parametrize("Sq,Sk", [(300, 200), (130, 515), (64, 65), (257, 257), (97, 64)])
def test_steps_in_which_a_warp_sees_no_key(cuda_device, Sq, Sk, D):
    """The cache form leaves the work of such steps out, the plain one masks it: the same bits, also for rows that
    see nothing at all (Sq > Sk)."""
    q, k, v = make_qkv(2, max(Sq, Sk), max(Sq, Sk), 4, 2, D, seed=11, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q[:, :Sq], k[:, :Sk], v[:, :Sk, :, :min(D, 128)])
    plain = _attend(Q, K, V, causal=True, variant=fa.VARIANT_WS64)
    used = torch.full((2,), Sk, dtype=torch.int32, device=cuda_device)
    cached = _attend(Q, K, V, causal=True, variant=fa.VARIANT_WS64, seqused_k=used)
    assert torch.equal(plain[0], cached[0]) and torch.equal(plain[1], cached[1])


@pytest.mark.parametrize("D", [64, 128, 192])
@pytest.mark.parametrize("window", [(None, None), (100, 0), (300, 0)], ids=["none", "narrow", "wide"])
@pytest.mark.parametrize("used", [None, 333], ids=["dense", "cache"])
def test_soft_cap_in_every_form(cuda_device, used, window, D):
    """Bound: the hardware tanh moves a score by up to softcap log2(e) 2^-11 in the exponent, and with it P values
    over rounding boundaries of the model (rel-RMS 0.05, as in the parity tests of the cap)."""
    q, k, v = make_qkv(1, 400, 400, 4, 2, D, seed=12, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q * 2.0, k * 2.0, v[..., :min(D, 128)])
    kw = {} if used is None else {"seqused_k": torch.tensor([used], dtype=torch.int32, device=cuda_device)}
    out, lse = _attend(Q, K, V, causal=True, softcap=2.0, window_size=window, **kw)
    n = 400 if used is None else used
    part = [Q, fa.NVFP4Tensor(K.data[:, :n], K.sf[:, :n], K.scale),
            fa.NVFP4Tensor(V.data[..., :(n + 31) // 32 * 16], V.sf[..., :(n + 31) // 32 * 2], V.scale, is_v=True)]
    oa, la, ob, lb = oracles(*part, True, softcap=2.0, window=window)
    o = out.float().cpu()
    assert torch.isfinite(o).all() and orc.error_metrics(o, ob)["rel_rms"] <= 0.05
    assert torch.equal(torch.isinf(lse.cpu()), torch.isinf(la))
    fin = torch.isfinite(la)
    assert (lse.cpu()[fin] - la[fin]).abs().max().item() <= 2e-3 * max(1.0, la[fin].abs().max().item())


@pytest.mark.parametrize("B,Sq,Sk,Hq,D,splits", [(1, 3, 1300, 3, 64, 9), (1, 130, 1300, 2, 64, 10), (2, 200, 700, 40, 64, 2),
                                                 (1, 129, 1300, 3, 128, 11), (1, 5, 4200, 1, 128, 33),
                                                 (1, 2048, 1300, 1, 64, 9), (1, 2049, 1300, 1, 64, 9), (1, 683, 1300, 3, 128, 9)])
def test_combine_by_one_and_by_four_warps(cuda_device, B, Sq, Sk, Hq, D, splits):
    """Up to eight splits, or with more than 2048 rows, a row is a warp's, else it is four warps'; at head dim 64 two rows are
    a warp's, the last of an odd number alone; 2 x 40 x 2 tiles of two splits are more than are merged inside clusters."""
    q, k, v = make_qkv(B, Sq, Sk, Hq, Hq, D, seed=13, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    out, lse = _attend(Q, K, V, causal=True, num_splits=splits, variant=fa.VARIANT_WS)
    assert_parity(out, lse, *oracles(Q, K, V, True, num_splits=splits, variant=fa.VARIANT_WS))


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,splits,paged", [(1, 1, 1, 4, 1, 1, False), (1, 1, 777, 32, 8, 0, False), (2, 2, 800, 8, 2, 3, False),
                                                         (1, 8, 4230, 8, 2, 1, False), (3, 1, 1000, 16, 1, 2, False),
                                                         (5, 1, 700, 8, 2, 2, False), (2, 1, 33, 8, 8, 1, False),
                                                         (2, 4, 768, 8, 2, 9, True), (1, 1, 9000, 4, 1, 2, True),
                                                         (1, 1, 170001, 16, 1, 0, False), (1, 1, 270080, 4, 1, 9, True)])
def test_decode_reads_linear_scales(cuda_device, B, Sq, Sk, Hq, Hkv, splits, paged, offset):
    """The decode kernel's own reading of linear scales -- one key, ragged key counts (a row of V's scales is then 2 or 6
    bytes more than a multiple of 8), more than 32 blocks a CTA, keys past the general line, pages, every base alignment, outer strides with
    holes -- against the tiled ones: the same bits."""
    rows, slots = (B * -(-Sk // 256), 256) if paged else (B, Sk)
    g = torch.Generator(device=cuda_device).manual_seed(14)
    q, k, v = (torch.randn(b, S, H, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
               for b, S, H in ((B, Sq, Hq), (rows, slots, Hkv), (rows, slots, Hkv)))
    Q, K, V = fa.quantize_qkv_fused(q, k, v)

    def moved(t):        # the same bytes `offset` into an allocation, a head more in the (possibly) strided dimension
        wide = torch.full((*t.shape[:-2], t.shape[-2] + 1, t.shape[-1]), 0x7f, dtype=torch.uint8, device=cuda_device)
        wide[..., :-1, :] = t
        buf = torch.empty(wide.numel() + 8, dtype=torch.uint8, device=cuda_device)
        at = buf[offset:offset + wide.numel()].view(wide.shape)
        at.copy_(wide)
        return at[..., :-1, :]

    kw = {"causal": True, "num_splits": splits, "return_lse": True, "variant": fa.VARIANT_DECODE}
    if paged:
        kw["page_table"] = torch.randperm(rows, generator=g, device=cuda_device).to(torch.int32).view(B, -1)
        kw["seqused_k"] = torch.full((B,), Sk, dtype=torch.int32, device=cuda_device)
    elif B == 5:
        kw["seqused_k"] = torch.tensor([0, 1, 700, 129, 300], dtype=torch.int32, device=cuda_device)
    scales = (Q.scale, K.scale, V.scale)
    want = fa.flash_attn_fp4_func(Q.data, K.data, V.data, *(t.tiled_sf() for t in (Q, K, V)), *scales, sf_layout="tiled", **kw)
    got = fa.flash_attn_fp4_func(Q.data, K.data, V.data, *(moved(t.sf) for t in (Q, K, V)), *scales, sf_layout="linear", **kw)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


def test_linear_decode_takes_device_scales_and_repeated_rows(cuda_device):
    """Per-tensor scales that have not left the device, and one head's scales for all heads (stride 0)."""
    q, k, v = make_qkv(2, 1, 700, 8, 2, 128, seed=15, device=cuda_device)
    kw = {"causal": True, "return_lse": True}
    known = fa.quantize_qkv_fused(q, k, v)
    scales = tuple(t.scale for t in known)
    data = [t.data for t in known]
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    want = fa.flash_attn_fp4_func(*data, *(t.sf for t in known), *scales, **kw)
    got = fa.flash_attn_fp4_func(Q.data, K.data, V.data, Q.sf, K.sf, V.sf, Q._scale, K._scale, V._scale, **kw)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])
    one = [Q.sf[:, :, :1].expand(-1, -1, 8, -1), K.sf[:, :, :1].expand(-1, -1, 2, -1), V.sf[:, :1].expand(-1, 2, -1, -1)]
    want = fa.flash_attn_fp4_func(*data, *(t.contiguous() for t in one), *scales, **kw)
    got = fa.flash_attn_fp4_func(*data, *one, *scales, **kw)
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("spare", [0, 3, 37], ids=["full", "line_moved", "no_line"])
def test_decode_from_a_pool_larger_than_the_table(cuda_device, spare):
    """Linear scales of a pool that other sequences share: the pages in use are read where they are, or the whole pool
    is tiled; either way the bits of the entry in a pool of its own."""
    rows, B, Sk = 12, 2, 6 * 256
    g = torch.Generator(device=cuda_device).manual_seed(16)
    q, k, v = (torch.randn(b, S, H, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
               for b, S, H in ((B, 1, 8), (rows, 256, 2), (rows, 256, 2)))
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    table = torch.randperm(rows, generator=g, device=cuda_device).view(B, -1)
    used = torch.tensor([Sk, 700], dtype=torch.int32, device=cuda_device)
    at = torch.randperm(rows + spare, generator=g, device=cuda_device)[:rows]       # where the pages went

    def pool(t):
        other = torch.full((rows + spare, *t.shape[1:]), 0x7f, dtype=torch.uint8, device=cuda_device)   # NaN scales
        other[at] = t
        return other

    def run(ops, where):
        return fa.flash_attn_fp4_func(Q.data, ops[0], ops[1], Q.sf, ops[2], ops[3], Q.scale, K.scale, V.scale, causal=True,
                                      return_lse=True, seqused_k=used, page_table=where.to(torch.int32).contiguous())

    ops = (K.data, V.data, K.sf, V.sf)
    want, got = run(ops, table), run([pool(t) for t in ops], at[table])
    torch.cuda.synchronize()
    fa.check_status(cuda_device)
    assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


@pytest.mark.parametrize("Sq,Hq,Hkv,Sk,lens,layout,paged,splits", [
    # one token: an empty entry, single keys, block edges; split and not; more splits than blocks
    (1, 32, 8, 13312, [13312, 0, 1, 127, 128], "tiled", True, 0),
    (1, 32, 8, 13312, [13312, 129, 4096, 4097, 1], "linear", False, 0),
    (1, 32, 8, 13312, [0, 0, 0, 0, 0], "tiled", False, 0),
    (1, 32, 8, 13312, [13312, 13312, 13311, 13185, 13184], "tiled", True, 3),
    (1, 32, 8, 13312, [13312, 900, 260, 300, 12000], "tiled", False, 128),
    (2, 8, 2, 9000, [9000, 1] + [33 * i for i in range(31)], "linear", False, 1),           # two chunks of entries
    (4, 16, 8, 3200, [3200, 300, 3199, 0, 4, 3] * 6, "tiled", True, 2),                    # eight rows, entries by length
    (4, 32, 8, 8704, [8704, 3, 130, 8000], "tiled", True, 0),                              # sixteen rows
    (8, 32, 8, 8704, [8704, 7, 130, 8000], "linear", False, 5),                            # 32 rows
    (1, 4, 4, 5120, [5120 - 40 * i for i in range(127)] + [0], "tiled", False, 2),  # more units than places, 128 entries
], ids=str)
def test_decode_dealt_by_the_lengths(cuda_device, Sq, Hq, Hkv, Sk, lens, layout, paged, splits):
    """CTAs dealt by the key counts, against each entry alone with the same splits: fp32 partials in another
    grouping, so bf16 neighbours (2^-8 of a value), and rows whose reference moves inside a split, which may round P anew behind
    it (two roundings of all of P differ by 0.16 rel-RMS; fewer than one row in 256 does that here)."""
    B = len(lens)
    assert fa.lib().fa4_nvfp4_decode_is_balanced(B, Sq, Sk, Hq, Hkv) == 1
    if splits == 0:
        splits = fa._lib.host().choose_decode_splits(B, Hkv, Sk, 148)
    rows, slots = (B * (Sk // 128), 128) if paged else (B, Sk)
    g = torch.Generator(device=cuda_device).manual_seed(21)
    q, k, v = (torch.randn(b, S, H, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
               for b, S, H in ((B, Sq, Hq), (rows, slots, Hkv), (rows, slots, Hkv)))
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    sf = (lambda t: t.sf) if layout == "linear" else (lambda t: t.tiled_sf())
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    table = torch.randperm(rows, generator=g, device=cuda_device).to(torch.int32).view(B, -1) if paged else None

    def call(b0, b1):
        part = (lambda x: x) if paged else (lambda x: x[b0:b1])
        return fa.flash_attn_fp4_func(Q.data[b0:b1], part(K.data), part(V.data), sf(Q)[b0:b1], part(sf(K)), part(sf(V)),
                                      Q.scale, K.scale, V.scale, causal=True, sf_layout=layout, num_splits=splits,
                                      seqused_k=used[b0:b1], page_table=None if table is None else table[b0:b1],
                                      return_lse=True)

    out, lse = call(0, B)
    alone = [call(b, b + 1) for b in range(B)]
    fa.check_status(cuda_device)
    ref, ref_lse = (torch.cat([a[i] for a in alone]) for i in (0, 1))
    assert torch.isfinite(out).all() and torch.equal(torch.isinf(lse), torch.isinf(ref_lse))
    fin = torch.isfinite(ref_lse)
    if fin.any():
        assert (lse[fin] - ref_lse[fin]).abs().max().item() <= 1e-4
    assert torch.equal(out.isfinite(), ref.isfinite()) and (out.float() - ref.float()).norm() <= 0.01 * ref.float().norm()
    assert torch.equal(out.permute(0, 2, 1, 3)[~fin], torch.zeros_like(out.permute(0, 2, 1, 3)[~fin]))


def test_decode_dealt_by_the_lengths_where_references_move(cuda_device):
    """Scores that grow and shrink along the keys by up to 40 log2 units, so that references move within splits, fall where one
    starts: against exact attention, no further off than the entries alone are (with the quarter that the parity tests allow
    P's rounding)."""
    B, Sk, Hq, Hkv = 6, 12288, 8, 8
    lens = [12288, 5000, 700, 12000, 3000, 129]
    g = torch.Generator(device=cuda_device).manual_seed(22)
    q = torch.randn(B, 1, Hq, 128, generator=g, device=cuda_device)
    k = torch.randn(B, Sk, Hkv, 128, generator=g, device=cuda_device)
    v = torch.randn(B, Sk, Hkv, 128, generator=g, device=cuda_device)
    wave = torch.sin(torch.arange(Sk, device=cuda_device) / torch.tensor([2000.0, 300.0, 90.0, 5000.0, 700.0, 40.0],
                                                                         device=cuda_device)[:, None]) * 14.0
    k = k + wave[:, :, None, None] * (q / q.norm(dim=-1, keepdim=True))
    Q, K, V = fa.quantize_qkv_fused(q.bfloat16(), k.bfloat16(), v.bfloat16())
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    for splits in (1, 3, 40):
        kw = dict(causal=True, num_splits=splits, return_lse=True)
        assert fa.lib().fa4_nvfp4_decode_is_balanced(B, 1, Sk, Hq, Hkv) == 1
        got, lse = fa.flash_attn_fp4_func(Q.data, K.data, V.data, Q.sf, K.sf, V.sf, Q.scale, K.scale, V.scale, seqused_k=used, **kw)
        for b, n in enumerate(lens):
            one = [t[b:b + 1] for t in (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)]
            alone, _ = fa.flash_attn_fp4_func(*one, Q.scale, K.scale, V.scale, seqused_k=used[b:b + 1], **kw)
            qd, kd, vd = (t.dequantize()[b:b + 1].float() for t in (Q, K, V))
            s = torch.einsum("bqhd,bkhd->bhqk", qd, kd[:, :n]) / math.sqrt(128)
            exact = torch.einsum("bhqk,bkhd->bqhd", s.softmax(-1), vd[:, :n])
            e_got, e_alone = ((x.float() - exact).norm() / exact.norm() for x in (got[b:b + 1], alone))
            assert e_got <= 1.25 * e_alone + 0.01, (splits, b, e_got, e_alone)
            assert (lse[b, :, 0] - s.logsumexp(-1)[0, :, 0]).abs().max() <= 1e-3 * s.abs().max()
    fa.check_status(cuda_device)


def _through_the_c_entry(Q, K, V, used, splits, short=0):
    """Decode with the workspace that is asked for, which is that of a dealt call, less `short` bytes."""
    B, Sq, Hq, _ = Q.data.shape
    Sk, Hkv = K.data.shape[1:3]
    L, dev = fa.lib(), Q.data.device
    assert L.fa4_nvfp4_decode_is_balanced(B, Sq, Sk, Hq, Hkv) == 1
    out = torch.full((B, Sq, Hq, 128), math.nan, dtype=torch.bfloat16, device=dev)
    lse = torch.full((B, Hq, Sq), math.nan, device=dev)
    p, x, sf = _params(Q, K, V, out, lse, True, DeviceStatus.word(dev)), _lib.Ext(), [t.tiled_sf() for t in (Q, K, V)]
    p.variant, (p.q_sf, p.k_sf, p.v_sf) = 4, (t.data_ptr() for t in sf)
    x.struct_size, x.num_splits, x.window_left, x.window_right = ctypes.sizeof(x), splits, -1, -1
    x.seqused_k = used.data_ptr()
    size = L.fa4_nvfp4_fwd_ex_workspace_bytes(ctypes.byref(p), ctypes.byref(x))
    workspace = torch.empty(size, dtype=torch.uint8, device=dev)
    x.workspace, x.workspace_bytes = workspace.data_ptr(), size - short
    stream = torch.cuda.current_stream(dev).cuda_stream
    assert L.fa4_nvfp4_fwd_ex(ctypes.byref(p), ctypes.byref(x), stream) == 0
    torch.cuda.synchronize(dev)
    fa.check_status(dev)
    return out, lse


@pytest.mark.parametrize("Sq,Hq,Hkv,Sk,lens,layout,splits", [
    (1, 32, 8, 8192, [8192, 300, 4000, 1, 129, 0, 2000, 8191] * 2, "tiled", 2),
    (1, 32, 8, 13312, [13312, 129, 4096, 4097, 1], "linear", 3),
    (1, 32, 8, 13312, [13312, 900, 260, 300, 12000], "tiled", 128),
    (2, 8, 2, 9000, [9000, 1] + [33 * i for i in range(31)], "linear", 1),
    (8, 32, 8, 8704, [8704, 7, 130, 8000], "tiled", 5),
], ids=str)
def test_a_chosen_split_count_gives_the_bits_of_the_entry_alone(cuda_device, Sq, Hq, Hkv, Sk, lens, layout, splits):
    """Batches that are dealt by the lengths where the split count is left open: with a count, and through the C entry point with
    a byte less than the workspace of a dealt call, an entry does not depend on its neighbours."""
    B = len(lens)
    g = torch.Generator(device=cuda_device).manual_seed(24)
    Q, K, V = fa.quantize_qkv_fused(*(torch.randn(B, S, H, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
                                      for S, H in ((Sq, Hq), (Sk, Hkv), (Sk, Hkv))))
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)

    def call(b0, b1):
        sf = [(t.sf if layout == "linear" else t.tiled_sf())[b0:b1] for t in (Q, K, V)]
        return fa.flash_attn_fp4_func(*(t.data[b0:b1] for t in (Q, K, V)), *sf, Q.scale, K.scale, V.scale, causal=True,
                                      sf_layout=layout, num_splits=splits, seqused_k=used[b0:b1], return_lse=True)

    out, lse = call(0, B)
    short_out, short_lse = _through_the_c_entry(Q, K, V, used, splits, short=1)
    for b in range(B):
        o, l = call(b, b + 1)
        assert torch.equal(out[b:b + 1], o) and torch.equal(lse[b:b + 1], l), lens[b]
        assert torch.equal(short_out[b:b + 1], o) and torch.equal(short_lse[b:b + 1], l), lens[b]
    fa.check_status(cuda_device)


@pytest.mark.parametrize("Sq,Hq,Hkv,Sk,lens,splits", [
    (1, 32, 8, 13312, [13312, 13312, 13311, 13185, 13184], 3),
    (1, 32, 8, 13312, [13312, 900, 260, 300, 12000], 128),
    (2, 8, 2, 9000, [9000, 1] + [33 * i for i in range(31)], 1),
    (4, 16, 8, 3200, [3200, 300, 3199, 0, 4, 3] * 6, 2),
    (8, 32, 8, 8704, [8704, 7, 130, 8000], 5),
    (1, 4, 4, 5120, [5120 - 40 * i for i in range(127)] + [0], 2),
], ids=str)
def test_decode_dealt_with_a_chosen_split_count(cuda_device, Sq, Hq, Hkv, Sk, lens, splits):
    """Through the C entry point, with the workspace for it: against the splits, within the bounds of
    test_decode_dealt_by_the_lengths."""
    B = len(lens)
    g = torch.Generator(device=cuda_device).manual_seed(25)
    Q, K, V = fa.quantize_qkv_fused(*(torch.randn(B, S, H, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
                                      for S, H in ((Sq, Hq), (Sk, Hkv), (Sk, Hkv))))
    used = torch.tensor(lens, dtype=torch.int32, device=cuda_device)
    out, lse = _through_the_c_entry(Q, K, V, used, splits)
    ref, ref_lse = fa.flash_attn_fp4_func(
        Q.data, K.data, V.data, Q.sf, K.sf, V.sf, Q.scale, K.scale, V.scale, causal=True, num_splits=splits, seqused_k=used,
        return_lse=True)
    fin = torch.isfinite(ref_lse)
    assert torch.isfinite(out).all() and torch.equal(torch.isinf(lse), torch.isinf(ref_lse))
    assert (lse[fin] - ref_lse[fin]).abs().max().item() <= 1e-4
    assert (out.float() - ref.float()).norm() <= 0.01 * ref.float().norm()
    assert not out.permute(0, 2, 1, 3)[~fin].any()


def _long_beside(device, B, Sq, Sk, Hq, Hkv, lens, level, v_mean, splits):
    """Dealt decode against a cache in which entry 0 has scores `level[key]` (log2 units, the same for all rows but a few per cent) plus
    noise, among entries of zeros.  Returns the relative error of entry 0 in the batch and of entry 0 alone (O), and the
    errors of the LSEs."""
    g = torch.Generator(device=device).manual_seed(23)
    n = lens[0]
    u = (torch.randint(0, 2, (Hkv, 1, 128), generator=g, device=device) * 2 - 1) / math.sqrt(128.0)
    q = torch.zeros(B, Sq, Hq, 128, device=device)
    k = torch.zeros(B, Sk, Hkv, 128, device=device, dtype=torch.bfloat16)
    v = torch.zeros(B, Sk, Hkv, 128, device=device, dtype=torch.bfloat16)
    # q = 8 u: a score in log2 units is 8 (u . k) / sqrt(128) * log2(e) = 1.0201 (u . k)
    rise = 1.0 + 0.05 * torch.rand(Sq, Hkv, Hq // Hkv, 1, generator=g, device=device)
    q[0] = (8.0 * rise * u).reshape(Sq, Hq, 128)
    # (as a thermometer over the eight scale blocks of a row, whose scales have steps of 6 to 12 %)
    lev = (level / 1.0201).to(device)
    top = lev.max() + 1e-3
    lev = (8.0 * lev[:, None] - top * torch.arange(8, device=device)).clamp(min=0.0).minimum(top).repeat_interleave(16, dim=1)
    k[0, :n] = (lev[:, None, :] * u[:, 0] + 0.05 * torch.randn(n, Hkv, 128, generator=g, device=device)).bfloat16()
    v[0, :n] = (v_mean[:, None, None].to(device) + 0.5 * (v_mean != 0)[:, None, None].to(device) *
                torch.randn(n, Hkv, 128, generator=g, device=device)).bfloat16()
    Q, K, V = fa.quantize_qkv_fused(q.bfloat16(), k, v)
    used = torch.tensor(lens, dtype=torch.int32, device=device)
    T = (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)
    call = lambda t, u, s: fa.flash_attn_fp4_func(*t, Q.scale, K.scale, V.scale, causal=True, num_splits=s, seqused_k=u,
                                                  return_lse=True)
    got, lse = (x[:1] for x in (call(T, used, 0) if splits == 0 else _through_the_c_entry(Q, K, V, used, splits)))
    if splits == 0:
        splits = fa._lib.host().choose_decode_splits(B, Hkv, Sk, 148)
    alone, lse_alone = call([t[:1] for t in T], used[:1], splits)
    fa.check_status(device)
    qd = Q.dequantize()[:1].double()
    kd = fa.quant.dequantize_lastdim(K.data[:1], K.sf[:1], K.scale)[0, :n].double()
    vd = fa.quant.dequantize_lastdim(V.data[:1], V.sf[:1], V.scale)[0, :, :, :n].double()
    qg = qd[0].view(Sq, Hkv, Hq // Hkv, 128)
    s = torch.einsum("shgd,nhd->hgsn", qg, kd) / math.sqrt(128)
    s = s.masked_fill(torch.arange(n, device=device)[None, :] > n - Sq + torch.arange(Sq, device=device)[:, None], -math.inf)
    exact = torch.einsum("hgsn,hdn->shgd", s.softmax(-1), vd).reshape(1, Sq, Hq, 128)
    exact_lse = s.logsumexp(-1).reshape(1, Hq, Sq)
    err = lambda x: ((x.double() - exact).norm() / exact.norm()).item()
    err_lse = lambda x: ((x.double() - exact_lse).abs().max() / max(1.0, exact_lse.abs().max().item())).item()
    assert torch.isfinite(alone).all()
    return err(got), err(alone), err_lse(lse), err_lse(lse_alone)


@pytest.mark.parametrize("Sq,group", [(1, 4), (1, 8), (4, 4), (8, 4)])
@pytest.mark.parametrize("fall", [1.0, 2.0, 3.0, 5.0])
def test_decode_of_maxima_that_fall_from_split_to_split(cuda_device, Sq, group, fall):
    """128 blocks, a split each, whose maxima fall by 128 to 640 log2 units in all, in an entry of a batch that leaves it to few
    CTAs: finite, and no further from exact attention than the entry alone (with the quarter that the parity tests allow
    P's rounding)."""
    n, B = 16384, 40
    level = fall * (127 - torch.arange(n) // 128)
    e, e_alone, l, _ = _long_beside(cuda_device, B, Sq, n, 8 * group, 8, [n] * B, level, torch.ones(n), 128)
    assert e <= 1.25 * e_alone + 0.01 and l <= 1e-3, (e, e_alone, l)


def test_decode_of_maxima_that_fall_with_chosen_splits(cuda_device):
    n, Sk, B = 4608, 288000, 8
    level = 4.0 * (35 - torch.arange(n) // 128)
    e, e_alone, l, _ = _long_beside(cuda_device, B, 1, Sk, 8, 1, [n] + [Sk] * (B - 1), level, torch.ones(n), 0)
    assert e <= 1.25 * e_alone + 0.01 and l <= 1e-3, (e, e_alone, l)


@pytest.mark.parametrize("Sq", [1, 8])
@pytest.mark.parametrize("height", [10.0, 12.0, 14.0, 16.0, 18.0, 40.0])
def test_decode_behind_a_first_key_without_a_value(cuda_device, Sq, height):
    """A first key far above the rest whose V is zero (an attention sink), ten splits of one block each: what the other splits add is
    the whole result, and is no further off than in the entry alone."""
    n, Sk, B = 1280, 16384, 40
    level, v_mean = torch.zeros(n), torch.ones(n)
    level[0], v_mean[0] = height, 0.0
    e, e_alone, l, _ = _long_beside(cuda_device, B, Sq, Sk, 32, 8, [n] + [Sk] * (B - 1), level, v_mean, 10)
    assert e <= 1.25 * e_alone + 0.01 and l <= 1e-3, (e, e_alone, l)
