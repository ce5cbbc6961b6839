"""GPU parity of the fused NVFP4 quantiser: bit-exact against the CPU oracle's quantiser."""
import ctypes

import numpy as np
import pytest
import torch

import flash_attention_b200 as fa
from oracle import nvfp4_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda_device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    fa.lib()
    return torch.device("cuda", 0)


def _oracle_qk(x):
    return orc.quantize_nvfp4(x.float().cpu().numpy())


def _oracle_v(v):
    # V is quantised key-contiguous with its key axis padded with zeros to a multiple of 32
    pad = (-v.shape[1]) % 32
    if pad:
        v = torch.cat([v, v.new_zeros(v.shape[0], pad, v.shape[2], v.shape[3])], dim=1)
    return orc.quantize_nvfp4(v.float().permute(0, 2, 3, 1).contiguous().cpu().numpy())


def _tiled(sf_np, mult):
    return orc.sf_linear_to_tiled(sf_np, mult)


CASES = [
    # B, S, Hq, Hkv, D, std
    (1, 256, 4, 4, 128, 1.0),
    (2, 208, 4, 2, 128, 1.0),      # ragged rows: zero padding of the tiled scales
    (1, 96, 2, 1, 64, 3.0),        # D = 64, Dv = 64 (half a d tile)
    (1, 1024, 3, 3, 192, 0.5),     # D = 192: three column tiles, two d tiles for V
]


@pytest.mark.parametrize("case", CASES, ids=[f"B{c[0]}_S{c[1]}_H{c[2]}_{c[3]}_D{c[4]}" for c in CASES])
def test_fused_quantiser_is_bit_exact(cuda_device, case):
    B, S, Hq, Hkv, D, std = case
    g = torch.Generator().manual_seed(11)
    q = (torch.randn(B, S, Hq, D, generator=g) * std).bfloat16()
    k = (torch.randn(B, S, Hkv, D, generator=g) * std).bfloat16()
    v = (torch.randn(B, S, Hkv, D, generator=g) * std).bfloat16()
    # exact ties and exact zeros exercise round-to-even and the sign of zero
    q[0, 0, 0, :16] = torch.tensor([0.25, -0.25, 0.75, -0.75, 1.25, 1.75, 2.5, -2.5, 3.5, 5.0, -5.0, 6.0,
                                    0.0, -0.0, 1e-3, -1e-3]).bfloat16() * 0.5
    k[0, 1, 0, 16:32] = 0.0
    Q, K, V = fa.quantize_qkv_fused(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
    for got, want, mult in ((Q, _oracle_qk(q), 1), (K, _oracle_qk(k), 1), (V, _oracle_v(v), 2)):
        assert got.scale == pytest.approx(want.scale, rel=0, abs=0)
        assert np.array_equal(got.sf.cpu().numpy(), want.sf)
        assert np.array_equal(got.data.cpu().numpy(), want.data)
        lin = want.sf if got.is_v else np.transpose(want.sf, (0, 2, 1, 3))
        assert np.array_equal(got.sf_tiled.cpu().numpy(), _tiled(lin, mult))


def test_tiny_magnitudes_take_the_exact_path(cuda_device):
    # tensor scale ~1e-36: the block denominators have no finite fp32 reciprocal
    g = torch.Generator().manual_seed(4)
    x = (torch.randn(1, 128, 2, 128, generator=g) * 1e-33).bfloat16()
    Q, _, V = fa.quantize_qkv_fused(x.to(cuda_device), x.to(cuda_device), x.to(cuda_device))
    for got, want in ((Q, _oracle_qk(x)), (V, _oracle_v(x))):
        assert got.scale == want.scale
        assert np.array_equal(got.sf.cpu().numpy(), want.sf)
        assert np.array_equal(got.data.cpu().numpy(), want.data)


def test_all_zero_tensor_and_strided_input(cuda_device):
    z = torch.zeros(1, 128, 2, 128, dtype=torch.bfloat16, device=cuda_device)
    Q, K, V = fa.quantize_qkv_fused(z, z, z)
    assert Q.scale == 1.0 and int(Q.data.max()) == 0 and int(Q.sf.max()) == 0
    g = torch.Generator(device=cuda_device).manual_seed(5)
    big = torch.randn(2, 256, 6, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
    view = big[:, 64:192, 1:5]                      # strided batch / seq / head view
    Qa, _, Va = fa.quantize_qkv_fused(view, view, view)
    Qb, _, Vb = fa.quantize_qkv_fused(view.contiguous(), view.contiguous(), view.contiguous())
    for a, b in ((Qa, Qb), (Va, Vb)):
        assert a.scale == b.scale and torch.equal(a.data, b.data) and torch.equal(a.sf, b.sf)
        assert torch.equal(a.sf_tiled, b.sf_tiled)


def test_fused_quantiser_feeds_the_attention_kernel(cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(2)
    q = torch.randn(1, 384, 4, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
    k = torch.randn(1, 384, 2, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
    v = torch.randn(1, 384, 2, 128, generator=g, device=cuda_device, dtype=torch.bfloat16)
    Q, K, V = fa.quantize_qkv_fused(q, k, v)
    o1, l1 = fa.flash_attn_func(Q, K, V, causal=True, return_lse=True)
    # same operands with the scales tiled by the separate conversion kernel
    Q2, K2, V2 = (fa.NVFP4Tensor(t.data, t.sf, t.scale, False, t.is_v) for t in (Q, K, V))
    o2, l2 = fa.flash_attn_func(Q2, K2, V2, causal=True, return_lse=True)
    fa.check_status(cuda_device)
    assert torch.equal(o1, o2) and torch.equal(l1, l2)
    # tiled-only output
    Q3, K3, V3 = fa.quantize_qkv_fused(q, k, v, linear_sf=False)
    o3, _ = fa.flash_attn_func(Q3, K3, V3, causal=True, return_lse=True)
    assert torch.equal(o1, o3)


def test_values_next_to_every_rounding_boundary(cuda_device):
    """Every denominator significand that a bf16 maximum and an e4m3 block scale can give (128 x 8), and for each
    the four bf16 values next to each of the seven rounding boundaries of e2m1: the oracle's bytes."""
    mids = np.array([.25, .75, 1.25, 1.75, 2.5, 3.5, 5.0])
    for a in range(128, 256):
        amax = 16.0 * a                                  # tensor scales around one
        g = np.float32(np.float32(amax) / np.float32(2688))
        x = np.zeros((5, 4, 16), dtype=np.float32)
        x[4, 0, 0] = amax
        for m in range(8, 16):
            denom = float(np.float32(m / 8) * g)
            frac, e = np.frexp(mids * denom)
            below = np.floor(np.ldexp(frac, 8))
            for half, (lo, hi) in enumerate(((0, 1), (-1, 2))):
                block = x[(m - 8) // 2, 2 * (m % 2) + half]
                for col, j in ((0, lo), (7, hi)):
                    n = below + j
                    n = np.where(n > 256, 2 * n - 256, np.where(n < 128, 64 + n / 2, n))      # eight bits
                    block[col:col + 7] = np.ldexp(n, e - 8) * (1 - 2 * (m % 2))
                block[14] = torch.tensor(6 * denom).bfloat16().float().item()
        x = torch.from_numpy(x.reshape(1, 5, 1, 64))
        assert torch.equal(x.bfloat16().float(), x)
        want = orc.quantize_nvfp4(x.numpy())
        assert np.array_equal(want.sf[0, :4, 0], 0x38 + np.repeat(np.arange(8), 2).reshape(4, 4))   # 1, 1.125 .. 1.875
        q = fa.quantize_qkv_fused(*(x.bfloat16().to(cuda_device),) * 3)[0]
        assert q.scale == want.scale
        assert np.array_equal(q.sf.cpu().numpy(), want.sf) and np.array_equal(q.data.cpu().numpy(), want.data), a


@pytest.mark.parametrize("B,S,Hq,Hkv,D,std", [
    (1, 130, 1, 1, 64, 1.0),         # four blocks a row: a warp's blocks lie in eight rows, two of them in the last tile
    (3, 77, 3, 1, 64, 1.0),          # twelve blocks a row
    (2, 2500, 32, 3, 128, 1.0),      # several items a thread, the last tile of rows not full, several V tiles a CTA
    (1, 96, 2, 1, 128, 1e25),        # tensor scales beyond the two-term reciprocals
    (1, 96, 2, 1, 128, 2.5e20),      # and just below that line: denominators near 1e20
])
def test_loads_in_stages_and_scales_at_the_ends(cuda_device, B, S, Hq, Hkv, D, std):
    g = torch.Generator().manual_seed(B * S)
    q, k, v = ((torch.randn(B, S, H, D, generator=g) * std).bfloat16() for H in (Hq, Hkv, Hkv))
    Q, K, V = fa.quantize_qkv_fused(q.to(cuda_device), k.to(cuda_device), v.to(cuda_device))
    for got, want, mult in ((Q, _oracle_qk(q), 1), (K, _oracle_qk(k), 1), (V, _oracle_v(v), 2)):
        assert got.scale == want.scale
        assert np.array_equal(got.sf.cpu().numpy(), want.sf)
        assert np.array_equal(got.data.cpu().numpy(), want.data)
        lin = want.sf if got.is_v else np.transpose(want.sf, (0, 2, 1, 3))
        assert np.array_equal(got.sf_tiled.cpu().numpy(), _tiled(lin, mult))


@pytest.mark.parametrize("m", range(9, 16))
def test_a_maximum_of_the_callers_own_with_significands_of_all_ones(cuda_device, m):
    """Tensor scales g from a chosen maximum for which m / 8 times g, the denominator of a block, is 2 - 2^-23 (m = 8: no maximum gives
    that g): the bytes of correctly rounded quotients for the values next to every boundary of e2m1, and for blocks near the
    smallest scale."""
    ones = np.float32(2) - np.float32(2) ** -23
    near = np.float32(float(ones) * 8 / m)
    g = next(c for c in (near, np.nextafter(near, np.float32(0)), np.nextafter(near, np.float32(9)))
             if np.float32(m / 8) * c == ones)
    amax = np.float32(float(g) * 2688)
    amax = next(c for c in (amax, np.nextafter(amax, np.float32(0)), np.nextafter(amax, np.float32(1e9))) if c / np.float32(2688) == g)
    x = np.zeros((4, 16), dtype=np.float32)
    mids = np.array([.25, .75, 1.25, 1.75, 2.5, 3.5, 5.0])
    for row, (lo, hi) in enumerate(((0, 1), (-1, 2))):
        frac, e = np.frexp(mids * float(ones))
        for col, j in ((0, lo), (7, hi)):
            n = np.floor(np.ldexp(frac, 8)) + j
            n = np.where(n > 256, 2 * n - 256, np.where(n < 128, 64 + n / 2, n))      # eight bits
            x[row, col:col + 7] = np.ldexp(n, e - 8)
        x[row, 14] = 12.0                                  # 6 denominators: the block's scale is m / 8
    x[2, 0], x[3, 0], x[3, 1] = 1.5 / 128, 1.5 / 64, -1.5 / 256
    x = torch.from_numpy(x).view(1, 1, 1, 64)
    assert torch.equal(x.bfloat16().float(), x)
    data, sf, _ = fa.quant.quantize_lastdim(x, float(g))
    assert sf.flatten()[0] == sf.flatten()[1] == 0x30 + m
    xd = x.bfloat16().to(cuda_device)
    got, got_sf = (torch.full_like(t, 255, device=cuda_device) for t in (data, sf))
    given = torch.tensor([float(amax)], device=cuda_device)
    assert fa.lib().fa4_nvfp4_quantize_qk_bf16(xd.data_ptr(), 1, 1, 1, 64, 64, 64, 64, given.data_ptr(), got.data_ptr(),
                                               got_sf.data_ptr(), None, None,
                                               ctypes.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)) == 0
    assert torch.equal(got_sf.cpu(), sf) and torch.equal(got.cpu(), data)


@pytest.mark.parametrize("amax", [1.0, 3.7, 1e-20, 2688.0, 1e30])
def test_infinities_under_a_maximum_of_the_callers_own(cuda_device, amax):
    """x / denominator of an infinity is an infinity and takes the largest magnitude with its sign; its neighbours keep theirs."""
    g = torch.Generator().manual_seed(6)
    x = (torch.randn(1, 40, 2, 64, generator=g) * (amax / 4)).bfloat16()
    at = torch.randperm(x.numel(), generator=g)[:60]
    x.view(-1)[at] = torch.tensor([torch.inf, -torch.inf]).repeat(30).bfloat16()
    data, sf, _ = fa.quant.quantize_lastdim(x.float(), float(np.float32(amax) / np.float32(2688)))
    xd, given = x.to(cuda_device), torch.tensor([amax], device=cuda_device)
    got, got_sf = (torch.full_like(t, 255, device=cuda_device) for t in (data, sf))
    assert fa.lib().fa4_nvfp4_quantize_qk_bf16(xd.data_ptr(), 1, 40, 2, 64, *xd.stride()[:3], given.data_ptr(), got.data_ptr(),
                                               got_sf.data_ptr(), None, None,
                                               ctypes.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)) == 0
    assert torch.equal(got_sf.cpu(), sf) and torch.equal(got.cpu(), data)
