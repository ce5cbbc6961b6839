"""The native host path beside other Python threads and beside the operands a caller may pass: what waits for
the GPU waits without the interpreter lock, what is not bytes is not read as bytes, and a call that fails
half-way leaves the buffers of the next one in order."""
import copy
import threading
import time

import pytest
import torch

import flash_attention_b200 as fa
from tests.helpers import make_qkv

pytestmark = pytest.mark.gpu


def _operands(device, B=1, S=256, Hq=4, Hkv=2, seed=31):
    q, k, v = make_qkv(B, S, S, Hq, Hkv, 128, seed=seed, device=device)
    return tuple(fa.NVFP4Tensor(t.data.to(device), t.sf.to(device), t.scale, is_v=t.is_v) for t in fa.quantize_qkv(q, k, v))


def _largest_gap(call, device, busy_s=0.5):
    """Runs `call` behind a kernel that keeps the stream busy; returns (its duration, the longest time another
    Python thread stood still meanwhile)."""
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    torch.cuda.synchronize(device)
    t = threading.Thread(target=tick)
    t.start()
    try:
        time.sleep(0.05)
        torch.cuda._sleep(int(busy_s * 1.9e9))
        t0 = time.perf_counter()
        call()
        took = time.perf_counter() - t0
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize(device)
    return took, max(gaps)


@pytest.mark.parametrize("waits_for", ["scale", "sink", "longest", "pageable operands"])
def test_a_call_that_waits_lets_other_threads_run(cuda_device, waits_for):
    Q, K, V = _operands(cuda_device)
    ops = (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)
    if waits_for == "scale":
        s = [torch.tensor([t.scale], device=cuda_device) for t in (Q, K, V)]
        call = lambda: fa.flash_attn_fp4_func(*ops, *s, causal=True)
    elif waits_for == "sink":
        sink = torch.zeros(4)
        call = lambda: fa.flash_attn_fp4_func(*ops, Q.scale, K.scale, V.scale, learnable_sink=sink)
    elif waits_for == "longest":
        cu = torch.tensor([0, 128, 256], dtype=torch.int32, device=cuda_device)
        call = lambda: fa.flash_attn_varlen_fp4_func(*(t[0] for t in ops), Q.scale, K.scale, V.scale, cu, cu)
    else:
        pipe = fa.HostPipeline(1, 256, 256, 4, 2, device=cuda_device)
        host = [t.cpu() for t in ops]
        out = torch.empty(1, 256, 4, 128, dtype=torch.bfloat16)
        call = lambda: pipe.run(*host, Q.scale, K.scale, V.scale, out, causal=True)
    call()                                       # allocations and module loading
    took, gap = _largest_gap(call, cuda_device)
    assert took > 0.2, f"the call did not wait ({took:.3f} s): nothing was tested"
    assert gap < 0.5 * took, f"another thread stood still for {gap:.3f} s of {took:.3f} s"
    fa.check_status(cuda_device)


def test_host_operands_of_wider_types_are_converted_to_bytes(cuda_device):
    Q, K, V = _operands(cuda_device)
    want, want_lse = fa.flash_attn_func(Q, K, V, causal=True, return_lse=True)
    host = [t.cpu() for t in (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)]
    pipe = fa.HostPipeline(1, 256, 256, 4, 2, device=cuda_device)
    for given in ([t.to(torch.int32) for t in host],                    # byte values in a wider type
                  host[:3] + [t.view(torch.float8_e4m3fn) for t in host[3:]],   # scale bytes under their own type
                  [host[0], host[1].to(torch.int64)] + host[2:]):
        out = torch.zeros(1, 256, 4, 128, dtype=torch.bfloat16).pin_memory()
        lse = torch.zeros(1, 4, 256).pin_memory()
        pipe.run(*given, Q.scale, K.scale, V.scale, out, lse, causal=True)
        pipe.wait()
        assert torch.equal(out, want.cpu()) and torch.equal(lse, want_lse.cpu()), [t.dtype for t in given]


def test_a_failed_call_keeps_its_buffers_until_its_copies_have_run(cuda_device):
    """An error behind the first copies: the pinned operands must not go back to their pool while those copies
    are on their way, wait() waits for them, and the next call is right."""
    Q, K, V = _operands(cuda_device)
    want = fa.flash_attn_func(Q, K, V, causal=True)[0]
    ops = (Q.data, K.data, V.data, Q.sf, K.sf, V.sf)
    pipe = fa.HostPipeline(1, 256, 256, 4, 2, device=cuda_device)
    out = torch.zeros(1, 256, 4, 128, dtype=torch.bfloat16).pin_memory()
    good = [t.cpu().pin_memory() for t in ops]
    pipe.run(*good, Q.scale, K.scale, V.scale, out, causal=True)          # allocations and module loading
    pipe.wait()
    cpu = [t.cpu() for t in ops]
    host = [t.pin_memory() for t in cpu]
    where = {t.data_ptr() for t in host}
    torch.cuda._sleep(int(0.5 * 1.9e9))
    with pytest.raises(ValueError):
        pipe.run(*host, 0.0, K.scale, V.scale, out, causal=True)          # refused when the first piece is launched
    assert not pipe.done.query()
    del host
    again = [t.pin_memory() for t in cpu]
    reused = where & {t.data_ptr() for t in again}
    still_copying = not pipe.done.query()
    pipe.wait()
    assert still_copying and not reused
    out.zero_()
    pipe.run(*again, Q.scale, K.scale, V.scale, out, causal=True)
    pipe.wait()
    assert torch.equal(out, want.cpu())


def test_a_captured_call_may_read_scales_on_the_device(cuda_device):
    """A capture on the quantiser's own stream takes the scales from the device.  They live as long as the
    operands, also when their values are read before the graph is replayed."""
    q, k, v = make_qkv(1, 256, 256, 4, 2, 128, seed=41, device=cuda_device)
    want = fa.flash_attn_func(*fa.quantize_qkv_fused(q, k, v), causal=True)[0]
    stream = torch.cuda.Stream(cuda_device)
    stream.wait_stream(torch.cuda.current_stream(cuda_device))
    with torch.cuda.stream(stream):
        ops = fa.quantize_qkv_fused(q, k, v)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = fa.flash_attn_func(*ops, causal=True)[0]
        assert all(t.scale > 0 for t in ops) and copy.copy(ops[0]).scale == ops[0].scale
        reused = [torch.full((128,), 3.0, device=cuda_device) for _ in range(64)]     # small blocks of the same stream
        graph.replay()
        stream.synchronize()
    assert torch.equal(out, want) and len(reused) == 64
    fa.check_status(cuda_device)


def test_scales_may_be_fetched_while_another_stream_captures(cuda_device):
    q, k, v = make_qkv(1, 256, 256, 4, 2, 128, seed=42, device=cuda_device)
    want = fa.flash_attn_func(*fa.quantize_qkv_fused(q, k, v), causal=True)[0]
    ops = fa.quantize_qkv_fused(q, k, v)         # its scales are read by nobody before the capture
    torch.cuda.synchronize(cuda_device)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fa.flash_attn_func(*ops, causal=True)[0]
    graph.replay()
    torch.cuda.synchronize(cuda_device)
    assert torch.equal(out, want)
    fa.check_status(cuda_device)
