"""Calls of one stream, each reading what the one before it wrote, without a synchronisation: a
kernel may start before its predecessor ends, so this has to give the bits of the same calls run
one at a time, eager, beside another stream, and captured in a graph."""
import ctypes

import pytest

import momms_gb300 as mg

pytestmark = pytest.mark.gpu

MODES = [("f64", mg.PREC_PLAIN, 0), ("f32", mg.PREC_PLAIN, 0), ("f32", mg.PREC_SPLIT_TF32, 0),
         ("f64", mg.PREC_OZAKI, 4), ("f64", mg.PREC_OZAKI, 8)]


def _chain(lib, prec, slices, a, cs, stream, each=None):
    """cs[i + 1] = a @ cs[i] / 2 + cs[i + 1], then doubled where i is odd, for each i."""
    import torch
    n = a.shape[0]
    w = cs[0].shape[1]
    for i in range(len(cs) - 1):
        d = mg.GemmDesc()
        d.dtype = mg.DTYPE_F64 if a.dtype == torch.float64 else mg.DTYPE_F32
        d.precision, d.slices = prec, slices
        d.m, d.n, d.k = n, w, n
        d.alpha, d.beta = 0.5, 1.0
        d.a = mg.Operand(a.data_ptr(), 1, n, mg.MEM_DEVICE, 0)
        d.b = mg.Operand(cs[i].data_ptr(), w, 1, mg.MEM_DEVICE, 0)
        d.c = mg.Operand(cs[i + 1].data_ptr(), w, 1, mg.MEM_DEVICE, 0)
        mg.check(lib.momms_gemm(ctypes.byref(d), ctypes.c_void_p(stream.cuda_stream)), lib)
        if i % 2:
            cs[i + 1].mul_(2.0)
        if each:
            each()


@pytest.mark.parametrize("mode", MODES, ids=["f64", "f32", "tf32", "s4", "s8"])
@pytest.mark.parametrize("n,w", [(40, 24), (300, 130), (1100, 700)])
def test_chained_calls_give_the_bits_of_separate_ones(gpu, mode, n, w):
    import torch
    dt, prec, slices = mode
    gen = torch.Generator().manual_seed(n + slices)
    dtype = torch.float64 if dt == "f64" else torch.float32
    a = (torch.randn(n, n, generator=gen, dtype=dtype) / n**0.5).cuda()
    c0 = [torch.randn(n, w, generator=gen, dtype=dtype).cuda() for _ in range(7)]
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    want = [c.clone() for c in c0]
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        _chain(gpu, prec, slices, a, want, s, torch.cuda.synchronize)
    two = [[c.clone() for c in c0] for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(3):  # both streams busy, no synchronisation inside
        for st, got in zip((s, t), two):
            with torch.cuda.stream(st):
                for x, y in zip(got, c0):
                    x.copy_(y)
                _chain(gpu, prec, slices, a, got, st)
    torch.cuda.synchronize()
    for got in two:
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    got = two[0]
    with torch.cuda.graph(graph, stream=s):
        for x, y in zip(got, c0):
            x.copy_(y)
        _chain(gpu, prec, slices, a, got, s)
    for x in got:
        x.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_captured_emulated_call_bounds_its_scratch(gpu):
    """A graph's scratch is allocated when it is launched: a captured call stays within the digit form's
    (or 512 MB), in more passes and with the bits of the call outside."""
    import torch
    m, n, k, slices = 4096, 1024, 4096, 7
    gen = torch.Generator(device="cuda").manual_seed(6)
    a, b = (torch.rand(x, dtype=torch.float64, device="cuda", generator=gen) - 0.5 for x in ((k, m), (n, k)))
    want, got = (torch.zeros((n, m), dtype=torch.float64, device="cuda") for _ in range(2))
    s = torch.cuda.Stream()

    def call(c):
        d = mg.GemmDesc()
        d.dtype, d.precision, d.slices = mg.DTYPE_F64, mg.PREC_OZAKI, slices
        d.m, d.n, d.k, d.alpha, d.beta = m, n, k, 1.0, 0.0
        d.a, d.b, d.c = (mg.Operand(x.data_ptr(), 1, ld, mg.MEM_DEVICE, 0) for x, ld in ((a, m), (b, k), (c, m)))
        mg.check(gpu.momms_gemm(ctypes.byref(d), ctypes.c_void_p(s.cuda_stream)), gpu)

    torch.cuda.synchronize()
    call(want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        call(got)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    graph.replay()
    torch.cuda.synchronize()
    held = free - torch.cuda.mem_get_info()[0]
    assert torch.equal(got, want)
    assert held <= max(2 * slices * (m + n) * k + 4 * slices * m * n, 512 << 20) + (64 << 20)


def test_a_thread_that_called_may_end_during_a_capture(gpu):
    """A thread whose automatic call read a result back ends while another one captures a stream in the
    global mode (torch's default): nothing is left to free that would break the capture."""
    import threading

    import torch
    n = 384
    gen = torch.Generator(device="cuda").manual_seed(8)
    a, b = (torch.rand((n, n), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for _ in range(2))
    cs = [torch.zeros((n, n), dtype=torch.float64, device="cuda") for _ in range(2)]
    s = torch.cuda.Stream()

    def call(c, stream, slices):
        d = mg.GemmDesc()
        d.dtype, d.precision, d.slices = mg.DTYPE_F64, mg.PREC_OZAKI, slices  # 0: chosen from the data
        d.m = d.n = d.k = n
        d.alpha, d.beta = 1.0, 0.0
        d.a, d.b, d.c = (mg.Operand(x.data_ptr(), 1, n, mg.MEM_DEVICE, 0) for x in (a, b, c))
        return gpu.momms_gemm(ctypes.byref(d), ctypes.c_void_p(stream.cuda_stream))

    called, end, results = threading.Event(), threading.Event(), []

    def other():
        results.append(call(cs[0], torch.cuda.Stream(), 0))
        called.set()
        end.wait(60)

    torch.cuda.synchronize()
    assert call(cs[1], s, 7) == mg.OK
    torch.cuda.synchronize()
    want = cs[1].clone()
    th = threading.Thread(target=other)
    th.start()
    assert called.wait(60) and results == [mg.OK]
    cs[1].zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        assert call(cs[1], s, 7) == mg.OK
        end.set()
        th.join()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(cs[1], want)
