"""Which calls of the quantised linears are accepted: host-side rules, read without a GPU."""
import ctypes as C

import pytest
import torch

from agens_engine_b200 import _lib

needs_no_gpu = pytest.mark.skipif(torch.cuda.is_available(), reason="the accepted calls would run on made-up addresses")


# (n, k, slices of k, rows): accepted by the limit in wq_gemv_noalloc.h, 2^20 scratch floats of the kernel with slices
FITS = [(40960, 8192, 1, 8), (151936, 6144, 1, 3), (151936, 8192, 1, 2), (57344, 8192, 1, 5), (11040, 28672, 2, 8), (256, 2048, 4, 3)]
TOO_LARGE = [(151936, 5120, 2, 32), (40960, 8192, 1, 16), (262176, 128, 1, 1)]


@needs_no_gpu
@pytest.mark.parametrize("n,k,ks,m,fits", [s + (True,) for s in FITS] + [s + (False,) for s in TOO_LARGE])
def test_allocation_free_gemv_accepts_what_its_header_says(n, k, ks, m, fits):
    """A refusal is 1 and launches nothing; an accepted call goes on to the device, which is not there (2)."""
    lib = _lib.cuda_lib()
    need = lib.b2_wq_gemv_scratch_floats(n, k, ks, 2, m)
    assert (need <= 1 << 20 and n // 32 <= 8192) == fits
    err = C.create_string_buffer(160)
    fn = lib.b2_wq_gemv_noalloc
    fn.argtypes = [C.c_void_p] + [C.c_int] * 5 + [C.c_void_p, C.c_long, C.c_int, C.c_void_p, C.c_long, C.c_void_p, C.c_void_p, C.c_char_p]
    fn.restype = C.c_int
    rc = fn(256, n, k, 4, 128, ks, 256, k, m, 256, n, None, None, err)
    assert rc == (2 if fits else 1), err.value


def _panel_reference(lin, x, panels):
    """fp64 results of some 32-row panels, from their packed bytes."""
    from agens_engine_b200.ops import linear as L
    size = L.fm_bytes(32, lin.k, lin.bits, lin.group)
    w = torch.cat([L.WqLinear(32, lin.k, lin.bits, lin.group, lin.wq[p * size:(p + 1) * size]).dequant_cpu() for p in panels])
    return x.double() @ w.double().to(x.device).t(), torch.cat([torch.arange(32 * p, 32 * p + 32) for p in panels])


# all rows at once, fewer rows at a time than asked for, and a shape of which not one row fits the newer kernel's scratch
@pytest.mark.gpu
@pytest.mark.parametrize("n,k,ks,m,bits", [(57344, 8192, 1, 3, 2), (40960, 8192, 1, 8, 4), (11040, 28672, 2, 7, 3), (40960, 81920, 4, 3, 2)])
def test_allocation_free_gemv_near_its_limit(n, k, ks, m, bits):
    """bf16 result of fp16 activations: two roundings of 2^-9 and 2^-11 relative to the norm, below 4e-3."""
    from agens_engine_b200.ops import linear as L
    lib = _lib.cuda_lib()
    fn = lib.b2_wq_gemv_noalloc
    fn.argtypes = [C.c_void_p] + [C.c_int] * 5 + [C.c_void_p, C.c_long, C.c_int, C.c_void_p, C.c_long, C.c_void_p, C.c_void_p, C.c_char_p]
    fn.restype = C.c_int
    lin = L.WqLinear.random(n, k, bits, 128, "cuda:0", seed=n, ks=ks)
    x = torch.randn(m, k, device="cuda:0").to(torch.bfloat16)
    y = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda:0")
    status, err = torch.full((1,), -1, dtype=torch.int32, device="cuda:0"), C.create_string_buffer(160)
    rc = fn(lin.wq.data_ptr(), n, k, bits, 128, ks, x.data_ptr(), k, m, y.data_ptr(), n, status.data_ptr(), _lib.current_stream(), err)
    assert rc == 0, err.value
    assert int(status.item()) == 0 and bool(torch.isfinite(y).all())
    ref, rows = _panel_reference(lin, x, [0, 1, n // 64, n // 32 - 1])
    assert (y[:, rows].double() - ref).norm() < 4e-3 * ref.norm()
    one = torch.full((1, n), float("nan"), dtype=torch.bfloat16, device="cuda:0")       # a row's bits do not depend on its company
    assert fn(lin.wq.data_ptr(), n, k, bits, 128, ks, x[m - 1].data_ptr(), k, 1, one.data_ptr(), n, None, _lib.current_stream(), err) == 0
    assert torch.equal(one[0], y[m - 1])


def test_workspace_growth_is_bounded():
    """Many small steps up: what is kept stays within twice the present size, and buffers handed out stay alive."""
    from agens_engine_b200.ops import linear as L
    ws = L.GemvWorkspace("cpu", floats=100, panels=4)
    first = ws.scratch.data_ptr()
    for n in range(100, 5000, 7):
        ws.ensure_scratch(n)
        assert ws.scratch.numel() >= n and sum(t.numel() for t in ws._outgrown) <= 2 * ws.scratch.numel()
    assert ws._outgrown[0].data_ptr() == first and ws.scratch.numel() < 1.5 * 5000 + 1
    ws.ensure_scratch(3)
    assert ws.scratch.numel() >= 5000 - 7


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,floats", [(151936, 5248, 4 << 20), (2048, 5248, 1 << 10)])
def test_gemv_grows_its_workspace(n, k, floats):
    """Slices of k (above 5120 inputs) hand every panel over through scratch; a workspace that is too small for that
    grows, and a graph captured before keeps its own."""
    from agens_engine_b200.ops import linear as L
    lin, small = L.WqLinear.random(n, k, 4, 128, "cuda:0", seed=n), L.WqLinear.random(64, 512, 4, 128, "cuda:0", seed=1)
    ws = L.GemvWorkspace("cuda:0", floats=floats)
    x, xs = torch.randn(8, k, device="cuda:0").to(torch.bfloat16), torch.randn(2, 512, device="cuda:0").to(torch.bfloat16)
    ys = L.gemv(small, xs, ws, epi=_lib.EPI_F32)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        L.gemv(small, xs, ws, epi=_lib.EPI_F32, out=ys)
    y = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
    assert ws.scratch.numel() > floats
    ref, rows = _panel_reference(lin, x, [0, n // 64, n // 32 - 1])
    assert (y[:, rows].double() - ref).norm() < 1e-3 * ref.norm()
    want = ys.clone()
    ys.zero_()
    graph.replay()
    assert torch.equal(ys, want) and torch.equal(L.gemv(lin, x, ws, epi=_lib.EPI_F32), y)
    assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("bits", [2, 4])
def test_gemv_of_very_many_inputs(bits):
    """33 slices of k, one more than the hand-over of the kernel for one to eight rows has lanes."""
    from agens_engine_b200.ops import linear as L
    n, k = 96, 164352
    assert not _lib.cuda_lib().b2_wq_gemv8_takes(n, k) and _lib.cuda_lib().b2_wq_gemv8_takes(n, 163840)
    lin = L.WqLinear.random(n, k, bits, 128, "cuda:0", seed=9)
    x = torch.randn(5, k, device="cuda:0").to(torch.bfloat16)
    ws = L.GemvWorkspace("cuda:0")
    y = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
    ref, rows = _panel_reference(lin, x, [0, 1, 2])
    assert (y[:, rows].double() - ref).norm() < 1e-3 * ref.norm()
    assert torch.equal(L.gemv(lin, x[3:4], ws, epi=_lib.EPI_F32)[0], y[3])
    assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0
