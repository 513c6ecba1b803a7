"""GPU gates of the mixed-bit GEMVs (model: the reference's kernels/bench/test_w4.cu and test_wq.cu: GEMV vs a
high-precision reference, batched == single bitwise, repack round trip).  ``L.gemv`` runs the kernel for one to eight rows,
which cuts k into slices of at most 5120 inputs by itself; ``_k_slices`` calls the one that takes ``ks`` and ``rb``."""
import ctypes as C

import pytest
import torch

from agens_engine_b200 import _lib
from agens_engine_b200.ops import linear as L
from agens_engine_b200.utils import quant

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mk(n, k, bits, group, seed=0, ks=None):
    torch.manual_seed(seed)
    w = torch.randn(n, k) * 0.02
    ql = quant.quantize(w, bits, group)
    return ql, L.WqLinear.from_quant(ql, DEV, ks=ks)


def _ref(ql, x):
    return x.float().cpu().double() @ ql.dequant().double().t()


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("n,k", [(160, 1024), (96, 5248), (64, 25600)])
def test_gemv_matches_fp64(bits, group, n, k):
    ql, lin = _mk(n, k, bits, group)
    ws = L.GemvWorkspace(DEV)
    ws.mm_min_rows = 33          # these tests exercise the GEMV at every row count
    for m in (1, 3, 8, 13, 32):
        x = (torch.randn(m, k) * 1.5).to(torch.bfloat16).to(DEV)
        y = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
        ref = _ref(ql, x)
        err = (y.cpu().double() - ref).abs().max().item()
        assert err < 2e-3 * ref.abs().max().item() + 1e-4, (bits, group, m, err)


@pytest.mark.parametrize("bits", [2, 3, 4])
def test_dequant_kernel_matches_cpu(bits):
    ql, lin = _mk(64, 512, bits, 128, seed=3)
    d = lin.dequant().float().cpu()
    assert torch.equal(d, ql.dequant().to(torch.bfloat16).float())
    assert torch.equal(lin.dequant_cpu(), ql.dequant())


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("sym", [False, True])
def test_device_repack_matches_cpu_pack(bits, sym):
    torch.manual_seed(5)
    n, k, group = 64, 512, 64
    w = torch.randn(n, k) * 0.02
    ql = quant.quantize(w, bits, group, symmetric=sym, scale_dtype=torch.bfloat16 if sym else torch.float16)
    packed = quant.pack_stream(ql.codes, bits)
    lin = L.WqLinear.from_checkpoint(packed, ql.scale.to(torch.bfloat16) if sym else ql.scale,
                                     None if sym else ql.zero, n, k, bits, group, DEV)
    assert torch.equal(lin.wq.cpu(), quant.pack_fm(ql).reshape(-1))


def test_rows_do_not_depend_on_batch():
    """Batch invariance: a token's output bits are the same at m = 1, inside m = 8 and inside m = 16."""
    for bits, k in ((2, 2048), (3, 5248), (4, 10368)):
        ql, lin = _mk(128, k, bits, 128, seed=bits)
        ws = L.GemvWorkspace(DEV)
        ws.mm_min_rows = 33          # these tests exercise the GEMV at every row count
        x = torch.randn(16, k).to(torch.bfloat16).to(DEV)
        y16 = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
        y8 = L.gemv(lin, x[:8].contiguous(), ws, epi=_lib.EPI_F32)
        y1 = L.gemv(lin, x[5:6].contiguous(), ws, epi=_lib.EPI_F32)
        assert torch.equal(y16[:8], y8)
        assert torch.equal(y16[5:6], y1)
        x32 = torch.cat([x, x], 0)
        y32 = L.gemv(lin, x32, ws, epi=_lib.EPI_F32)
        assert torch.equal(y32[:16], y16) and torch.equal(y32[16:], y16)


def test_gemv_is_deterministic():
    ql, lin = _mk(256, 4096, 3, 128, seed=9, ks=4)
    ws = L.GemvWorkspace(DEV)
    ws.mm_min_rows = 33          # these tests exercise the GEMV at every row count
    x = torch.randn(4, 4096).to(torch.bfloat16).to(DEV)
    y0 = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
    for _ in range(20):
        assert torch.equal(L.gemv(lin, x, ws, epi=_lib.EPI_F32), y0)


def test_norm_prologue_and_residual_epilogue():
    torch.manual_seed(11)
    d, n = 1024, 256
    ql, lin = _mk(n, d, 4, 128, seed=1)
    qlo, lino = _mk(d, n, 4, 128, seed=2, ks=1)
    ws = L.GemvWorkspace(DEV)
    ws.mm_min_rows = 33          # these tests exercise the GEMV at every row count
    m = 3
    h = torch.randn(m, d).to(torch.bfloat16).to(DEV)
    nw = (1 + 0.1 * torch.randn(d)).to(torch.bfloat16).to(DEV)
    ss = torch.zeros(4, L.SS_LD, dtype=torch.float32, device=DEV)
    hf = h.float()
    # partial sums of squares over 4 column slices
    for p in range(4):
        ss[p, :m] = (hf[:, p * 256:(p + 1) * 256] ** 2).sum(-1)
    y = L.gemv(lin, h, ws, pro=_lib.PRO_NORM, ss_in=ss, ss_parts=4, norm_w=nw, eps=1e-6, epi=_lib.EPI_F32)
    xn = (hf * torch.rsqrt((hf ** 2).mean(-1, keepdim=True) + 1e-6) * nw.float()).to(torch.bfloat16)
    ref = _ref(ql, xn)
    assert (y.cpu().double() - ref).abs().max().item() < 3e-3 * ref.abs().max().item() + 1e-4
    # residual epilogue: y = bf16(acc + resid), ss_out = per panel sums of squares of y
    x2 = torch.randn(m, n).to(torch.bfloat16).to(DEV)
    resid = torch.randn(m, d).to(torch.bfloat16).to(DEV)
    ss_out = torch.zeros(lino.n_panels(), L.SS_LD, dtype=torch.float32, device=DEV)
    out = L.gemv(lino, x2, ws, epi=_lib.EPI_RESID, resid=resid, ss_out=ss_out)
    ref2 = (_ref(qlo, x2) + resid.float().cpu().double())
    assert (out.float().cpu().double() - ref2).abs().max().item() < 0.02 * ref2.abs().max().item()
    tot = ss_out[:, :m].sum(0).cpu()
    assert torch.allclose(tot, (out.float() ** 2).sum(-1).cpu(), rtol=1e-4)


def test_swiglu_epilogue():
    torch.manual_seed(12)
    f, d, m = 256, 512, 5
    gate = torch.randn(f, d) * 0.05
    up = torch.randn(f, d) * 0.05
    ql = quant.quantize(quant.interleave_gate_up(gate, up), 4, 128)
    lin = L.WqLinear.from_quant(ql, DEV, ks=2)
    x = torch.randn(m, d).to(torch.bfloat16).to(DEV)
    act = L.gemv(lin, x, L.GemvWorkspace(DEV), epi=_lib.EPI_SWIGLU)
    wd = ql.dequant().reshape(f // 8, 16, d)
    g = (x.float().cpu() @ wd[:, :8].reshape(f, d).t()).to(torch.bfloat16).float()
    u = (x.float().cpu() @ wd[:, 8:].reshape(f, d).t()).to(torch.bfloat16).float()
    ref = (torch.nn.functional.silu(g) * u)
    assert (act.float().cpu() - ref).abs().max().item() < 0.02 * ref.abs().max().item() + 1e-3


def test_argmax_epilogue():
    from agens_engine_b200.ops import basic
    torch.manual_seed(13)
    n, d, m = 1000 * 16, 512, 4
    ql, lin = _mk(n, d, 4, 128, seed=4, ks=2)
    x = torch.randn(m, d).to(torch.bfloat16).to(DEV)
    val = torch.empty(lin.n_panels(), L.SS_LD, dtype=torch.float32, device=DEV)
    idx = torch.empty(lin.n_panels(), L.SS_LD, dtype=torch.int32, device=DEV)
    logits = torch.empty(m, n, dtype=torch.float32, device=DEV)
    L.gemv(lin, x, L.GemvWorkspace(DEV), epi=_lib.EPI_ARGMAX, amax_val=val, amax_idx=idx, n_valid=n - 100, yf=logits)
    ids = basic.argmax_final(val, idx, lin.n_panels(), m, L.SS_LD)
    assert torch.equal(ids.long().cpu(), logits[:, : n - 100].argmax(-1).cpu())
    assert torch.equal(basic.argmax_rows(logits, n - 100).long().cpu(), logits[:, : n - 100].argmax(-1).cpu())


def test_random_init_on_device_is_a_valid_quantisation():
    lin = L.WqLinear.random(64, 512, 3, 128, DEV, seed=42)
    w = lin.dequant_cpu()
    assert abs(w.std().item() - 0.02) < 0.004 and abs(w.mean().item()) < 0.002
    assert torch.equal(lin.dequant().float().cpu(), w.to(torch.bfloat16).float())


# one, two and five slices of k; panels that CTAs share and that they do not (one slice, many panels)
@pytest.mark.parametrize("n,k", [(128, 1024), (37888, 256), (128, 5248), (96, 25600)])
@pytest.mark.parametrize("bits,group", [(4, 128), (3, 64)])
def test_every_epilogue_over_slices_of_k(n, k, bits, group):
    """The norm prologue (its offset into every slice) and each epilogue, finished by whichever CTA arrives last, against
    fp64; rows 0, 2 and 7 on their own and among eight and nine give the same bits.  fp32 results carry the fp16 rounding of the
    activations (below 1e-3 of the norm, 2e-3 where bf16 roundings of the norm flip), bf16 results 2^-9 on top."""
    torch.manual_seed(n + k)
    lin = L.WqLinear.random(n, k, bits, group, DEV, seed=k)
    w = lin.dequant_cpu().double().to(DEV)
    ws = L.GemvWorkspace(DEV)
    ws.mm_min_rows = 33
    M, parts = 9, 5
    h = torch.randn(M, k, device=DEV).to(torch.bfloat16)
    nw = (1 + 0.1 * torch.randn(k, device=DEV)).to(torch.bfloat16)
    ss = torch.zeros(parts, L.SS_LD, device=DEV)
    ss[:, :M] = torch.stack([c.float().pow(2).sum(-1) for c in h.chunk(parts, -1)])
    xn = (h.float() * torch.rsqrt(h.float().pow(2).mean(-1, keepdim=True) + 1e-6) * nw.float()).to(torch.bfloat16)
    resid = torch.randn(M, n, device=DEV).to(torch.bfloat16)
    plain, normed = h.double() @ w.t(), xn.double() @ w.t()
    near = lambda a, b, tol: bool((a.double() - b).norm() < tol * b.norm())

    def run(rows):
        x, r = h[rows].contiguous(), resid[rows].contiguous()
        m = x.shape[0]
        s = torch.zeros(parts, L.SS_LD, device=DEV)
        s[:, :m] = ss[:, rows]
        norm = dict(pro=_lib.PRO_NORM, ss_in=s, ss_parts=parts, norm_w=nw, eps=1e-6)
        sso = torch.zeros(lin.n_panels(), L.SS_LD, device=DEV)
        val, idx = torch.empty_like(sso), torch.empty(lin.n_panels(), L.SS_LD, dtype=torch.int32, device=DEV)
        yf = torch.empty(m, n, device=DEV)
        L.gemv(lin, x, ws, epi=_lib.EPI_ARGMAX, amax_val=val, amax_idx=idx, n_valid=n - 40, yf=yf, **norm)
        out = dict(store=L.gemv(lin, x, ws), f32=L.gemv(lin, x, ws, epi=_lib.EPI_F32, **norm), swiglu=L.gemv(lin, x, ws, epi=_lib.EPI_SWIGLU, **norm),
                   resid=L.gemv(lin, x, ws, epi=_lib.EPI_RESID, resid=r, ss_out=sso), ss=sso[:, :m].t().contiguous(), yf=yf,
                   val=val[:, :m].t().contiguous(), idx=idx[:, :m].t().contiguous())
        assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0
        return out

    y = run(list(range(M)))
    assert near(y["store"], plain, 4e-3) and near(y["f32"], normed, 2e-3) and torch.equal(y["yf"], y["f32"])
    assert near(y["resid"], plain + resid.double(), 4e-3)
    assert near(y["ss"], y["resid"].double().pow(2).view(M, -1, 32).sum(-1), 1e-6)
    g, u = normed.view(M, -1, 2, 8).unbind(2)
    assert near(y["swiglu"], (torch.nn.functional.silu(g) * u).reshape(M, -1), 1e-2)
    ok = y["yf"].masked_fill(torch.arange(n, device=DEV) >= n - 40, float("-inf")).view(M, -1, 32)
    assert torch.equal(y["val"], ok.amax(-1))
    live = y["val"] > float("-inf")
    assert torch.equal(y["idx"][live].long(), (ok.argmax(-1) + 32 * torch.arange(n // 32, device=DEV))[live])
    for rows in ([0], [2], [7], [0, 2, 7], list(range(8))):
        for name, v in run(rows).items():
            assert torch.equal(v, y[name][rows]), (rows, name)


def _k_slices(lin, x, ks, rb, epi, ws, **kw):
    """b2_wq_gemv itself: the kernel that the tensor-parallel epilogue runs on."""
    lib, ptr = _lib.cuda_lib(), _lib.ptr
    a = _lib.WqGemvArgs()
    a.wq, a.n, a.k, a.m, a.bits, a.group, a.ks, a.rb = ptr(lin.wq), lin.n, lin.k, x.shape[0], lin.bits, lin.group, ks, rb
    a.vworkers, a.fmax = lib.b2_wq_gemv_vworkers(lin.n, lin.k, ks, rb), lib.b2_wq_gemv_fmax(lin.n, lin.k, ks, rb)
    a.x, a.ldx, a.epi, a.ss_ld = ptr(x), x.stride(0), epi, L.SS_LD
    out = torch.empty(x.shape[0], lin.n, dtype=torch.float32 if epi == _lib.EPI_F32 else torch.bfloat16, device=DEV)
    a.yf, a.y, a.ldy = (ptr(out), None, lin.n) if epi == _lib.EPI_F32 else (None, ptr(out), lin.n)
    if "resid" in kw:
        a.resid, a.ldr, a.ss_out = ptr(kw["resid"]), kw["resid"].stride(0), ptr(kw["ss_out"])
    if "tp" in kw:
        a.tp = kw["tp"]
    ws.ensure_scratch(lib.b2_wq_gemv_scratch_floats(lin.n, lin.k, ks, rb, x.shape[0]))
    a.scratch, a.counters, a.status = ptr(ws.scratch), ptr(ws.counters), ptr(ws.status)
    assert lib.b2_wq_gemv(C.byref(a), _lib.current_stream()) == 0
    return out


@pytest.mark.parametrize("bits,group", [(2, 128), (3, 64), (4, 128)])
@pytest.mark.parametrize("ks", [1, 2, 8])
def test_kernel_with_k_slices(bits, group, ks):
    """fp64, and the same bits whatever the rows per item and the rows that travel together."""
    n, k = 160, 1024
    ql, lin = _mk(n, k, bits, group)
    ws = L.GemvWorkspace(DEV)
    x = (torch.randn(32, k) * 1.5).to(torch.bfloat16).to(DEV)
    y = _k_slices(lin, x, ks, 2, _lib.EPI_F32, ws)
    ref = _ref(ql, x)
    assert (y.cpu().double() - ref).norm() < 1e-3 * ref.norm()
    for m, rb in ((1, 2), (1, 4), (3, 2), (8, 4), (13, 4), (16, 2)):
        assert torch.equal(_k_slices(lin, x[:m], ks, rb, _lib.EPI_F32, ws), y[:m]), (m, rb)
    assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0


@pytest.mark.parametrize("ks,m", [(1, 1), (2, 5), (4, 16)])
def test_push_epilogue_of_a_single_rank(ks, m):
    """A group of one: the rank pushes into its own inbox and sums that, so the result is the residual epilogue's, bit for
    bit, and the slot named for clearing is armed again."""
    n, k = 96, 1024
    ql, lin = _mk(n, k, 4, 128, seed=6)
    ws = L.GemvWorkspace(DEV)
    x, resid = torch.randn(m, k).to(torch.bfloat16).to(DEV), torch.randn(m, n).to(torch.bfloat16).to(DEV)
    slot = m * n
    inbox = torch.full((2 * slot,), -0.0, device=DEV)
    inbox[slot:] = 3.0                                        # the slot that this call re-arms
    tp = _lib.TpPush()
    tp.inbox[0], tp.rank, tp.size, tp.slot_off, tp.clear_off, tp.slot_stride = inbox.data_ptr(), 0, 1, 0, slot, slot
    tp.status, tp.timeout_ns = ws.status.data_ptr(), 1_000_000_000
    ss = [torch.zeros(lin.n_panels(), L.SS_LD, device=DEV) for _ in range(2)]
    want = _k_slices(lin, x, ks, 2, _lib.EPI_RESID, ws, resid=resid, ss_out=ss[0])
    got = _k_slices(lin, x, ks, 2, _lib.EPI_TP_RESID, ws, resid=resid, ss_out=ss[1], tp=tp)
    assert int(ws.status.item()) == 0
    assert torch.equal(got, want) and torch.equal(ss[0], ss[1])
    assert bool((inbox[slot:] == 0).all()) and bool(torch.signbit(inbox[slot:]).all())
