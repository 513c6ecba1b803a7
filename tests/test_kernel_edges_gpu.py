"""Edges of the kernels' work splits: the sizes, alignments and values at which a share, a tile or a ring is not full."""
import pytest
import torch

from agens_engine_b200 import _lib
from agens_engine_b200.ops import basic
from agens_engine_b200.ops import linear as L
from agens_engine_b200.utils import quant
from tests.test_spec_gpu import _params, ref_sample

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# a row is cut into eight shares of a multiple of four logits: shares that are empty, ragged, unaligned (odd leading
# dimension), longer than the shared memory that caches them (above 327680 logits), and rows of few distinct values
@pytest.mark.parametrize("vocab,ld,kind", [(1, 1, "normal"), (5, 8, "normal"), (33, 35, "normal"), (4097, 4099, "normal"),
                                           (20000, 20000, "ties"), (16384, 16384, "masked"), (330001, 330004, "normal")])
def test_sampler_shares(vocab, ld, kind):
    torch.manual_seed(vocab)
    rows = 2 if vocab > 100000 else 6
    x = torch.randn(rows, vocab) * 3
    if kind == "ties":
        x = torch.round(x)
    if kind == "masked":
        x[:, ::3] = float("-inf")
    buf = torch.zeros(rows, ld, device=DEV)
    buf[:, :vocab] = x.to(DEV)
    T, k, p, mp = [0.8, 1.1, 0.0, 0.7, 1.0, 0.9][:rows], [0, 40, 0, 0, 3, 0][:rows], [0.9, 0.95, 1.0, 1.0, 1.0, 0.5][:rows], [0, 0, 0, 0.1, 0, 0][:rows]
    seeds, pos = [99 + i for i in range(rows)], [7 * i for i in range(rows)]
    out = basic.sample_rows(buf, *_params(DEV, rows, T, k, p, mp, seeds, pos), n_valid=vocab).cpu().tolist()
    assert out == [ref_sample(x[i], T[i], k[i], p[i], mp[i], seeds[i], pos[i]) for i in range(rows)]


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("offset", [0, 4])
def test_dequant_blocks(bits, group, offset):
    """(code - zero) * scale rounded once to bf16, bit for bit, from aligned and from merely word-aligned buffers and
    into rows wider than the matrix; 3 x 3 blocks do not fill the last CTA."""
    n, k, ldo = 96, 384, 392
    torch.manual_seed(bits)
    ql = quant.quantize(torch.randn(n, k) * 0.02, bits, group)
    wq = quant.pack_fm(ql).reshape(-1)
    buf = torch.zeros(wq.numel() + 16, dtype=torch.uint8, device=DEV)
    buf[offset:offset + wq.numel()] = wq.to(DEV)
    out = torch.full((n, ldo), 7.0, dtype=torch.bfloat16, device=DEV)
    rc = _lib.cuda_lib().b2_wq_dequant(buf.data_ptr() + offset, n, k, bits, group, out.data_ptr(), ldo, _lib.current_stream())
    assert rc == 0
    assert torch.equal(out[:, :k].cpu(), ql.dequant().to(torch.bfloat16)) and bool((out[:, k:] == 7.0).all())


# one unit, one panel, k in two and more slices (above 5120 inputs), panels shared by CTAs, panels cut between CTAs
@pytest.mark.parametrize("n,k", [(32, 128), (160, 1024), (96, 5248), (64, 25600), (37888, 128)])
@pytest.mark.parametrize("bits,group", [(2, 64), (3, 128), (4, 128)])
def test_gemv_work_split(n, k, bits, group):
    """Every row count gives the same bits, and they agree with fp64 within the fp16 activations that carry 1 / c
    (three roundings of 2^-11 on inputs of random sign: below 1e-3 of the result's norm)."""
    lin = L.WqLinear.random(n, k, bits, group, DEV, seed=7)
    torch.cuda.synchronize()
    ws = L.GemvWorkspace(DEV)
    ws.mm_min_rows = 33
    torch.manual_seed(3)
    x = torch.randn(19, k, device=DEV).to(torch.bfloat16)
    ref = x.double() @ lin.dequant_cpu().double().to(DEV).t()
    y = L.gemv(lin, x, ws, epi=_lib.EPI_F32)
    assert (y.double() - ref).norm() < 1e-3 * ref.norm()
    for m in (1, 2, 7, 8, 9):
        assert torch.equal(L.gemv(lin, x[:m], ws, epi=_lib.EPI_F32), y[:m]), m
    assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0


# 128-row tiles, two per CTA (one up to 148 CTAs), blocks of 128 keys: chunks that leave the second tile empty or ragged, contexts at and around
# a block's end, one to 128 query heads per KV head, scores that keep growing (the reference maximum moves several times)
@pytest.mark.parametrize("T,pos0,hq,hkv,grow", [(1, 0, 8, 8, 0), (64, 63, 16, 8, 0), (64, 64, 16, 8, 0), (65, 64, 64, 8, 0), (300, 511, 8, 1, 0),
                                                (130, 700, 16, 8, 1), (3, 250, 128, 1, 1), (330, 511, 64, 8, 0), (321, 64, 64, 8, 1)])
def test_prefill_attention_tiles(T, pos0, hq, hkv, grow):
    """Against fp64; P is bf16 (relative 2^-9 per term, random), the result is rounded to bf16: below 6e-3 of the norm.
    Slots of the pool that the sequence does not use hold NaN."""
    torch.manual_seed(T + pos0)
    n = pos0 + T
    npg = (n + 15) // 16
    k, v = torch.randn(n, hkv, 128, device=DEV).to(torch.bfloat16), torch.randn(n, hkv, 128, device=DEV).to(torch.bfloat16)
    q = torch.randn(T, hq, 128, device=DEV).to(torch.bfloat16)
    if grow:
        k[:, :, 0] += torch.arange(n, device=DEV).to(torch.bfloat16)[:, None] / 20
        q[:, :, 0] = 20.0
    pool = torch.full((npg + 2, 2, hkv, 16, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    perm = torch.randperm(npg + 2)[:npg]
    for i in range(npg):
        c = min(16, n - 16 * i)
        pool[perm[i], 0, :, :c] = k[16 * i:16 * i + c].transpose(0, 1)
        pool[perm[i], 1, :, :c] = v[16 * i:16 * i + c].transpose(0, 1)
    from agens_engine_b200.ops import attention as A
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = A.attn_prefill_tc(q.reshape(T, -1).contiguous(), pool, perm.to(torch.int32)[None].to(DEV), 0, pos0, hq, hkv, status=status)
    s = torch.einsum("thd,lhd->htl", q.double(), k.double().repeat_interleave(hq // hkv, 1)) / 128 ** 0.5
    s = s.masked_fill(torch.arange(n, device=DEV)[None, None] > (pos0 + torch.arange(T, device=DEV))[None, :, None], float("-inf"))
    ref = torch.einsum("htl,lhd->thd", torch.softmax(s, -1), v.double().repeat_interleave(hq // hkv, 1)).reshape(T, -1)
    assert int(status.item()) == 0
    assert (out.double() - ref).norm() < 6e-3 * ref.norm()


# token counts around the padding (16) and the sizes at which the pipeline changes (64 / 65: two units a step or one; 128 /
# 129: two accumulators or one; 160 / 161: four operand buffers or three); one unit, an odd number of batches, a ragged
# last row tile, tiles that several CTAs share
@pytest.mark.parametrize("n,k", [(32, 128), (160, 640), (4128, 384), (256, 2176)])
@pytest.mark.parametrize("bits,group", [(2, 128), (3, 64), (4, 128)])
def test_mm_steps(n, k, bits, group):
    """Against fp64; weights are rounded to fp16 (2^-11) and the result to fp32: below 1e-3 of the norm.  A row's bits do
    not depend on the rows that travel with it."""
    lin = L.WqLinear.random(n, k, bits, group, DEV, seed=5)
    torch.cuda.synchronize()
    ws = L.GemvWorkspace(DEV)
    torch.manual_seed(4)
    x = torch.randn(256, k, device=DEV).to(torch.bfloat16)
    ref = x.double() @ lin.dequant_cpu().double().to(DEV).t()
    y = L.mm(lin, x, ws, epi=_lib.EPI_F32)
    assert (y.double() - ref).norm() < 1e-3 * ref.norm()
    for m in (1, 16, 17, 64, 65, 128, 129, 160, 161):
        assert torch.equal(L.mm(lin, x[:m], ws, epi=_lib.EPI_F32), y[:m]), m
    assert int(ws.status.item()) == 0 and int(ws.counters.abs().sum().item()) == 0


# CTAs that walk one, two and three tiles (148 CTAs; 357 and 162 tiles), ragged rows and columns, fewer k than a stage
@pytest.mark.parametrize("M,N,K", [(2100, 5128, 128), (257, 13576, 72), (1, 8, 8)])
def test_gemm_tiles(M, N, K):
    """Against fp64 in fp32 output: products are exact, sums are fp32 (K roundings of 2^-24)."""
    from agens_engine_b200.ops import gemm as G
    torch.manual_seed(M)
    a, b = torch.randn(M, K, device=DEV).to(torch.bfloat16), torch.randn(N, K, device=DEV).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    d = G.gemm_bf16(a, b, out_f32=True, status=status)
    ref = a.double() @ b.double().t()
    assert int(status.item()) == 0
    assert (d.double() - ref).norm() < 1e-5 * ref.norm()


# CTAs per row: eight (with greedy rows on one), four, two and one, by rows and vocabulary, more of them for a row on its own
@pytest.mark.parametrize("rows,vocab,ld", [(40, 190001, 190004), (80, 20000, 20000), (50, 40000, 40000), (80, 20001, 20003), (300, 1000, 1000), (300, 7, 9)])
def test_sampler_rows_do_not_depend_on_their_company(rows, vocab, ld):
    torch.manual_seed(rows)
    buf = torch.zeros(rows, ld, device=DEV)
    x = torch.randn(rows, vocab, device=DEV) * 3
    x[1::3] = torch.round(x[1::3])
    x[2::5, ::2] = float("-inf")
    x[4] = float("-inf")
    x[9, : vocab // 2] = float("nan")
    buf[:, :vocab] = x
    i = list(range(rows))
    T, k, p, mp = [0.0 if j % 4 == 0 or j == 9 else 0.6 + 0.1 * (j % 5) for j in i], [(0, 1, 40, 3)[j % 4] for j in i], [(1.0, 0.9, 0.5)[j % 3] for j in i], [(0.0, 0.05)[j % 2] for j in i]
    seeds, pos = [99 + j for j in i], [7 * j for j in i]
    args = _params(DEV, rows, T, k, p, mp, seeds, pos)
    out = basic.sample_rows(buf, *args, n_valid=vocab).cpu()
    one = [int(basic.sample_rows(buf[j:j + 1], *(a[j:j + 1].contiguous() for a in args), n_valid=vocab)) for j in i]
    assert out.tolist() == one
    greedy = [j for j in i if T[j] == 0.0 and j != 9]
    assert out[greedy].tolist() == x[greedy].argmax(-1).tolist()
    assert int(out[9]) == vocab // 2 + int(x[9, vocab // 2:].argmax())
