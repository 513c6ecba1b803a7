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
