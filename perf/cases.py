"""The work that a user of this engine has it do, as cases that can be timed and checked.

Every case goes through an entry point that a program calls: the quantised linears (``ops.linear.gemv`` / ``mm``,
``ops.gemm.wq_linear``), paged attention (``ops.attention.attn_decode`` / ``attn_prefill``), the sampler
(``ops.basic.sample_rows``) and the model (``DenseModel.forward_rows`` / ``prefill``).  Sizes are those of the engine's
own configurations (``dense_32b``, ``drafter_0p6b``), of its serving defaults (page size 16, 64-key splits, prefill
chunks of 256 to 2048 rows) and odd ones between them.  Weights are Gaussian values quantised to 2, 3 or 4 bits in the
checkpoint container (bit stream, fp16 scale and zero point per group), which the engine repacks on the device as its
loader does; the 64-bit results unpack the same containers in plain torch.
"""
from __future__ import annotations

import math

import torch

from agens_engine_b200._lib import EPI_RESID, EPI_SWIGLU, PRO_NORM
from agens_engine_b200.models import config as C
from agens_engine_b200.models.dense import DenseModel
from agens_engine_b200.ops import attention as A
from agens_engine_b200.ops import basic
from agens_engine_b200.ops import gemm as G
from agens_engine_b200.ops import linear as L

DEV = "cuda:0"
EPS = 1e-6
# d_model, q heads, kv heads, ffn of the engine's two dense configurations (head dimension 128)
DIMS = {"dense": (5120, 64, 8, 25600), "drafter": (1024, 16, 8, 3072)}
HD = 128
VOCAB = 151936
LINEARS = ("qkv", "o", "gate_up", "down")


# ---------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one token of the companion drafter: its layers' linears one after the other, in a CUDA graph as a drafting loop
        # replays them (four small products a layer, bound by launches and latency)
        dict(name="drafter_layers_1row", family="layers", dims="drafter", rows=1, layers=4, bits="4444", group=128),
        # one token of the 32B decoder, greedy decode of a single conversation: two layers' linears in a CUDA graph
        dict(name="layers_1row", family="layers", dims="dense", rows=1, layers=2, bits="3424", group=128),
        # a verify block of a draft of five tokens: the same products for six rows
        dict(name="layers_6rows", family="layers", dims="dense", rows=6, layers=2, bits="4233", group=128),
        # batched decode of 24 conversations
        dict(name="layers_24rows", family="layers", dims="dense", rows=24, layers=2, bits="4342", group=128),
        # one product of a prefill chunk that is not full (the default chunk is 256 rows)
        dict(name="linear_200rows", family="linear", dims="dense", linear="o", rows=200, bits=3, group=64),
        # the widest product of a 2048-row prefill chunk (long prompts)
        dict(name="linear_2048rows", family="linear", dims="dense", linear="gate_up", rows=2048, bits=4, group=128),
        # attention of a decode step of 16 conversations with contexts of different lengths
        dict(name="attn_decode_16seqs", family="attn_decode", dims="dense", seqs=16, rows=1, ctx=3000),
        # attention of a verify block of four rows at the end of one long context
        dict(name="attn_verify_long", family="attn_decode", dims="dense", seqs=1, rows=4, ctx=30011),
        # attention of a 2048-row prefill chunk after 6144 tokens
        dict(name="attn_prefill_2048", family="attn_prefill", dims="dense", rows=2048, pos0=6144),
        # sampling of a decode step of 16 conversations (temperature, top-k, top-p, min-p and greedy rows)
        dict(name="sample_16rows", family="sample", rows=16, vocab=VOCAB),
        # a whole verify step through the model: eight rows of two conversations, logits out, rolled back afterwards
        dict(name="model_step_8rows", family="model_step", layers=2, seqs=2, rows=4, ctx=500),
        # a whole prompt through the model in chunks of the default size, the last chunk ragged, logits out
        dict(name="model_prefill_700", family="model_prefill", layers=2, tokens=700, chunk=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["layers", "layers", "layers", "linear", "linear", "attn_decode", "attn_decode", "attn_prefill", "sample",
                         "model_step", "model_prefill"])
    bits = lambda: "".join(rng.choice("234") for _ in range(4))
    if family == "layers":
        dims = rng.choice(["dense", "dense", "drafter"])
        return dict(family=family, dims=dims, rows=_log(rng, 1, 32), layers=rng.choice([1, 2]), bits=bits(), group=rng.choice([64, 128, 128]))
    if family == "linear":
        return dict(family=family, dims="dense", linear=rng.choice(LINEARS), rows=_log(rng, 33, 2048), bits=rng.choice([2, 3, 4]),
                    group=rng.choice([64, 128, 128]))
    if family == "attn_decode":
        if rng.random() < 0.5:
            return dict(family=family, dims=rng.choice(["dense", "dense", "drafter"]), seqs=_log(rng, 2, 32), rows=rng.randint(1, 4),
                        ctx=_log(rng, 40, 4000))
        return dict(family=family, dims="dense", seqs=1, rows=rng.randint(1, 8), ctx=_log(rng, 100, 60000))
    if family == "attn_prefill":
        return dict(family=family, dims=rng.choice(["dense", "dense", "drafter"]), rows=_log(rng, 64, 2048), pos0=rng.choice([0, _log(rng, 16, 6144)]))
    if family == "sample":
        return dict(family=family, rows=_log(rng, 1, 32), vocab=rng.choice([VOCAB, VOCAB, 32000, 65537]))
    if family == "model_step":
        seqs = rng.randint(1, 4)
        return dict(family=family, layers=rng.choice([1, 2]), seqs=seqs, rows=rng.randint(1, 8 // max(seqs // 2, 1)), ctx=_log(rng, 20, 700))
    return dict(family=family, layers=rng.choice([1, 2]), tokens=_log(rng, 30, 1100), chunk=rng.choice([256, 512]))


# ------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _shape(dims, linear):
    d, hq, hkv, ffn = DIMS[dims]
    return {"qkv": ((hq + 2 * hkv) * HD, d), "o": (d, hq * HD), "gate_up": (2 * ffn, d), "down": (d, ffn)}[linear]


def _weights(seed, n, k, bits, group):
    """One quantised linear in the checkpoint container: int32 [n, k * bits / 32] bit stream, fp16 scale and zero point
    [n, k / group] of Gaussian weights whose range of about three deviations each way fills the code range."""
    g = _gen(seed)
    top = (1 << bits) - 1
    std = 0.5 / math.sqrt(k)
    scale = (std * 6.0 / (top + 1) * (0.8 + 0.4 * torch.rand(n, k // group, device=DEV, generator=g))).half()
    zero = (top / 2.0 + 0.5 * (torch.rand(n, k // group, device=DEV, generator=g) - 0.5)).half()
    packed = torch.empty(n, k * bits // 32, dtype=torch.int32, device=DEV)
    step = max(1, (16 << 20) // k)
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        c = torch.randn(r1 - r0, k, device=DEV, generator=g).mul_((top + 1) / 6.0).add_(top / 2.0).round_().clamp_(0, top).to(torch.int64)
        c = c.view(r1 - r0, k // 32, 32)
        words = torch.zeros(r1 - r0, k // 32, bits, dtype=torch.int64, device=DEV)
        for i in range(32):
            w, s = divmod(i * bits, 32)
            words[..., w] |= (c[..., i] << s) & 0xFFFFFFFF
            if s + bits > 32:
                words[..., w + 1] |= c[..., i] >> (32 - s)
        packed[r0:r1] = torch.where(words >= (1 << 31), words - (1 << 32), words).to(torch.int32).view(r1 - r0, -1)
    return packed, scale, zero


def _linear(seed, n, k, bits, group):
    packed, scale, zero = _weights(seed, n, k, bits, group)
    return L.WqLinear.from_checkpoint(packed, scale, zero, n, k, bits, group, DEV)


def _bits(case, linear):
    return int(case["bits"][LINEARS.index(linear)])


def _norm_weight(g, d):
    return (1.0 + 0.05 * torch.randn(d, device=DEV, generator=g)).to(torch.bfloat16)


def _layers_inputs(case, seed):
    d, hq, hkv, ffn = DIMS[case["dims"]]
    g = _gen(seed)
    h = torch.randn(case["rows"], d, device=DEV, generator=g).to(torch.bfloat16)
    per = [dict(attn=torch.randn(case["rows"], hq * HD, device=DEV, generator=g).to(torch.bfloat16), ln1=_norm_weight(g, d), ln2=_norm_weight(g, d))
           for _ in range(case["layers"])]
    return h, per


def _prepare_layers(case, seed):
    d, hq, hkv, ffn = DIMS[case["dims"]]
    m = case["rows"]
    h, per = _layers_inputs(case, seed)
    ws = L.GemvWorkspace(DEV, floats=16 << 20)
    parts = max(d // 32, 1)
    bf = lambda n: torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    ss0 = torch.zeros(parts, L.SS_LD, dtype=torch.float32, device=DEV)
    basic.sumsq(h, ss0)
    layers, outs = [], []
    for l, p in enumerate(per):
        lay = dict(p)
        for i, lin in enumerate(LINEARS):
            n, k = _shape(case["dims"], lin)
            lay[lin] = _linear(seed * 1000 + l * 8 + i + 1, n, k, _bits(case, lin), case["group"])
        lay["y"] = dict(qkv=bf((hq + 2 * hkv) * HD), h1=bf(d), act=bf(ffn), h2=bf(d))
        lay["ss1"], lay["ss2"] = torch.zeros_like(ss0), torch.zeros_like(ss0)
        layers.append(lay)
        outs += [lay["y"][x] for x in ("qkv", "h1", "act", "h2")]

    def body():
        x, ss, ssp = h, ss0, 1
        for lay in layers:
            y = lay["y"]
            L.gemv(lay["qkv"], x, ws, pro=PRO_NORM, ss_in=ss, ss_parts=ssp, norm_w=lay["ln1"], eps=EPS, out=y["qkv"])
            L.gemv(lay["o"], lay["attn"], ws, epi=EPI_RESID, resid=x, out=y["h1"], ss_out=lay["ss1"])
            L.gemv(lay["gate_up"], y["h1"], ws, pro=PRO_NORM, ss_in=lay["ss1"], ss_parts=lay["o"].n_panels(), norm_w=lay["ln2"], eps=EPS,
                   epi=EPI_SWIGLU, out=y["act"])
            L.gemv(lay["down"], y["act"], ws, epi=EPI_RESID, resid=y["h1"], out=y["h2"], ss_out=lay["ss2"])
            x, ss, ssp = y["h2"], lay["ss2"], lay["down"].n_panels()

    # decode steps are captured once per shape and replayed, as DenseModel.decode_graph does
    st = torch.cuda.Stream(device=DEV)
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        body()
    torch.cuda.current_stream().wait_stream(st)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        body()
    return dict(family="layers", graph=graph, outs=outs, keep=(h, ss0, layers, ws, st))


def _linear_inputs(case, seed):
    n, k = _shape(case["dims"], case["linear"])
    return torch.randn(case["rows"], k, device=DEV, generator=_gen(seed)).to(torch.bfloat16)


class _Owner:
    """Holds the buffers that the engine keeps between calls (the dequantised weights of a long prefill chunk)."""


def _attn_inputs(case, seed):
    d, hq, hkv, ffn = DIMS[case["dims"]]
    g = _gen(seed)
    if case["family"] == "attn_prefill":
        ctx = [case["pos0"] + case["rows"]]
        rows = case["rows"]
    else:
        # contexts between a third of the nominal length and all of it (one conversation: exactly that length)
        cpu = torch.Generator().manual_seed(int(case["ctx"]) * 131 + case["seqs"])
        ctx = [case["ctx"]] if case["seqs"] == 1 else [max(case["rows"], int(case["ctx"] * (1.0 / 3 + 2.0 / 3 * float(torch.rand(1, generator=cpu)))))
                                                       for _ in range(case["seqs"])]
        ctx = [max(c, case["rows"]) for c in ctx]
        rows = case["rows"]
    per = [(c + 15) // 16 for c in ctx]
    pages = sum(per) + 3
    kv = torch.randn(pages, 2, hkv, 16, HD, device=DEV, generator=g).to(torch.bfloat16)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(int(seed)))
    cap = max(per)
    table = torch.full((len(ctx), cap), -1, dtype=torch.int32)
    at = 0
    for s, p in enumerate(per):
        table[s, :p] = order[at:at + p].to(torch.int32)
        at += p
    n_tok = rows * len(ctx)
    q = torch.randn(n_tok, hq * HD, device=DEV, generator=g).to(torch.bfloat16)
    return ctx, rows, kv, table.to(DEV), q


def _sample_inputs(case, seed):
    g = _gen(seed)
    r = case["rows"]
    logits = 2.5 * torch.randn(r, case["vocab"], device=DEV, generator=g)
    i = torch.arange(r, device=DEV)
    # most rows with top-k and top-p, every fourth without top-k, every fifth with min-p, every seventh greedy
    temp = torch.where(i % 7 == 6, 0.0, 0.7 + 0.05 * (i % 5)).float()
    top_k = torch.where(i % 4 == 3, 0, 20 + 10 * (i % 4)).int()
    top_p = torch.where(i % 6 == 5, 1.0, 0.9).float()
    min_p = torch.where(i % 5 == 4, 0.02, 0.0).float()
    seeds = torch.randint(1, 1 << 40, (r,), device=DEV, generator=g)
    pos = torch.randint(1, 5000, (r,), device=DEV, generator=g).int()
    return dict(logits=logits, temperature=temp, top_k=top_k, top_p=top_p, min_p=min_p, seed=seeds, position=pos)


def _model_parts(case, seed):
    """Weights of a cut of the 32B configuration: per layer the four linears and two norms, embedding, norm, head."""
    cfg = C.scaled(C.dense_32b(seed=0), case["layers"])
    g = _gen(seed)
    norms = [(_norm_weight(g, cfg.d_model), _norm_weight(g, cfg.d_model)) for _ in range(cfg.n_layers)]
    final = _norm_weight(g, cfg.d_model)
    embed = torch.empty(cfg.vocab, cfg.d_model, dtype=torch.bfloat16, device=DEV).normal_(0, 1, generator=g)
    return cfg, norms, final, embed


def _model_seed(seed, layer, i):
    return seed * 1000 + layer * 8 + i + 1


def _build_model(case, seed, **kw):
    cfg, norms, final, embed = _model_parts(case, seed)
    m = DenseModel(cfg, DEV, **kw)
    for l in range(cfg.n_layers):
        lay = {"ln1": norms[l][0], "ln2": norms[l][1]}
        for i, lin in enumerate(LINEARS):
            n, k = _shape("dense", lin)
            lay[lin] = _linear(_model_seed(seed, l, i), n, k, cfg.bits_of(l, lin), cfg.group)
        m.layers.append(lay)
    m.embed, m.final_norm = embed, final
    m.lm_head = _linear(_model_seed(seed, 999, 7), cfg.vocab, cfg.d_model, cfg.lm_head_bits, cfg.group)
    return m.finalize()


def _prompt(seed, n, salt):
    return torch.randint(0, VOCAB, (n,), generator=torch.Generator().manual_seed(int(seed) * 7 + salt))


def prepare(case, seed):
    f = case["family"]
    if f == "layers":
        return _prepare_layers(case, seed)
    if f == "linear":
        n, k = _shape(case["dims"], case["linear"])
        lin = _linear(seed * 1000 + 1, n, k, case["bits"], case["group"])
        return dict(family=f, lin=lin, x=_linear_inputs(case, seed), ws=L.GemvWorkspace(DEV, floats=16 << 20), owner=_Owner())
    if f == "attn_decode":
        d, hq, hkv, ffn = DIMS[case["dims"]]
        ctx, rows, kv, table, q = _attn_inputs(case, seed)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        splits = (max(ctx) + 63) // 64
        n_tok = q.shape[0]
        return dict(family=f, q=q, kv=kv, table=table, g0=i32([i * rows for i in range(len(ctx))]), gc=i32([rows] * len(ctx)),
                    pos=i32([c - rows + j for c in ctx for j in range(rows)]), seq=i32([s for s in range(len(ctx)) for _ in range(rows)]),
                    hq=hq, hkv=hkv, splits=splits,
                    part_o=torch.empty(n_tok, hq, splits, HD, dtype=torch.float32, device=DEV),
                    part_ml=torch.empty(n_tok, hq, splits, 2, dtype=torch.float32, device=DEV),
                    status=torch.zeros(1, dtype=torch.int32, device=DEV), out=torch.empty(n_tok, hq * HD, dtype=torch.bfloat16, device=DEV))
    if f == "attn_prefill":
        d, hq, hkv, ffn = DIMS[case["dims"]]
        ctx, rows, kv, table, q = _attn_inputs(case, seed)
        return dict(family=f, q=q, kv=kv, table=table, pos0=case["pos0"], hq=hq, hkv=hkv, status=torch.zeros(1, dtype=torch.int32, device=DEV))
    if f == "sample":
        return dict(family=f, args=_sample_inputs(case, seed))
    if f == "model_step":
        m = _build_model(case, seed, max_seqs=case["seqs"], max_ctx=1024)
        m.row_graphs = True
        for s in range(case["seqs"]):
            m.new_seq(s)
            m.prefill(s, _prompt(seed, case["ctx"] + 3 * s, s))
        ids = _prompt(seed, case["seqs"] * case["rows"], 99).tolist()
        state = dict(family=f, model=m, ids=ids, seqs=[s for s in range(case["seqs"]) for _ in range(case["rows"])],
                     lens=[case["ctx"] + 3 * s for s in range(case["seqs"])])
        run(state)
        return state
    m = _build_model(case, seed, max_seqs=1, max_ctx=1280, prefill_chunk=case["chunk"])
    m.new_seq(0)
    return dict(family=f, model=m, prompt=_prompt(seed, case["tokens"], 0).to(torch.int32).to(DEV))


# --------------------------------------------------------------------------------------------------------------- passes
def run(state):
    f = state["family"]
    if f == "layers":
        state["graph"].replay()
        return state["outs"]
    if f == "linear":
        # the engine's rule for a prefill chunk: up to 256 rows multiply the packed weights, longer chunks expand them first
        if state["x"].shape[0] <= 256:
            return L.mm(state["lin"], state["x"], state["ws"])
        return G.wq_linear(state["lin"], state["x"], state["owner"])
    if f == "attn_decode":
        s = state
        return A.attn_decode(s["q"], s["kv"], s["table"], s["g0"], s["gc"], s["pos"], s["seq"], s["hq"], s["hkv"], HD, 64, s["splits"],
                             part_o=s["part_o"], part_ml=s["part_ml"], status=s["status"], out=s["out"])
    if f == "attn_prefill":
        s = state
        return A.attn_prefill(s["q"], s["kv"], s["table"], 0, s["pos0"], s["hq"], s["hkv"], HD, status=s["status"])
    if f == "sample":
        return basic.sample_rows(**state["args"])
    m = state["model"]
    if f == "model_step":
        out, logits = m.forward_rows(state["ids"], state["seqs"], want_logits=True)
        for s, n in enumerate(state["lens"]):
            m.truncate(s, n)                 # every draft rejected: the rows are rolled back
        return out, logits
    tok, logits = m.prefill(0, state["prompt"], want_logits=True)
    m.truncate(0, 0)
    return logits


# ------------------------------------------------------------------------------------------------- least work of a pass
def _wbytes(n, k, bits, group):
    return n * k * bits / 8 + n * (k / group) * 4


def work(case):
    f = case["family"]
    if f == "layers":
        m = case["rows"]
        b = fl = 0.0
        for lin in LINEARS:
            n, k = _shape(case["dims"], lin)
            b += _wbytes(n, k, _bits(case, lin), case["group"]) + 2 * m * (k + n)
            fl += 2.0 * m * n * k
        return {"bytes": b * case["layers"], "flops": fl * case["layers"]}
    if f == "linear":
        n, k = _shape(case["dims"], case["linear"])
        return {"bytes": _wbytes(n, k, case["bits"], case["group"]) + 2.0 * case["rows"] * (n + k), "flops": 2.0 * case["rows"] * n * k}
    if f == "attn_decode":
        d, hq, hkv, ffn = DIMS[case["dims"]]
        keys = case["ctx"] * (1 if case["seqs"] == 1 else 2.0 / 3 * case["seqs"])
        return {"bytes": keys * hkv * HD * 4 + 4.0 * case["seqs"] * case["rows"] * hq * HD, "flops": 4.0 * keys * case["rows"] * hq * HD}
    if f == "attn_prefill":
        d, hq, hkv, ffn = DIMS[case["dims"]]
        t = case["rows"]
        pairs = t * case["pos0"] + t * (t + 1) / 2
        return {"bytes": (case["pos0"] + t) * hkv * HD * 4 + 4.0 * t * hq * HD, "flops": 4.0 * pairs * hq * HD}
    if f == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 4.0 * case["rows"] * case["vocab"]}
    cfg = C.scaled(C.dense_32b(seed=0), case["layers"])
    wb = lin_w = 0.0
    for l in range(cfg.n_layers):
        for lin in LINEARS:
            n, k = _shape("dense", lin)
            wb += _wbytes(n, k, cfg.bits_of(l, lin), cfg.group)
            lin_w += n * k
    head = _wbytes(cfg.vocab, cfg.d_model, cfg.lm_head_bits, cfg.group)
    attn = lambda q, ctx: cfg.n_layers * 4.0 * q * ctx * cfg.n_heads * HD
    if case["family"] == "model_step":
        rows = case["seqs"] * case["rows"]
        kv = cfg.n_layers * case["seqs"] * case["ctx"] * cfg.n_kv_heads * HD * 4.0
        return {"bytes": wb + head + kv + rows * cfg.vocab * 4.0, "flops": 2.0 * rows * (lin_w + cfg.vocab * cfg.d_model) + attn(rows, case["ctx"])}
    t = case["tokens"]
    return {"bytes": wb + head + t * cfg.d_model * 2.0 + cfg.vocab * 4.0,
            "flops": 2.0 * t * lin_w + 2.0 * cfg.vocab * cfg.d_model + attn(t, t / 2)}


def tolerance(case):
    # about four times the distance from the 64-bit results that bf16 results and bf16 operands between kernels show
    # (2e-3 for one product, 6e-3 where layers follow one another, 4e-3 for the logits)
    return {"layers": {"rel": 2e-2}, "linear": {"rel": 1e-2}, "attn_decode": {"rel": 1e-2}, "attn_prefill": {"rel": 1e-2},
            # masses and counts are whole numbers and the draw depends on the seed and the position alone
            "sample": "exact",
            # chosen tokens may change where two logits are close; the logits themselves are compared
            "model_step": {"rel": 1.5e-2, "differ": 0.3}, "model_prefill": {"rel": 1.5e-2}}[case["family"]]


# ------------------------------------------------------------------------------------------------------ 64-bit results
def _weights64(seed, n, k, bits, group):
    """Row blocks of the 64-bit weights of `_weights(seed, ...)`: yields (first row, float64 [rows, k])."""
    packed, scale, zero = _weights(seed, n, k, bits, group)
    step = max(32, ((16 << 20) // k) // 32 * 32)
    for r0 in range(0, n, step):
        p = packed[r0:r0 + step].to(torch.int64) & 0xFFFFFFFF
        rows = p.shape[0]
        p = p.view(rows, k // 32, bits)
        c = torch.empty(rows, k // 32, 32, dtype=torch.int64, device=DEV)
        for i in range(32):
            w, s = divmod(i * bits, 32)
            v = p[..., w] >> s
            if s + bits > 32:
                v = v | (p[..., w + 1] << (32 - s))
            c[..., i] = v & ((1 << bits) - 1)
        c = c.view(rows, k // group, group).double()
        yield r0, ((c - zero[r0:r0 + step].double().unsqueeze(-1)) * scale[r0:r0 + step].double().unsqueeze(-1)).view(rows, k)


def _mul64(x, seed, n, k, bits, group):
    y = torch.empty(x.shape[0], n, dtype=torch.float64, device=DEV)
    for r0, w in _weights64(seed, n, k, bits, group):
        y[:, r0:r0 + w.shape[0]] = x @ w.t()
    return y


def _rms64(h, w):
    return h * torch.rsqrt((h * h).mean(-1, keepdim=True) + EPS) * w.double()


def _swiglu64(gu):
    v = gu.view(gu.shape[0], -1, 2, 8)                       # blocks of eight gate rows and their eight up rows
    return (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(gu.shape[0], -1)


def _attend64(q, kk, vv, pos):
    """q [T, hq, 128], kk / vv [S, hkv, 128], pos [T]: causal softmax attention in 64 bits."""
    hq, hkv = q.shape[1], kk.shape[1]
    out = torch.empty_like(q)
    keys = torch.arange(kk.shape[0], device=DEV)
    for h in range(hkv):
        qs = q[:, h * (hq // hkv):(h + 1) * (hq // hkv)]
        for t0 in range(0, q.shape[0], 256):
            s = torch.einsum("tgd,sd->gts", qs[t0:t0 + 256], kk[:, h]) / math.sqrt(HD)
            s = s.masked_fill(keys[None, None, :] > pos[t0:t0 + 256][None, :, None], -math.inf)
            out[t0:t0 + 256, h * (hq // hkv):(h + 1) * (hq // hkv)] = torch.einsum("gts,sd->tgd", torch.softmax(s, -1), vv[:, h])
    return out


def _rope64(x, pos, theta):
    half = HD // 2
    inv = theta ** (-2.0 * torch.arange(half, dtype=torch.float64, device=DEV) / HD)
    ang = pos.double()[:, None] * inv[None]
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _model64(case, seed, prompts):
    """64-bit logits of every row of every prompt that `keep` rows long ends it: [(ids, keep)] -> list of [keep, vocab]."""
    cfg, norms, final, embed = _model_parts(case, seed)
    hs = [embed[ids.to(DEV)].double() for ids, _ in prompts]
    for l in range(cfg.n_layers):
        def mul(x, lin, i):
            n, k = _shape("dense", lin)
            return _mul64(x, _model_seed(seed, l, i), n, k, cfg.bits_of(l, lin), cfg.group)
        cut = [h.shape[0] for h in hs]
        h = torch.cat(hs)
        qkv = mul(_rms64(h, norms[l][0]), "qkv", 0)
        att = []
        for x in qkv.split(cut):
            pos = torch.arange(x.shape[0], device=DEV)
            q = _rope64(x[:, :cfg.q_dim].view(-1, cfg.n_heads, HD), pos, cfg.rope_theta)
            kk = _rope64(x[:, cfg.q_dim:cfg.q_dim + cfg.kv_dim].view(-1, cfg.n_kv_heads, HD), pos, cfg.rope_theta)
            vv = x[:, cfg.q_dim + cfg.kv_dim:].view(-1, cfg.n_kv_heads, HD)
            att.append(_attend64(q, kk, vv, pos).view(x.shape[0], -1))
        h = h + mul(torch.cat(att), "o", 1)
        act = _swiglu64(mul(_rms64(h, norms[l][1]), "gate_up", 2))
        h = h + mul(act, "down", 3)
        hs = list(h.split(cut))
    last = torch.cat([h[-keep:] for h, (_, keep) in zip(hs, prompts)])
    return _mul64(_rms64(last, final), _model_seed(seed, 999, 7), cfg.vocab, cfg.d_model, cfg.lm_head_bits, cfg.group)


def exact(case, seed):
    f = case["family"]
    if f == "layers":
        x, per = _layers_inputs(case, seed)
        x = x.double()
        outs = []
        for l, p in enumerate(per):
            def mul(v, lin, i):
                n, k = _shape(case["dims"], lin)
                return _mul64(v, seed * 1000 + l * 8 + i + 1, n, k, _bits(case, lin), case["group"])
            qkv = mul(_rms64(x, p["ln1"]), "qkv", 0)
            h1 = x + mul(p["attn"].double(), "o", 1)
            act = _swiglu64(mul(_rms64(h1, p["ln2"]), "gate_up", 2))
            x = h1 + mul(act, "down", 3)
            outs += [qkv, h1, act, x]
        return outs
    if f == "linear":
        n, k = _shape(case["dims"], case["linear"])
        return _mul64(_linear_inputs(case, seed).double(), seed * 1000 + 1, n, k, case["bits"], case["group"])
    if f in ("attn_decode", "attn_prefill"):
        d, hq, hkv, ffn = DIMS[case["dims"]]
        ctx, rows, kv, table, q = _attn_inputs(case, seed)
        outs = []
        for s, c in enumerate(ctx):
            pages = table[s, :(c + 15) // 16].long()
            k2 = kv[pages].double().permute(1, 0, 3, 2, 4).reshape(2, -1, hkv, HD)[:, :c]
            pos = torch.arange(c - rows, c, device=DEV)
            outs.append(_attend64(q[s * rows:(s + 1) * rows].double().view(rows, hq, HD), k2[0], k2[1], pos).view(rows, -1))
        return torch.cat(outs)
    if f == "sample":
        return None
    if f == "model_step":
        rows = case["rows"]
        ids = _prompt(seed, case["seqs"] * rows, 99)
        prompts = [(torch.cat([_prompt(seed, case["ctx"] + 3 * s, s), ids[s * rows:(s + 1) * rows]]), rows) for s in range(case["seqs"])]
        return None, _model64(case, seed, prompts)
    return _model64(case, seed, [(_prompt(seed, case["tokens"], 0), 1)])[0]
