"""The work this library is used for, as cases that can be timed and compared: training layers, forward scoring, streaming
decode, the lm_head loss, slot lists and the query side, over the sizes a user meets.

A case is a dict with a "kind" and its sizes.  prepare(case, seed) makes what a program holds before the call, run(state)
is one pass through the public operators.
"""
import math

import numpy as np
import torch

import mathbrain_b200 as mb
from mathbrain_b200.decode import DecodeState
from mathbrain_b200.feeder import ChunkFeeder
from mathbrain_b200.lmhead import lm_head_cross_entropy

HD = 64                     # head width of every configuration of the model
VOCAB = 50257


def listed():
    return [
        # the 46M model's training step, two of its six layers: 56 chunks of 512 steps, prefixes to 8192 tokens, bf16
        dict(name="train 46M", kind="train", B=56, T=512, N=64, H=8, V=VOCAB, prefix=8192, min_fill=64, bursty=False,
             bf16=True, rows=False, skip_pad=False, layers=2),
        # long chunks with bursty repeats, 128 channels: one layer forward and backward
        dict(name="train long chunks", kind="train", B=8, T=4096, N=128, H=8, V=VOCAB, prefix=2048, min_fill=4096, bursty=True,
             bf16=True, rows=False, skip_pad=False, layers=1),
        # a small training batch of ragged chunks as hosted.train_step_loss runs a layer: K/V rows projected once per
        # distinct token, padded steps skipped
        dict(name="train ragged rows", kind="train", B=6, T=300, N=64, H=8, V=VOCAB, prefix=3000, min_fill=20, bursty=False,
             bf16=True, rows=True, skip_pad=True, layers=2),
        # the configuration the model's CPU path is checked on, in the exact fp32 mode, forward and backward
        dict(name="train exact fp32", kind="train", B=2, T=128, N=64, H=8, V=VOCAB, prefix=0, min_fill=128, bursty=False,
             bf16=False, rows=False, skip_pad=False, layers=1, mode="fp32"),
        # evaluation of a batch of documents: forward only, fp32 activations
        dict(name="score batch", kind="score", B=16, T=512, N=64, H=8, V=VOCAB, prefix=4096, min_fill=100, bursty=False,
             bf16=False, layers=2),
        # one short text scored alone (an interactive prompt): every launch and host step shows
        dict(name="score one prompt", kind="score", B=1, T=77, N=64, H=8, V=VOCAB, prefix=0, min_fill=77, bursty=False,
             bf16=True, layers=6),
        # serving: 64 sequences, 6 layers, about 3400 slots seen, one graph replay a token
        dict(name="decode 64 sequences", kind="decode", B=64, K=3400, N=64, H=8, V=VOCAB, layers=6, graph=True, bf16=True),
        # one interactive sequence, launched step by step
        dict(name="decode one sequence", kind="decode", B=1, K=700, N=64, H=8, V=VOCAB, layers=6, graph=False, bf16=True),
        # the tied lm_head and its masked loss over a training batch, forward and backward
        dict(name="lm_head loss", kind="loss", R=28672, D=512, V=VOCAB, valid=0.53, bf16=True),
        # the next chunk of 56 documents in flight: slot lists, chunk-start states, scan, advance
        dict(name="feed 56 documents", kind="feed", B=56, T=512, N=64, V=VOCAB, history=6, min_fill=64),
        # the query side of one layer alone: scan, gate and LayerNorm, forward and backward, ragged
        dict(name="query side", kind="query", B=9, T=777, N=64, D=512, V=VOCAB, prefix=1000, min_fill=300, bf16=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "score", "score", "decode", "decode", "loss", "feed", "query"])
    H = rng.choice([4, 8, 8])
    N = rng.choice([64, 64, 128])
    V = rng.choice([VOCAB, VOCAB, 32000])
    if kind == "train":
        if rng.random() < 0.25:         # exact mode, small, any channel count
            T = _log(rng, 30, 300)
            return dict(kind="train", B=rng.randint(1, 3), T=T, N=rng.choice([32, 64, 96, 128]), H=rng.choice([2, 4, 8]), V=V,
                        prefix=rng.choice([0, 200]), min_fill=max(1, T // 2), bursty=False, bf16=rng.random() < 0.5, rows=False,
                        skip_pad=False, layers=1, mode="fp32")
        T = _log(rng, 64, 4096)
        B = max(1, min(56, _log(rng, 1, 28672 // T)))
        rows = rng.random() < 0.4
        return dict(kind="train", B=B, T=T, N=N, H=H, V=V, prefix=_log(rng, 64, 8192 if T <= 512 else 2048),
                    min_fill=_log(rng, 16, T) if rng.random() < 0.6 else T, bursty=rng.random() < 0.3, bf16=rng.random() < 0.8,
                    rows=rows, skip_pad=rows or rng.random() < 0.3, layers=1)
    if kind == "score":
        T = _log(rng, 20, 2048)
        return dict(kind="score", B=max(1, min(32, _log(rng, 1, max(1, 8192 // T)))), T=T, N=N, H=H, V=V, prefix=_log(rng, 16, 4096),
                    min_fill=max(1, T // 3), bursty=rng.random() < 0.3, bf16=rng.random() < 0.6, layers=rng.choice([1, 2, 6]))
    if kind == "decode":
        return dict(kind="decode", B=_log(rng, 1, 64), K=_log(rng, 150, 4000), N=64, H=H, V=V, layers=rng.choice([2, 6]),
                    graph=rng.random() < 0.5, bf16=True)
    if kind == "loss":
        return dict(kind="loss", R=_log(rng, 300, 28672), D=rng.choice([256, 512]), V=V, valid=round(rng.uniform(0.3, 1.0), 3),
                    bf16=rng.random() < 0.9)
    if kind == "feed":
        T = _log(rng, 64, 1024)
        return dict(kind="feed", B=_log(rng, 2, 56), T=T, N=N, V=V, history=rng.randint(1, 8), min_fill=max(2, T // 4))
    T = _log(rng, 64, 4096)
    return dict(kind="query", B=max(1, min(56, _log(rng, 1, 28672 // T))), T=T, N=N, D=64 * H, V=V, prefix=_log(rng, 16, 4096),
                min_fill=max(1, T // 3), bf16=rng.random() < 0.7)


# ------------------------------------------------------------------------------------------------ inputs
def _distinct(V, n):
    """Distinct tokens expected among n Zipf(1.1) draws."""
    p = np.arange(1, V + 1, dtype=np.float64) ** -1.1
    return float((1.0 - np.exp(n * np.log1p(-p / p.sum()))).sum())


def _width(V, n):
    """Columns of the slot lists of documents of up to n tokens: what n draws give, and some to spare."""
    return max(16, min(n, V, int(1.1 * _distinct(V, n)) + 64))


def _rhos(N):
    h = torch.logspace(math.log10(1024.0), math.log10(4096.0), N)          # half-lives of the model's default configuration
    return torch.exp(-math.log(2.0) / h)


def _zipf(rng, V, n):
    p = np.arange(1, V + 1, dtype=np.float64) ** -1.1
    cdf = np.cumsum(p / p.sum())
    return np.minimum(np.searchsorted(cdf, rng.random(n)), V - 1).astype(np.int64)


def _tokens(rng, V, n, bursty):
    tok = _zipf(rng, V, n)
    if bursty:              # with probability 0.2 a token of the last 64 positions comes again
        src = np.arange(n)
        src = np.where(rng.random(n) < 0.2, np.maximum(src - rng.integers(1, 65, n), 0), src)
        while True:
            nxt = src[src]
            if np.array_equal(nxt, src):
                break
            src = nxt
        tok = tok[src]
    return tok


def _chunks(seed, B, T, N, V, prefix, min_fill, bursty=False, **_):
    """A batch of single-document chunks as the model's loader hands them over: the chunk's sorted distinct tokens first,
    then those of the document's prefix alone, each with its state at the chunk's first step, in lists of one width for all
    batches of a configuration (static shapes)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    rhos = _rhos(N)
    decay = rhos.double().numpy()[None, :] ** np.arange(prefix + 1, dtype=np.float64)[:, None]
    K = _width(V, prefix + T)
    xs, keys, states, fills = [], [], [], []
    for _ in range(B):
        P = int(rng.integers(0, prefix + 1))
        fill = int(rng.integers(min(min_fill, T), T + 1))
        doc = _tokens(rng, V, P + fill, bursty)
        pre, chunk = doc[:P], doc[P:]
        cu = np.unique(chunk)
        own = np.concatenate([cu, np.setdiff1d(pre, cu)])[:K]
        st = np.zeros((len(own), N), np.float32)
        if P:
            order = np.argsort(pre, kind="stable")
            tok = pre[order]
            first = np.flatnonzero(np.concatenate([[True], tok[1:] != tok[:-1]]))
            sums = np.add.reduceat(decay[P - order], first, axis=0)
            at = np.full(V, -1)
            at[own] = np.arange(len(own))
            at = at[tok[first]]
            st[at[at >= 0]] = sums[at >= 0]
        xs.append(np.concatenate([chunk, np.zeros(T - fill, np.int64)]))
        keys.append(own)
        states.append(st)
        fills.append(fill)
    unique = np.zeros((B, K), np.int64)
    mask = np.zeros((B, K), bool)
    c_base = np.zeros((B, K, N), np.float32)
    for b in range(B):
        k = len(keys[b])
        unique[b, :k], mask[b, :k], c_base[b, :k] = keys[b], True, states[b]
    d = dict(x=np.stack(xs), unique=unique, mask=mask, c_base=c_base, fill=np.array(fills, np.int32))
    return {k: torch.from_numpy(v).cuda() for k, v in d.items()}, rhos.cuda()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=0.02, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _linear(g, n_in, n_out):
    m = torch.nn.Linear(n_in, n_out, bias=False, device="cuda")
    with torch.no_grad():
        m.weight.copy_(_randn(g, n_out, n_in))              # the model's initialisation
    return m


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


def _prepare_layers(case, seed):
    c = case
    batch, rhos = _chunks(seed, **{k: v for k, v in c.items() if k not in ("name", "kind")})
    g = _gen(seed)
    D, N, train = HD * c["H"], c["N"], c["kind"] == "train"
    dt = torch.bfloat16 if c["bf16"] else torch.float32
    K = batch["unique"].shape[1]
    layers = []
    for _ in range(c["layers"]):
        lay = dict(pe=_linear(g, N, D), ln=torch.nn.LayerNorm(D, device="cuda"), qp=_linear(g, D, D),
                   x_q=_randn(g, c["B"], c["T"], D, std=1.0))
        if c.get("rows"):
            lay.update(ln_kv=torch.nn.LayerNorm(D, device="cuda"), kp=_linear(g, D, D), vp=_linear(g, D, D))
        else:
            lay.update(E_k=_randn(g, c["B"], K, D, dtype=dt), E_v=_randn(g, c["B"], K, D, dtype=dt))
        if train:
            lay["dO"] = _randn(g, c["B"], c["H"], c["T"], HD)
            for k in ("x_q", "E_k", "E_v"):
                if k in lay:
                    lay[k].requires_grad_(True)
        layers.append(lay)
    E = _randn(g, c["V"], D).requires_grad_(True) if c.get("rows") else None
    return dict(case=c, batch=batch, rhos=rhos, layers=layers, E=E)


def _layers(s, train):
    """Scan, snapshots and the layers' gate and attention, the calls of the model's forward, and each layer's backward."""
    c, b, rhos = s["case"], s["batch"], s["rhos"]
    B, T, H, D = c["B"], c["T"], c["H"], HD * c["H"]
    out = []
    with mb.options(mode=c.get("mode", "auto")), torch.set_grad_enabled(train):
        C_seq = mb.compute_query_ema_history(b["x"], rhos, c["V"], b["c_base"], b["unique"])
        slots = b["unique"].clone()
        slots[~b["mask"]] = -1
        K = slots.shape[1]
        states = mb.precompute_boundaries(b["x"], slots, rhos, 64, c_init=b["c_base"],
                                          seq_lens=b["fill"] if c.get("skip_pad") else None)
        out.append(C_seq)
        if c.get("rows"):
            tokens, row_index = mb.shared_slot_rows(slots)
            s["E"].grad = None
        for lay in s["layers"]:
            leaves = [lay[k] for k in ("x_q", "E_k", "E_v") if k in lay]
            leaves += [p for k in ("pe", "ln", "qp", "ln_kv", "kp", "vp") if k in lay for p in lay[k].parameters()]
            for p in leaves:
                p.grad = None
            with torch.autocast("cuda", dtype=torch.bfloat16, enabled=c["bf16"]):
                Q = mb.fused_apply_symmetric_query_gating(lay["x_q"], C_seq, lay["pe"], lay["ln"], lay["qp"], True)
                Q = Q.view(B, T, H, HD).transpose(1, 2).contiguous()
                W = lay["pe"].weight.t().contiguous()
                if c.get("rows"):
                    Ek, Ev = mb.project_slot_rows(s["E"], tokens, lay["ln_kv"], lay["kp"], lay["vp"])
                    O = mb.FlashEMARowsFunction.apply(Q, b["x"], Ek, Ev, row_index, W, rhos, c["V"], slots, K, states, True)
                else:
                    O = mb.FlashEMAFunction.apply(Q, b["x"], lay["E_k"], lay["E_v"], W, rhos, c["V"], slots, K, states, True)
            out.append(O.detach())
            if train:
                O.backward(lay["dO"])
                out += [p.grad for p in leaves]
        if c.get("rows"):
            out.append(s["E"].grad)
    return out


def _prepare_decode(case, seed):
    c = case
    g = _gen(seed)
    B, V, N, K, D, t0 = c["B"], c["V"], c["N"], c["K"], HD * c["H"], 8192
    st = DecodeState(B, V, _rhos(N).cuda(), capacity=K + 512)
    for b in range(B):                      # K distinct slots seen by each sequence at earlier steps
        seen = torch.randperm(V, generator=g, device="cuda")[:K]
        st.active[b, :K] = seen.int()
        st.last_t[b, seen] = torch.randint(0, t0, (K,), generator=g, device="cuda").int()
        st.state[b, seen] = torch.rand(K, N, generator=g, device="cuda") * 3 + 1
    st.n_active.fill_(K)
    dt = torch.bfloat16 if c["bf16"] else torch.float32
    lay = [dict(q=_randn(g, B, c["H"], HD, dtype=dt, std=0.45), E_k=_randn(g, V, D, dtype=dt), E_v=_randn(g, V, D, dtype=dt),
                W=_randn(g, N, D)) for _ in range(c["layers"])]
    tok = torch.from_numpy(_zipf(np.random.Generator(np.random.PCG64(seed)), V, B)).cuda()
    s = dict(case=c, st=st, layers=lay, tok=tok, t=t0)
    if c["graph"]:
        st.use_device_step(t0)
        s["static"] = tok.clone()
        s["graph"], s["outs"], s["C_q"] = st.capture_step([x["q"] for x in lay], [x["E_k"] for x in lay], [x["E_v"] for x in lay],
                                                         [x["W"] for x in lay], s["static"])
    return s


def _run_decode(s):
    st = s["st"]
    if s["case"]["graph"]:
        s["static"].copy_(s["tok"])
        s["graph"].replay()
        outs, C_q = s["outs"], s["C_q"]
    else:
        outs = [st.attend(x["q"], x["E_k"], x["E_v"], x["W"], s["t"]) for x in s["layers"]]
        C_q = st.update(s["tok"], s["t"])
        s["t"] += 1
    return list(outs) + [C_q, st.state, st.last_t, st.active, st.n_active]


def _prepare_loss(case, seed):
    c = case
    g = _gen(seed)
    dt = torch.bfloat16 if c["bf16"] else torch.float32
    y = torch.randint(0, c["V"], (c["R"],), generator=g, device="cuda")
    y[torch.rand(c["R"], generator=g, device="cuda") >= c["valid"]] = -1
    return dict(case=c, h=_randn(g, c["R"], c["D"], std=1.0, dtype=dt).requires_grad_(True), y=y,
                E=_randn(g, c["V"], c["D"]).requires_grad_(True))


def _run_loss(s):
    s["h"].grad = s["E"].grad = None
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=s["case"]["bf16"]):
        loss = lm_head_cross_entropy(s["h"], s["E"], s["y"], ignore_index=-1)
    loss.backward()
    return [loss.detach(), s["h"].grad, s["E"].grad]


def _prepare_feed(case, seed):
    c = case
    rng = np.random.Generator(np.random.PCG64(seed))
    B, T = c["B"], c["T"]
    rhos = _rhos(c["N"]).cuda()
    feeder = ChunkFeeder(B, c["V"], rhos, capacity=8192)
    n = (c["history"] + 1) * T
    docs = _zipf(rng, c["V"], B * n).reshape(B, n)
    # the first document has the most distinct tokens, as many as the widest list of such documents holds
    own = rng.permutation(c["V"])[:_width(c["V"], n)]
    docs[0] = rng.permutation(np.concatenate([own, rng.choice(own, n - len(own))]))
    full = torch.full((B,), T, dtype=torch.int32, device="cuda")
    for i in range(c["history"]):           # the documents' earlier chunks
        x = torch.from_numpy(docs[:, i * T:(i + 1) * T].copy()).cuda()
        batch = feeder.next_batch(x, full)
        feeder.advance(x, full, mb.compute_query_ema_history(x, rhos, c["V"], batch["c_base"], batch["unique_slots"]))
    fill = rng.integers(c["min_fill"], T + 1, B).astype(np.int32)
    fill[0] = T
    x = docs[:, -T:].copy()
    x[np.arange(T)[None, :] >= fill[:, None]] = 0
    return dict(case=c, feeder=feeder, rhos=rhos, x=torch.from_numpy(x).cuda(), fill=torch.from_numpy(fill).cuda())


def _run_feed(s):
    f = s["feeder"]
    batch = f.next_batch(s["x"], s["fill"])
    C_seq = mb.compute_query_ema_history(s["x"], s["rhos"], s["case"]["V"], batch["c_base"], batch["unique_slots"])
    f.advance(s["x"], s["fill"], C_seq)
    return [batch["unique_slots"], batch["pad_mask"], batch["c_base"], C_seq, f.state, f.last_t, f.seen, f.n_seen, f.t0]


def _prepare_query(case, seed):
    c = case
    batch, rhos = _chunks(seed, c["B"], c["T"], c["N"], c["V"], c["prefix"], c["min_fill"])
    g = _gen(seed)
    D = c["D"]
    return dict(case=c, batch=batch, rhos=rhos, pe=_linear(g, c["N"], D), ln=torch.nn.LayerNorm(D, device="cuda"), qp=_linear(g, D, D),
                x_q=_randn(g, c["B"], c["T"], D, std=1.0).requires_grad_(True),
                dQ=_randn(g, c["B"], c["T"], D, dtype=torch.bfloat16 if c["bf16"] else torch.float32))


def _run_query(s):
    c, b = s["case"], s["batch"]
    leaves = [s["x_q"]] + [p for k in ("pe", "ln", "qp") for p in s[k].parameters()]
    for p in leaves:
        p.grad = None
    C_seq = mb.compute_query_ema_history(b["x"], s["rhos"], c["V"], b["c_base"], b["unique"])
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=c["bf16"]):
        Q = mb.fused_apply_symmetric_query_gating(s["x_q"], C_seq, s["pe"], s["ln"], s["qp"], True)
    Q.backward(s["dQ"])
    return [C_seq, Q.detach()] + [p.grad for p in leaves]


_PREPARE = dict(train=_prepare_layers, score=_prepare_layers, decode=_prepare_decode, loss=_prepare_loss, feed=_prepare_feed,
                query=_prepare_query)
_RUN = dict(train=lambda s: _layers(s, True), score=lambda s: _layers(s, False), decode=_run_decode, loss=_run_loss,
            feed=_run_feed, query=_run_query)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _slots(c):
    """About how many distinct tokens a sample lists."""
    n = c.get("prefix", 0) / 2 + (c.get("min_fill", c["T"]) + c["T"]) / 2
    return _distinct(c["V"], n + c.get("history", 0) * c["T"])


def work(case):
    c, k = case, case["kind"]
    if k in ("train", "score"):
        B, T, N, D, L = c["B"], c["T"], c["N"], HD * c["H"], c["layers"]
        e = 2 if c["bf16"] else 4
        K = _slots(c)
        steps = (c["min_fill"] + T) / 2 if c.get("skip_pad") else T
        slot_rows = B * K if not c.get("rows") else min(B * K, c["V"])
        table = slot_rows * D * (4 if c.get("rows") else 2 * e)
        # tokens, slot keys and states in, query states out; then x_q, E rows in and O out of every layer
        nbytes = B * T * (8 + 4 * N) + B * K * (8 + 4 * N) + L * (B * T * D * 8 + table)
        # the products of a step with a slot: score and value (2 x 2 D); their four gradients
        flops = L * (4 * D * B * steps * K + 2 * B * T * D * (N + D))
        if k == "train":                    # dO in; the gradients of x_q and of the E rows out
            nbytes += L * (B * T * D * 8 + table)
            flops *= 3
        return dict(bytes=nbytes, flops=flops)
    if k == "decode":                       # a sequence's state rows once, each layer's distinct E rows once, queries and outputs
        B, D, L = c["B"], HD * c["H"], c["layers"]
        rows = c["V"] * (1.0 - (1.0 - c["K"] / c["V"]) ** B)
        return dict(bytes=B * c["K"] * (4 * c["N"] + 8) + L * (rows * D * 4 + B * D * 6),
                    flops=L * B * c["K"] * D * (2 * c["N"] + 4))
    if k == "loss":                         # three products over the valid rows
        n = c["R"] * c["valid"]
        return dict(bytes=2 * c["R"] * c["D"] * (2 if c["bf16"] else 4) + 8 * c["V"] * c["D"], flops=6 * n * c["V"] * c["D"])
    if k == "feed":                         # tokens in; lists, masks and states out; the touched states in and out
        B, T, N, K = c["B"], c["T"], c["N"], _slots(c)
        return dict(bytes=B * (T * (16 + 4 * N) + K * (8 + 1 + 8 * N) + T * 4 * N), flops=B * (K + T) * N)
    B, T, N, D = c["B"], c["T"], c["N"], c["D"]
    return dict(bytes=B * T * (8 + 8 * N + D * (4 + 2 + 2 + 4)) + B * _slots(c) * (8 + 4 * N), flops=6 * B * T * D * (N + D))


def tolerance(case):
    k = case["kind"]
    if k == "feed":
        return {"rel": 1e-5}                # fp32 states; the lists are whole numbers
    if k in ("train", "score") and case.get("mode") == "fp32" and not case["bf16"]:
        return {"rel": 1e-4}
    return {"rel": 1e-2}                    # 16-bit operands of the gate, score and gradient products
