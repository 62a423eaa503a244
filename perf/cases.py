"""The work a user has this framework do, as cases that can be timed and compared: single projections, whole-token decoding and
prompts of the quantized engine, prompts and token-by-token runs of models described block by block.

Weights are random codes in the file formats (kronos_2t_b200.synth); models that are deep are cut to a few of their layers, which are
alike, so that a state is made quickly.  All sizes are those of the shapes in synth.py and of the tests and benchmark, or lie between them.

Kinds
  linear   rotate + quantize + multiply for a list of matrices, on device buffers (optionally as one captured graph, as a decode
           loop holds them) or on pinned host buffers (queued, one wait per pass)
  decode   engine.decode_greedy: `steps` tokens from position `ctx` of a filled cache; tokens and the last logits
  prompt   engine.forward_token_ids: `n` tokens from position `past`; the last logits
  blocks   block engine: `n` tokens as a prompt, then `steps` given tokens one by one (a host that samples); all these logits.
           past > 0: the sequence starts behind `past` cached positions (latent attention only: it can be continued anywhere)
"""
import math

import numpy as np
import torch

import kronos_2t_b200 as k2
from kronos_2t_b200 import synth

SWEEP = "2048x2048,2048x8192,8192x2048,2048x49152"          # cols x rows
MODELS = {
    "smollm2_135m": dict(cfg=synth.SMOLLM2_135M, mode="b4"),
    "smollm2_1p7b": dict(cfg=synth.SMOLLM2_1_7B, mode="nf4g128"),
    "qwen2_7b": dict(cfg=synth.QWEN2_7B, mode="b4", modes=synth.P55454, qkv_bias=True, untied=True),
    "qwen3_30b_a3b": dict(cfg=synth.QWEN3_30B_A3B, mode="nf4g128", moe=dict(n_experts=128, top_k=8, d_ff=768, bits=3, sgc=2)),
}


def listed():
    return [
        # one small projection by itself (the qkv product of the 135M shape): launches and latency
        dict(name="linear_small", kind="linear", sizes="576x960", modes="b4", n_tok=1, where="device", graph=False),
        # the benchmark's sweep: 16 matrices of four formats, one token, resident activations
        dict(name="sweep_device", kind="linear", sizes=SWEEP, modes="b4,b5,b6,nf4g128", n_tok=1, where="device", graph=True),
        # the same from and to host memory: a host engine that hands its projections over
        dict(name="sweep_host", kind="linear", sizes=SWEEP, modes="b4,b5,b6,nf4g128", n_tok=1, where="host", graph=False),
        # chat on the small model, short context
        dict(name="decode_135m", kind="decode", model="smollm2_135m", layers=30, kv_bits=8, window=0, ctx=128, steps=32),
        # generating behind a long document
        dict(name="decode_1p7b_long", kind="decode", model="smollm2_1p7b", layers=12, kv_bits=8, window=0, ctx=4000, steps=16),
        # sparse experts, short context
        dict(name="decode_moe", kind="decode", model="qwen3_30b_a3b", layers=3, kv_bits=8, window=0, ctx=300, steps=32),
        # a page of text as the prompt
        dict(name="prompt_1p7b", kind="prompt", model="smollm2_1p7b", layers=12, kv_bits=8, past=0, n=1000),
        # a short question of odd length, large model with mixed bit planes, grouped heads
        dict(name="prompt_7b_short", kind="prompt", model="qwen2_7b", layers=4, kv_bits=8, past=0, n=77),
        # prompt through the experts
        dict(name="prompt_moe", kind="prompt", model="qwen3_30b_a3b", layers=3, kv_bits=8, past=0, n=300),
        # prompts of the block models, bf16
        dict(name="prompt_folizen", kind="blocks", design="folizen", shape="medium", layers=12, past=0, n=2048, steps=0),
        dict(name="prompt_zasesun", kind="blocks", design="zasesun", shape="medium", layers=4, past=0, n=2048, steps=0),
        # a short prompt and its answer token by token
        dict(name="answer_folizen", kind="blocks", design="folizen", shape="medium", layers=12, past=0, n=100, steps=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "decode", "decode", "prompt", "prompt", "prompt", "blocks", "blocks"])
    if kind == "linear":
        cols, mode = 64 * _log(rng, 3, 128), rng.choice(["b4", "b5", "b6", "nf4g128", "nf4"])
        rows = _log(rng, 64, 49152 if cols <= 2048 else 8192)
        if mode.startswith("nf"):
            rows = max(32, rows // 32 * 32)
        where = rng.choice(["device", "device", "host"])
        return dict(kind=kind, sizes=f"{cols}x{rows}", modes=mode, n_tok=rng.choice([1, 1, 2, 3, _log(rng, 4, 200)]), where=where,
                    graph=where == "device" and rng.random() < 0.5)
    if kind in ("decode", "prompt"):
        model = rng.choice(list(MODELS))
        layers = {"smollm2_135m": 30, "smollm2_1p7b": rng.randint(4, 12), "qwen2_7b": rng.randint(2, 4), "qwen3_30b_a3b": rng.randint(2, 3)}[model]
        longest = {"smollm2_135m": 440, "smollm2_1p7b": 4000, "qwen2_7b": 2000, "qwen3_30b_a3b": 1000}[model]
        kv_bits = rng.choice([8, 8, 8, 4])
        if kind == "decode":
            ctx = _log(rng, 16, longest)
            return dict(kind=kind, model=model, layers=layers, kv_bits=kv_bits, window=256 if model != "smollm2_135m" and rng.random() < 0.15 else 0,
                        ctx=ctx, steps=rng.randint(4, 16))
        n = _log(rng, 2, min(longest, 1000))
        past = _log(rng, 1, longest - n) if rng.random() < 0.3 and longest - n > 1 else 0
        return dict(kind=kind, model=model, layers=layers, kv_bits=kv_bits, past=past, n=n)
    design = rng.choice(["folizen", "zasesun"])
    shape = rng.choice(["small", "medium"])
    layers = rng.randint(2, 12) if design == "folizen" else rng.randint(2, 4)
    if rng.random() < 0.6:
        return dict(kind=kind, design=design, shape=shape, layers=layers, past=0, n=_log(rng, 2, 2048), steps=0)
    if design == "zasesun":
        return dict(kind=kind, design=design, shape=shape, layers=layers, past=_log(rng, 16, 4000), n=0, steps=rng.randint(4, 24))
    return dict(kind=kind, design=design, shape=shape, layers=layers, past=0, n=_log(rng, 2, 1500), steps=rng.randint(4, 20))


# ------------------------------------------------------------------------------------------------ states
_CTX = {}


def _context():
    """One context per process, on a stream of torch's (calls of all states are ordered on it)."""
    if not _CTX:
        ctx, stream = k2.Context(0), torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        _CTX.update(ctx=ctx, stream=stream)
    return _CTX["ctx"], _CTX["stream"]


class _Linear:
    """Matrices, their inputs and outputs."""

    def __init__(self, case, seed):
        self.ctx, self.stream = _context()
        self.host, self.n_tok, self.items, self.graph = case["where"] == "host", case["n_tok"], [], None
        for dm, x in zip(_linear_matrices(case, seed, self.ctx), _linear_inputs(case, seed)):
            cols, rows, nc = dm.cols, dm.rows, dm.cols // 64
            it = dict(dm=dm)
            if self.host:
                it.update(x=x.pin_memory(), out=torch.empty(self.n_tok, rows).pin_memory())
            else:
                it.update(x=x.cuda(), q=torch.empty(self.n_tok, cols, dtype=torch.int8, device="cuda"), s=torch.empty(self.n_tok, nc, device="cuda"),
                          m=torch.empty(self.n_tok, nc, dtype=torch.int32, device="cuda"), out=torch.empty(self.n_tok, rows, device="cuda"))
            self.items.append(it)
        if case["graph"]:
            torch.cuda.synchronize()
            self.launch()
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph, stream=self.stream):
                self.launch()

    def launch(self):
        n = self.n_tok
        if self.host:
            for it in self.items:
                self.ctx.linear_async_ptr(it["dm"], it["x"].data_ptr(), n, it["out"].data_ptr())
            self.ctx.synchronize()
            return
        for it in self.items:
            q, s, m = it["q"].data_ptr(), it["s"].data_ptr(), it["m"].data_ptr()
            self.ctx.fwht_quant_dev(it["x"].data_ptr(), n, it["dm"].cols, q, s, m)
            self.ctx.gemv_dev(it["dm"], q, s, m, n, it["out"].data_ptr())

    def __call__(self):
        if self.graph is not None:
            with torch.cuda.stream(self.stream):
                self.graph.replay()
        else:
            self.launch()
        return [it["out"] for it in self.items]

    def __del__(self):
        self.graph = None
        torch.cuda.synchronize()
        for it in self.items:
            it["dm"].free()


def _linear_list(case):
    """[(cols, rows, mode)] of a case."""
    return [(int(z.split("x")[0]), int(z.split("x")[1]), m) for z in case["sizes"].split(",") for m in case["modes"].split(",")]


def _linear_matrices(case, seed, ctx):
    for i, (cols, rows, mode) in enumerate(_linear_list(case)):
        m = synth.random_matrix(seed * 1000 + i, rows, cols, mode)
        if m.kind == 0:
            yield ctx.upload_bipolar(rows, cols, m.planes, m.data, m.scales)
        else:
            yield ctx.upload_nf(rows, cols, m.bits, m.sgc, m.codebook, m.pair, m.tail)


def _linear_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(case["n_tok"], cols, generator=g) for cols, _, _ in _linear_list(case)]


class _Model:
    """An engine with a filled cache, and the tokens of the pass."""

    def __init__(self, case, seed):
        self.engine = None
        ctx, _ = _context()
        spec = _spec(case, seed)
        self.tokens, filled = _tokens(case, seed, spec["cfg"]["vocab"])
        self.case, self.filled = case, filled.size
        self.engine = k2.Engine(ctx, spec)
        if filled.size:
            self.engine.forward_token_ids(filled)

    def __call__(self):
        c, e = self.case, self.engine
        if c["kind"] == "decode":
            toks, logits = e.decode_greedy(int(self.tokens[0]), self.filled, c["steps"], want_logits=True)
            return dict(tokens=toks, logits=logits)
        if c["kind"] == "prompt":
            return e.forward_token_ids(self.tokens, pos_start=self.filled)
        n, pos, out = c["n"], self.filled, []
        if n:
            out.append(e.forward_token_ids(self.tokens[:n], pos_start=pos))
        for i in range(c["steps"]):
            out.append(e.forward_token_ids(self.tokens[n + i:n + i + 1], pos_start=pos + n + i))
        return np.stack(out)

    def __del__(self):
        if self.engine is not None:
            self.engine.close()


def _spec(case, seed):
    if case["kind"] == "blocks":
        make = synth.random_folizen if case["design"] == "folizen" else synth.random_zasesun
        return make(case["shape"], seed=seed, max_seq=max(64, case["past"] + case["n"] + case["steps"]), layers=case["layers"])
    m = dict(MODELS[case["model"]])
    cfg = dict(m.pop("cfg"), layers=case["layers"], kv_bits=case["kv_bits"], kv_window=case.get("window", 0), kv_sinks=4)
    end = case["ctx"] + case["steps"] if case["kind"] == "decode" else case["past"] + case["n"]
    cfg["max_seq"] = max(64, end + 16, cfg["kv_window"] + 513 if cfg["kv_window"] else 0)
    return synth.random_model(cfg, m.pop("mode"), seed=seed % 1000003, share_layers=True, **m)


def _tokens(case, seed, vocab):
    """(tokens of the pass, tokens that fill the cache)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    filled = case["ctx"] if case["kind"] == "decode" else case["past"]
    n = 1 if case["kind"] == "decode" else case["n"] + case.get("steps", 0)
    return rng.integers(0, vocab, n).astype(np.uint32), rng.integers(0, vocab, filled).astype(np.uint32)


def prepare(case, seed):
    return _Linear(case, seed) if case["kind"] == "linear" else _Model(case, seed)


def run(state):
    return state()


# ------------------------------------------------------------------------------------------------ work
def _quantized_weights(case):
    """(file bytes read for one token, multiply-adds of one token's layer projections, of the head)."""
    m = MODELS[case["model"]]
    c, moe = m["cfg"], m.get("moe")
    md = dict(dict(qkv=m["mode"], o=m["mode"], gate_up=m["mode"], down=m["mode"], head=m["mode"]), **m.get("modes", {}))
    h, hd = c["hidden"], c["head_dim"]
    q, kv = c["n_q"] * hd, c["n_kv"] * hd
    mats = [(q + 2 * kv, h, md["qkv"]), (h, q, md["o"])]
    if moe:
        nf = f"nf{moe['bits']}g128"
        experts = moe["top_k"] * (_file_bytes(2 * moe["d_ff"], h, nf) + _file_bytes(h, moe["d_ff"], nf)) + 4 * moe["n_experts"] * h
        macs = moe["top_k"] * 3 * moe["d_ff"] * h + moe["n_experts"] * h
    else:
        experts, macs = 0, 0
        mats += [(2 * c["inter"], h, md["gate_up"]), (h, c["inter"], md["down"])]
    L = case["layers"]
    head = _file_bytes(c["vocab"], h, md["head"])
    return L * (sum(_file_bytes(*x) for x in mats) + experts) + head, L * (sum(r * k for r, k, _ in mats) + macs), c["vocab"] * h


def _file_bytes(rows, cols, mode):
    if mode.startswith("b"):
        return synth.file_bytes("bipolar", rows, cols, int(mode[1]))
    return synth.file_bytes("nf", rows, cols, int(mode[2]), 2 if mode.endswith("g128") and cols // 64 % 2 == 0 else 1)


def work(case):
    if case["kind"] == "linear":
        b = f = 0
        for cols, rows, mode in _linear_list(case):
            b += _file_bytes(rows, cols, mode) + case["n_tok"] * 4 * (cols + rows)
            f += 2 * rows * cols * case["n_tok"]
        return dict(bytes=b, flops=f)
    if case["kind"] in ("decode", "prompt"):
        c = MODELS[case["model"]]["cfg"]
        wb, macs, head = _quantized_weights(case)
        row = c["head_dim"] + 4 if case["kv_bits"] == 8 else c["head_dim"] // 2 + c["head_dim"] // 32
        pos_bytes = 2 * case["layers"] * c["n_kv"] * row
        att = 2 * case["layers"] * c["n_q"] * c["head_dim"]          # multiply-adds per pair of positions
        if case["kind"] == "decode":
            seen = min(case["ctx"], case["window"] or case["ctx"])
            return dict(bytes=case["steps"] * (wb + seen * pos_bytes), flops=2 * case["steps"] * (macs + head + att * seen))
        n, past = case["n"], case["past"]
        moe = MODELS[case["model"]].get("moe")
        if moe:          # the tokens of a prompt take nearly every expert: each is read once
            taken = moe["n_experts"] * (1.0 - (1.0 - moe["top_k"] / moe["n_experts"]) ** n)
            nf = f"nf{moe['bits']}g128"
            wb += int(case["layers"] * (taken - moe["top_k"]) * (_file_bytes(2 * moe["d_ff"], c["hidden"], nf) + _file_bytes(c["hidden"], moe["d_ff"], nf)))
        return dict(bytes=wb + (past + n) * pos_bytes, flops=2 * (n * macs + head + att * n * (past + (n + 1) / 2)))
    n, past, steps, L = case["n"], case["past"], case["steps"], case["layers"]
    if case["design"] == "folizen":
        c = synth.FOLIZEN_SHAPES[case["shape"]]
        h, hd, kv, side = c["hidden"], c["heads"] * c["dim"], c["kv_heads"] * c["dim"], 2 * c["side_dim"] * c["hidden"]
        na, nd = (L + 1) // 2, L // 2
        attn, delta = (hd + 2 * kv) * h + h * hd + 2 * c["ff"] * h + side, (5 * hd + c["rank"]) * h + hd * c["rank"] + h * hd + side
        macs, row, win = na * attn + nd * delta, na * 2 * kv * 2, c["window"]
        pair, state = na * 2 * hd, nd * c["heads"] * c["dim"] ** 2
        bytes_w = macs
    else:
        c = synth.ZASESUN_SHAPES[case["shape"]]
        h, H = c["hidden"], c["heads"]
        attn = (c["q_rank"] + c["kv_rank"] + c["rot_dim"]) * h + H * (c["dim"] + c["rot_dim"]) * c["q_rank"] + H * (c["dim"] + c["vdim"]) * c["kv_rank"] + h * H * c["vdim"]
        ne, nd = L // 2, (L + 1) // 2
        shared, one = (c["experts"] + 2 * c["shared_ff"]) * h, 2 * c["expert_ff"] * h
        macs = L * attn + nd * 3 * c["ff"] * h + ne * (shared + c["top"] * one)
        bytes_w = macs
        if n > 1:
            bytes_w += ne * (c["experts"] * (1.0 - (1.0 - c["top"] / c["experts"]) ** n) - c["top"]) * one
        row, win, pair, state = L * (c["kv_rank"] + c["rot_dim"]) * 2, 1 << 30, L * H * (c["dim"] + c["rot_dim"] + c["vdim"]), 0
    head = c["vocab"] * h
    by = fl = 0
    if n:
        by += 2 * (bytes_w + head) + n * row + 8 * state
        fl += 2 * (n * macs + head + n * min(past + (n + 1) / 2, win) * pair + 3 * n * state)
    seen = min(past + n, win)
    by += steps * (2 * (macs + head) + seen * row + 8 * state)
    fl += 2 * steps * (macs + head + seen * pair + 3 * state)
    return dict(bytes=by, flops=fl)


def tolerance(case):
    """Quantized paths follow one order of summation and are the same bit for bit.  Block models round activations to bf16 in
    front of every product: four times their distance from exact() (3.4e-3 with 12 blocks of folizen, 6e-3 with 4 of zasesun, whose
    experts change for a token now and then), the largest of some 50000 normal errors being 4.5 times their root mean square."""
    if case["kind"] != "blocks":
        return "exact"
    return dict(rel=1.4e-2, max=8e-2) if case["design"] == "folizen" else dict(rel=2.4e-2, max=1.2e-1)


# ------------------------------------------------------------------------------------------------ exact values
def exact(case, seed):
    """64-bit values.  Whole quantized models have none: every layer rounds its activations to int8, and a run in other precision takes
    other integers from the second layer on (their outputs are compared bit for bit instead)."""
    if case["kind"] == "linear":
        return _exact_linear(case, seed)
    if case["kind"] == "blocks":
        return _exact_blocks(case, seed)
    return None


def _signs(n_chunks):
    """[n_chunks][64] of +-1: one SplitMix64 stream per 64-column chunk, the lowest bit of every word."""
    mask = (1 << 64) - 1
    out = np.empty((n_chunks, 64))
    for b in range(n_chunks):
        s = (0x9E3779B97F4A7C15 + b * 0xBF58476D1CE4E5B9) & mask
        for i in range(64):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            out[b, i] = -1.0 if (z ^ (z >> 31)) & 1 else 1.0
    return torch.from_numpy(out)


def _bf16(u16):
    return torch.from_numpy((np.asarray(u16, np.uint16).astype(np.uint32) << 16).view(np.float32)).cuda().double()


def _dequantized(m):
    """[rows][cols] of a host matrix in the file formats, in 64 bits."""
    rows, cols, nc = m.rows, m.cols, m.cols // 64
    ns = (rows + 15) // 16
    if m.kind == 0:          # [stripe][cols / 8][plane][16 rows], a bit per column; scales [stripe][chunk][16 rows]
        d = torch.from_numpy(m.data).cuda().view(ns, cols // 8, m.planes, 16)
        code = torch.zeros(ns, cols // 8, 16, 8, device="cuda")
        for p in range(m.planes):
            for k in range(8):
                code[..., k] += ((d[:, :, p] >> k) & 1) << p
        w = (2.0 * code - (2 ** m.planes - 1)).permute(0, 2, 1, 3).reshape(ns * 16, nc, 64).double()
        return (w * _bf16(m.scales).view(ns, nc, 16).permute(0, 2, 1).reshape(ns * 16, nc, 1)).reshape(ns * 16, cols)[:rows]
    # pairs of stripes: per scale group 64 bytes of scales, then per chunk 512 bytes of each stripe: [k 4][g 4][half 2][j 4][t 4],
    # the low nibble holds column 16 k + 8 half + t of row 4 g + j, the high one column 16 k + 8 half + 4 + t
    d = torch.from_numpy(m.pair).cuda().view(rows // 32, nc // m.sgc, 64 + m.sgc * 1024)
    sc = _bf16(d[:, :, :64].contiguous().cpu().numpy().view(np.uint16)).view(rows // 32, nc // m.sgc, 1, 32)
    c = d[:, :, 64:].reshape(rows // 32, nc // m.sgc, m.sgc, 2, 4, 4, 2, 4, 4)
    book = torch.from_numpy(m.codebook.astype(np.float64)).cuda()
    w = torch.stack([book[(c & 15).long()], book[(c >> 4).long()]], dim=-2)          # [pair][group][chunk][stripe][k][g][half][j][nibble][t]
    w = w.permute(0, 1, 2, 3, 5, 7, 4, 6, 8, 9).reshape(rows // 32, nc // m.sgc, m.sgc, 32, 64) * sc.unsqueeze(-1)
    return w.permute(0, 3, 1, 2, 4).reshape(rows, cols)


def _exact_linear(case, seed):
    out = []
    had = torch.ones(1, 1, dtype=torch.float64)
    for _ in range(6):
        had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)], 0)
    for i, ((cols, rows, mode), x) in enumerate(zip(_linear_list(case), _linear_inputs(case, seed))):
        nc = cols // 64
        v = (x.double().view(-1, nc, 64) * _signs(nc) / 8.0) @ had
        top = v.abs().amax(-1, keepdim=True)
        q = torch.round(v * (127.0 / top)) * (top / 127.0)
        w = _dequantized(synth.random_matrix(seed * 1000 + i, rows, cols, mode))
        y = q.reshape(-1, cols).cuda() @ w.T
        out.append(y.cpu() if case["where"] == "host" else y)
    return out


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _f64(v):
    return torch.from_numpy(np.asarray(v)).cuda().double() if v.dtype != np.uint16 else _bf16(v)


def _causal(q, k, v, scale, slope, window):
    """q [T][H][d], k [T][G][d], v [T][G][dv]: softmax attention of head h over key head h // (H / G)."""
    T, H, _ = q.shape
    G = k.shape[1]
    dist = torch.arange(T, device="cuda").view(-1, 1) - torch.arange(T, device="cuda")
    hide = (dist < 0) | (dist >= window)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale[h] - slope[h] * dist
        out.append(torch.softmax(s.masked_fill(hide, -math.inf), -1) @ v[:, h * G // H])
    return torch.stack(out, 1)


def _window_mixer(x, b, p, eps):
    T, H, G, d, dv = x.shape[0], b["heads"], b["kv_heads"], b["dim"], b["vdim"]
    y = x @ p["in_proj"].T
    q, k, v = (t.view(T, -1, n) for t, n in zip(y.split([H * d, G * d, G * dv], -1), (d, d, dv)))
    o = _causal(_rms(q, eps) * p["q_norm"], _rms(k, eps) * p["k_norm"], v, p["head_scale"], p["head_slope"], b["window"] or 1 << 30)
    return o.reshape(T, -1) @ p["o_proj"].T


def _delta_mixer(x, b, p, eps):
    T, H, d = x.shape[0], b["heads"], b["dim"]
    n = H * d
    r, k, v, g, a, low = (x @ p["in_proj"].T).split([n, n, n, n, n, b["decay_rank"]], -1)
    decay = torch.tanh(low) @ p["decay_proj"].T + p["decay_bias"]
    w = torch.exp(-b["decay_scale"] * torch.sigmoid(decay)).view(T, H, d, 1)
    a = torch.sigmoid(a + p["rate_bias"]).view(T, H, d)
    r, k, v = (t.view(T, H, d) for t in (r, k, v))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + b["unit_eps"])
    au, kc, vr, ur, rr = (a * u).unsqueeze(-1), k.unsqueeze(-1), v.unsqueeze(-2), u.unsqueeze(-2), r.unsqueeze(-2)
    S, out = torch.zeros(H, d, d, device="cuda", dtype=torch.float64), []
    for t in range(T):          # S <- diag(w) S - (a u)(u^T S) + k v^T, o = S^T r
        S = torch.baddbmm(torch.baddbmm(w[t] * S, au[t], torch.bmm(ur[t], S), alpha=-1.0), kc[t], vr[t])
        out.append(torch.bmm(rr[t], S).squeeze(1))
    o = _rms(torch.stack(out), eps).reshape(T, n) * p["out_norm"] * torch.sigmoid(g)
    return o @ p["o_proj"].T


def _latent_mixer(x, b, p, eps):
    T, H, d, dr, dv, rank = x.shape[0], b["heads"], b["dim"], b["rot_dim"], b["vdim"], b["kv_rank"]
    y = x @ p["in_proj"].T
    ql, c, kr = y.split([b["q_rank"], rank, dr], -1)
    q = ((_rms(ql, eps) * p["q_latent_norm"]) @ p["q_up"].T).view(T, H, d + dr)
    kv = (_rms(c, eps) * p["kv_latent_norm"]) @ p["kv_up"].T
    cs = p["rot_cos_sin"][:T].view(T, 1, dr // 2, 2)          # (cos, sin) of the pairs (2 i, 2 i + 1)

    def turn(z):
        z = z.reshape(T, -1, dr // 2, 2)
        return torch.stack([z[..., 0] * cs[..., 0] - z[..., 1] * cs[..., 1], z[..., 1] * cs[..., 0] + z[..., 0] * cs[..., 1]], -1).reshape(T, -1, dr)

    k = torch.cat([kv[:, :H * d].view(T, H, d), turn(kr).expand(T, H, dr)], -1)
    q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
    one = torch.ones(H, device="cuda", dtype=torch.float64)
    o = _causal(q, k, kv[:, H * d:].view(T, H, dv), one * b["score_scale"], 0.0 * one, 1 << 30)
    return o.reshape(T, H * dv) @ p["o_proj"].T


def _feed_forward(x, b, p, eps):
    if b.get("experts"):
        E, ff = b["experts"], b["ff"]
        y = x @ p["router"].T
        score, chosen = torch.softmax(y[:, :E], -1).topk(b["experts_top"], -1)
        out = torch.relu(y[:, E:]) ** 2 @ p["shared_down"].T
        up, down = p["up_proj"].view(E, ff, -1), p["down_proj"].view(E, -1, ff)
        for e in range(E):
            t, slot = torch.nonzero(chosen == e, as_tuple=True)
            if t.numel():
                out[t] += score[t, slot].unsqueeze(-1) * (torch.relu(x[t] @ up[e].T) ** 2 @ down[e].T)
        return out
    z = x @ p["up_proj"].T
    if b.get("act", 0) == 1:          # rows 2 i = gate, 2 i + 1 = up
        return (_gelu(z[:, 0::2]) * z[:, 1::2]) @ p["down_proj"].T
    a1, a2, a3, a0 = (float(v) for v in b["act_coef"])
    return (a1 * _rms(z, eps) + a2 * _rms(z * z, eps) + a3 * _rms(z ** 3, eps) + a0) @ p["down_proj"].T


def _exact_blocks(case, seed):
    """The whole sequence at once; the logits of the prompt's last token and of every token after it."""
    spec = _spec(case, seed)
    c, eps, mult = spec["cfg"], spec["cfg"]["eps"], spec["cfg"].get("residual_mult", 1.0)
    toks, filled = _tokens(case, seed, c["vocab"])
    ids = np.concatenate([filled, toks]).astype(np.int64)
    mixers = {1: _window_mixer, 2: _delta_mixer, 3: _latent_mixer}
    sd = c.get("side_dim", 0)
    x = _bf16(spec["embed"][ids])
    kept = {}
    for i, b in enumerate(spec["blocks"]):
        if id(b) not in kept:
            kept[id(b)] = {k: _f64(v) for k, v in b.items() if isinstance(v, np.ndarray) and k != "act_coef"}
        p = kept[id(b)]
        pre = lambda name: _rms(x, eps) * p[name] if name in p else x  # noqa: E731
        x = x + mult * _rms(mixers[b["mixer"]](pre("pre_norm1"), b, p, eps), eps) * p["norm1"]
        if b.get("ff", 0):
            x = x + mult * _rms(_feed_forward(pre("pre_norm2"), b, p, eps), eps) * p["norm2"]
        if sd:
            e = _bf16(spec["side_embed"][ids, i * sd:(i + 1) * sd])
            x = x + _rms((_gelu(x @ p["side_gate"].T) * e) @ p["side_proj"].T, eps) * p["side_norm"]
    first = len(filled) + max(case["n"], 1) - 1
    y = (_rms(x[first:], eps) * _f64(spec["final_norm"])) @ _bf16(spec["head"]).T
    cap = c.get("logit_softcap", 0.0)
    return (cap * torch.tanh(y / cap) if cap else y).cpu().numpy()
