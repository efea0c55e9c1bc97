"""The workloads whose speed this repository follows: what a program that uses the framework asks of it, through the entry
points that it calls, over the sizes that the configurations, tests and benchmarks here use.

Two engines serve two kinds of program.  The single-sequence decoder (`Decoder`) answers one user: `generate` decodes,
`prefill_tf32` takes a prompt in.  The sequence-batch engine (`kllm_seq_*`) serves many: one step carries the prompts or the
next tokens of all of them through layers that are described by data.  Both rest on matrix products that can be called alone.

A case is a dict of plain values; "kind" says which of these it is:

  decode    `Decoder.generate` of a few tokens behind a context, then the logits
  prefill   `Decoder.prefill_tf32` of a prompt, then the logits
  product   `kllm_seq_gemm`: a block of tokens against a weight matrix
  prompt    one engine step with the prompts of several new sequences, logits of every prompt's last token
  score     one engine step with several texts, logits of every token
  serve     prompts of several sequences in one step, then steps that bring one token of each, logits of every step
"""
import ctypes
import math
from dataclasses import replace

import numpy as np
import torch

from kuiperllama_b200 import Decoder, SHAPES, synth_weights
from kuiperllama_b200 import sequence as sq

FAMILY_MIXERS = ("attention", "latent", "linear")


# ---- the cases ----------------------------------------------------------------------------------------------------------
def engine_case(name, kind, mixer, ff, dtype, width, heads, kv_heads, dim, ff_size, entries, tokens, **more):
    c = {"kind": kind, "mixer": mixer, "ff": ff, "dtype": dtype, "width": width, "heads": heads, "kv_heads": kv_heads,
         "dim": dim, "ff_size": ff_size, "entries": entries, "tokens": tokens, "layers": 1, "steps": 0, "vocab": 8192,
         "experts": 0, "top": 0, "window": 0}
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the headline: one user's chat on the 1.1B checkpoint, half-way through its context; nearly all of a session's time
        {"name": "decode-1b-fp32", "kind": "decode", "shape": "tinyllama-1.1b", "layers": 22, "numerics": "fast",
         "context": 500, "steps": 12},
        # the quantised 7B checkpoint: a quarter of its layers at full width, early in a chat
        {"name": "decode-7b-int8", "kind": "decode", "shape": "llama2-7b-int8", "layers": 8, "numerics": "fast",
         "context": 200, "steps": 12},
        # the smallest model, one token per call as an interactive loop asks for it: latency only
        {"name": "step-15m-fp32", "kind": "decode", "shape": "stories15m", "layers": 6, "numerics": "exact",
         "context": 41, "steps": 1},
        # a document read in before the chat starts: the prompt path of the single-sequence decoder
        {"name": "prefill-1b-tf32", "kind": "prefill", "shape": "tinyllama-1.1b", "layers": 4, "tokens": 900},
        # the products that carry a prompt step: a feed-forward's projection over a full block of tokens
        {"name": "product-bf16-block", "kind": "product", "dtype": "bf16", "tokens": 2048, "in_dim": 2048, "out_dim": 8192},
        # the same projection for a decode batch: a few dozen users, one token each
        {"name": "product-bf16-batch", "kind": "product", "dtype": "bf16", "tokens": 40, "in_dim": 4096, "out_dim": 4096},
        # checkpoints kept in fp32: a prompt of an odd length
        {"name": "product-fp32-block", "kind": "product", "dtype": "fp32", "tokens": 517, "in_dim": 1024, "out_dim": 3072},
        # four documents arriving at once at a server, one layer of a dense model with grouped-query attention
        engine_case("prompt-attention-bf16", "prompt", "attention", "dense", "bf16", 2048, 16, 4, 128, 4096, 4, 6001),
        # texts scored token by token through a layer of routed experts with a shared one
        engine_case("score-experts-bf16", "score", "attention", "moe", "bf16", 2048, 16, 4, 128, 768, 3, 1501,
                    experts=32, top=4, vocab=256),
        # two prompts for a model kept in fp32
        engine_case("prompt-attention-fp32", "prompt", "attention", "dense", "fp32", 1024, 16, 4, 64, 2048, 2, 700),
        # two dozen chats decoded together: the serving loop's steady state
        engine_case("serve-attention-bf16", "serve", "attention", "dense", "bf16", 2048, 16, 4, 128, 4096, 24, 1200,
                    layers=4, steps=12),
        # three chats on a model with a retention in every layer: state instead of a cache
        engine_case("serve-linear-bf16", "serve", "linear", "dense", "bf16", 1024, 16, 16, 64, 2048, 3, 210, layers=4, steps=12),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "product", "product", "prompt", "prompt", "score", "serve", "serve"])
    if kind == "decode":
        shape, layers = rng.choice([("tinyllama-1.1b", 8), ("llama2-7b-int8", 4), ("qwen2.5-0.5b", 6), ("stories15m", 6)])
        top = 240 if shape == "stories15m" else 700
        return {"kind": kind, "shape": shape, "layers": rng.randint(layers // 2, layers), "numerics": rng.choice(["fast", "exact"]),
                "context": log_int(rng, 3, top), "steps": rng.randint(1, 10)}
    if kind == "prefill":
        return {"kind": kind, "shape": rng.choice(["tinyllama-1.1b", "qwen2.5-0.5b"]), "layers": rng.randint(2, 3),
                "tokens": log_int(rng, 30, 800)}
    if kind == "product":
        dtype = rng.choice(["bf16", "bf16", "fp32"])
        return {"kind": kind, "dtype": dtype, "tokens": log_int(rng, 1, 2048 if dtype == "bf16" else 500),
                "in_dim": 8 * rng.randint(36, 512), "out_dim": rng.randint(288, 6000)}
    mixer = rng.choice(FAMILY_MIXERS)
    dtype = rng.choice(["bf16", "bf16", "fp32"])
    dim = rng.choice([64, 128])
    heads = rng.choice([8, 16])
    kv = rng.choice([2, 4, heads]) if mixer == "attention" else heads
    width = 64 * rng.randint(8, 32)
    more = {"window": rng.choice([0, 0, 512]) if mixer != "linear" else 0}
    if kind == "prompt":
        return engine_case(None, kind, mixer, "dense", dtype, width, heads, kv, dim, 2 * width, rng.randint(1, 6),
                           log_int(rng, 60, 3000 if dtype == "bf16" else 600), **more)
    if kind == "score":
        return engine_case(None, kind, mixer, "moe", dtype, width, heads, kv, dim, 64 * rng.randint(4, 12), rng.randint(1, 4),
                           log_int(rng, 60, 1500 if dtype == "bf16" else 400), experts=rng.choice([16, 32]), top=rng.choice([2, 4]),
                           vocab=256, **more)
    entries = log_int(rng, 1, 64)
    return engine_case(None, kind, mixer, "dense", dtype, width, heads, kv, dim, 2 * width, entries,
                       entries * rng.randint(4, 60), layers=rng.randint(1, 4), steps=rng.randint(2, 12), **more)


# ---- shared ---------------------------------------------------------------------------------------------------------------
def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def shape_of(case):
    return replace(SHAPES[case["shape"]], layer_num=case["layers"])


def lengths(case):
    """Prompt lengths of the entries: unequal, together `tokens`."""
    n, total = case["entries"], case["tokens"]
    share = [4 + (7 * i) % 5 for i in range(n)]
    out = [max(1, total * s // sum(share)) for s in share]
    out[0] += max(0, total - sum(out))
    return out


def token_ids(seed, n, vocab):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(seed)).tolist()


# ---- the single-sequence decoder -----------------------------------------------------------------------------------------
def decoder_tokens(case, seed):
    n = case["context"] + case["steps"] if case["kind"] == "decode" else case["tokens"]
    return token_ids(seed, n, SHAPES[case["shape"]].vocab_size)


def prepare_decoder(case, seed):
    shape = shape_of(case)
    dec = Decoder(shape, synth_weights(shape, "cuda", seed), numerics=case.get("numerics", "exact"))
    tokens = decoder_tokens(case, seed)
    if case["kind"] == "decode":  # what was said so far is in the cache
        dec.prompt(tokens[:case["context"]])
    return {"case": case, "dec": dec, "tokens": tokens}


def run_decoder(s):
    case, dec, tokens = s["case"], s["dec"], s["tokens"]
    if case["kind"] == "prefill":
        dec.prefill_tf32(tokens)
    elif case["steps"] == 1:
        dec.step(tokens[-1], case["context"])
    else:  # given tokens: the work is that of greedy decoding, and every position has one right answer
        dec.generate(tokens[case["context"]], case["context"], case["steps"], teacher=tokens[case["context"]:])
    return dec.logits()


def decoder_positions(case):
    return range(case["context"], case["context"] + case["steps"]) if case["kind"] == "decode" else range(case["tokens"])


def work_decoder(case):
    s = shape_of(case)
    per_token = 2 * (s.layer_num * (2 * s.dim * s.dim + 2 * s.kv_dim * s.dim + 3 * s.hidden_dim * s.dim))
    head = 2 * s.vocab_size * s.dim
    attend = sum(4 * s.layer_num * s.dim * (p + 1) for p in decoder_positions(case))
    if case["kind"] == "prefill":
        n = case["tokens"]
        return {"bytes": s.weight_bytes_per_token() + s.kv_bytes_at(n) + 4 * n * s.dim + 4 * s.vocab_size,
                "flops": n * per_token + head + attend}
    n = case["steps"]
    return {"bytes": sum(s.weight_bytes_per_token() + s.kv_bytes_at(p) for p in decoder_positions(case)) + 4 * s.vocab_size,
            "flops": n * (per_token + head) + attend}


def rms(x, w, eps):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if w is None else x * w.double()


def rotate(x, pos, base, dims, pairs):
    """x [T, heads, dim]: rotary positions on the first `dims` coordinates, neighbours paired or halves."""
    f = base ** (-2.0 * torch.arange(dims // 2, device=x.device, dtype=torch.float64) / dims)
    a = pos.double()[:, None] * f
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if pairs else (x[..., :dims // 2], x[..., dims // 2:dims])
    p, q = u * c - v * s, v * c + u * s
    r = torch.stack([p, q], -1).flatten(-2) if pairs else torch.cat([p, q], -1)
    return torch.cat([r, x[..., dims:]], -1)


def attend(q, k, v, scale, window=0):
    """q [T, heads, d], k and v [T, kv_heads, d]: causal softmax attention, head by head."""
    t = q.shape[0]
    i = torch.arange(t, device=q.device)
    seen = i[:, None] >= i[None, :]
    if window:
        seen &= i[:, None] - i[None, :] < window
    per = q.shape[1] // k.shape[1]
    out = []
    for h in range(q.shape[1]):
        sc = (q[:, h] @ k[:, h // per].T * scale).masked_fill(~seen, -math.inf)
        out.append(torch.softmax(sc, -1) @ v[:, h // per])
    return torch.stack(out, 1)


def exact_decoder(case, seed):
    s = shape_of(case)
    w = synth_weights(s, "cuda", seed)
    tokens = torch.tensor(decoder_tokens(case, seed), device="cuda")
    qwen = s.flavour == "qwen2"
    eps, base = (1e-6, 1e6) if qwen else (1e-5, 1e4)

    def mat(name, layer=None):
        m = w[name] if layer is None else w[name][layer]
        if s.group_size:
            sc = w["s" + name[1:]] if layer is None else w["s" + name[1:]][layer]
            return (m.double().reshape(-1, s.group_size) * sc.double().reshape(-1, 1)).reshape(m.shape)
        return m.double()

    pos = torch.arange(len(tokens), device="cuda")
    x = w["tok_emb"][tokens].double()
    for l in range(s.layer_num):
        h = rms(x, w["attn_norm"][l], eps)
        q, k, v = h @ mat("wq", l).T, h @ mat("wk", l).T, h @ mat("wv", l).T
        if "bq" in w:
            q, k, v = q + w["bq"][l].double(), k + w["bk"][l].double(), v + w["bv"][l].double()
        q, k, v = (t.reshape(len(tokens), -1, s.head_size) for t in (q, k, v))
        q, k = rotate(q, pos, base, s.head_size, not qwen), rotate(k, pos, base, s.head_size, not qwen)
        x = x + attend(q, k, v, s.head_size ** -0.5).flatten(1) @ mat("wo", l).T
        h = rms(x, w["ffn_norm"][l], eps)
        x = x + (torch.nn.functional.silu(h @ mat("w1", l).T) * (h @ mat("w3", l).T)) @ mat("w2", l).T
    x = rms(x[-1], w["final_norm"], eps)
    return (x @ (mat("wcls") if w["wcls"] is not None else w["tok_emb"].double()).T).cpu().numpy()


# ---- a product ------------------------------------------------------------------------------------------------------------
def product_inputs(case, seed):
    td = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    g = gen(seed)
    a = torch.randn(case["tokens"], case["in_dim"], device="cuda", generator=g).to(td)
    w = (torch.randn(case["out_dim"], case["in_dim"], device="cuda", generator=g) * case["in_dim"] ** -0.5).to(td)
    return a, w


def prepare_product(case, seed):
    a, w = product_inputs(case, seed)
    return {"case": case, "a": a, "w": w, "lib": sq.load_seq_library(),
            "out": torch.empty(case["tokens"], case["out_dim"], device="cuda")}


def run_product(s):
    case = s["case"]
    rc = s["lib"].kllm_seq_gemm(sq.BF16 if case["dtype"] == "bf16" else sq.F32, s["a"].data_ptr(), s["w"].data_ptr(),
                                s["out"].data_ptr(), case["tokens"], case["in_dim"], case["out_dim"],
                                torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError(f"kllm_seq_gemm: {rc}")
    return s["out"]


# ---- the sequence-batch engine ----------------------------------------------------------------------------------------------
EPS, ROPE_BASE = 1e-5, 1e4


def engine_weights(case, seed):
    """Weights of a model with case["layers"] equal layers; matrices in the compute type, vectors in fp32."""
    td = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    g = gen(seed)
    W, H, KV, D = case["width"], case["heads"], case["kv_heads"], case["dim"]

    def mat(rows, cols, lead=()):
        return (torch.randn(*lead, rows, cols, device="cuda", generator=g) * cols ** -0.5).to(td).contiguous()

    def vec(n):
        return 1 + 0.05 * torch.randn(n, device="cuda", generator=g)

    layers = []
    for _ in range(case["layers"]):
        p = {"norm1": vec(W), "norm2": vec(W)}
        if case["mixer"] == "attention":
            p["w_in"] = mat((H + 2 * KV) * D, W)
            p["q_norm"], p["k_norm"] = vec(D), vec(D)
        elif case["mixer"] == "latent":  # half of a head's coordinates again as rotated ones, a latent of two heads' size
            p["w_in"] = mat(H * (D + D // 2) + 2 * D + D // 2, W)
            p["kv_norm"] = vec(2 * D)
            p["w_ukv"] = mat(2 * H * D, 2 * D)
        else:
            p["w_in"] = mat(4 * H * D, W)
            p["decay"] = torch.tensor([1.0 - 2.0 ** (-5 - h % 8) for h in range(H)], device="cuda")
        p["w_out"] = mat(W, H * D)
        F, E = case["ff_size"], case["experts"]
        if case["ff"] == "dense":
            p["up"], p["down"] = mat(2 * F, W), mat(W, F)
        else:
            p["router"] = torch.randn(E, W, device="cuda", generator=g) * W ** -0.5
            p["gate_up"], p["expert_down"] = mat(2 * F, W, (E,)), mat(W, F, (E,))
            p["shared_up"], p["shared_down"] = mat(4 * F, W), mat(W, 2 * F)
            p["shared_gate"] = torch.randn(W, device="cuda", generator=g) * W ** -0.5
        layers.append(p)
    return {"layers": layers, "embed": torch.randn(case["vocab"], W, device="cuda", generator=g).to(td),
            "final": vec(W), "head": mat(case["vocab"], W)}


class Engine:
    """A `kllm_seq_engine` over weights that it keeps alive."""

    def __init__(self, case, weights):
        self.lib = sq.load_seq_library()
        self.weights = weights
        W, H, KV, D, F = case["width"], case["heads"], case["kv_heads"], case["dim"], case["ff_size"]
        layers = (sq.Layer * case["layers"])()
        for L, p in zip(layers, weights["layers"]):
            L.pre_mixer, L.pre_ff = sq.Norm(p["norm1"].data_ptr(), None, 1), sq.Norm(p["norm2"].data_ptr(), None, 1)
            if case["mixer"] == "attention":
                L.mixer_kind, a = 1, L.attn
                a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.qk_norm, a.window = H, KV, D, D, D ** -0.5, 1, case["window"]
                a.rope_dims, a.rope_base = D, ROPE_BASE
                a.q_norm_w, a.k_norm_w = p["q_norm"].data_ptr(), p["k_norm"].data_ptr()
            elif case["mixer"] == "latent":
                L.mixer_kind, a = 2, L.latent
                a.heads, a.dim, a.rot_dim, a.vdim, a.q_rank, a.kv_rank = H, D, D // 2, D, 0, 2 * D
                a.scale, a.window, a.rope_dims, a.rope_base = (D + D // 2) ** -0.5, case["window"], D // 2, ROPE_BASE
                a.kv_norm_w, a.w_uk = p["kv_norm"].data_ptr(), p["w_ukv"].data_ptr()
                a.w_uv = p["w_ukv"][H * D:].data_ptr()
            else:
                L.mixer_kind, a = 3, L.linear
                a.heads, a.dim, a.vdim, a.decay, a.qkv_act = H, D, D, p["decay"].data_ptr(), 1
                a.rope_dims, a.rope_base, a.k_scale, a.out_norm, a.gate_act = D, ROPE_BASE, D ** -0.5, 1, 1
            a.w_in, a.w_out = p["w_in"].data_ptr(), p["w_out"].data_ptr()
            if case["ff"] == "dense":
                L.ff_kind = 2
                L.dense.ff, L.dense.act, L.dense.up, L.dense.down = F, 5, p["up"].data_ptr(), p["down"].data_ptr()
            else:
                L.ff_kind, m = 1, L.moe
                m.experts, m.top, m.ff, m.router_scale = case["experts"], case["top"], F, 1.0
                m.w_router, m.gate_up, m.down = p["router"].data_ptr(), p["gate_up"].data_ptr(), p["expert_down"].data_ptr()
                m.shared_ff, m.shared_gate_up, m.shared_down = 2 * F, p["shared_up"].data_ptr(), p["shared_down"].data_ptr()
                m.w_shared_gate = p["shared_gate"].data_ptr()
        d = sq.Desc()
        d.dtype, d.width, d.vocab, d.norm_eps = sq.BF16 if case["dtype"] == "bf16" else sq.F32, W, case["vocab"], EPS
        order = (ctypes.c_int32 * case["layers"])(*range(case["layers"]))
        d.n_layers, d.layers, d.n_runs, d.run_layer = case["layers"], layers, case["layers"], order
        d.embed, d.final_norm, d.head = weights["embed"].data_ptr(), sq.Norm(weights["final"].data_ptr(), None, 1), \
            weights["head"].data_ptr()
        d.max_tokens, d.max_seqs = sum(lengths(case)) + case["entries"] * case["steps"] + 64, case["entries"]
        self.handle = ctypes.c_void_p()
        torch.cuda.synchronize()  # the engine has a stream of its own
        self.check(self.lib.kllm_seq_create(ctypes.byref(d), None, ctypes.byref(self.handle)))

    def check(self, rc):
        if rc != 0:
            raise RuntimeError(f"sequence engine: {self.lib.kllm_error_string(rc).decode()} ({rc})")

    def __del__(self):
        if getattr(self, "handle", None):
            self.lib.kllm_seq_destroy(self.handle)


def engine_plan(case, seed):
    """The tokens of every step: [[tokens of entry 0, tokens of entry 1, ...], ...]."""
    ns = lengths(case)
    ids = token_ids(seed, sum(ns) + case["entries"] * case["steps"], case["vocab"])
    plan, at = [[]], 0
    for n in ns:
        plan[0].append(ids[at:at + n])
        at += n
    for _ in range(case["steps"]):
        plan.append([[t] for t in ids[at:at + case["entries"]]])
        at += case["entries"]
    return plan


def prepare_engine(case, seed):
    """An engine, and for every step its tokens as host arrays and a pinned buffer for its logits."""
    steps = []
    for entries in engine_plan(case, seed):
        flat = [t for e in entries for t in e]
        if case["kind"] == "score":
            want = list(range(len(flat)))
        else:
            want = (np.cumsum([len(e) for e in entries]) - 1).tolist()
        steps.append({"counts": (ctypes.c_int32 * len(entries))(*[len(e) for e in entries]),
                      "tokens": (ctypes.c_int32 * len(flat))(*flat), "n": len(want),
                      "want": (ctypes.c_int32 * len(want))(*want),
                      "logits": torch.empty(len(want), case["vocab"], pin_memory=True)})
    return {"case": case, "engine": Engine(case, engine_weights(case, seed)), "steps": steps}


def run_engine(s):
    eng, n = s["engine"], s["case"]["entries"]
    lib, seqs = eng.lib, (ctypes.c_int32 * n)()
    for i in range(n):
        one = ctypes.c_int32(-1)
        eng.check(lib.kllm_seq_open(eng.handle, ctypes.byref(one)))
        seqs[i] = one.value
    for st in s["steps"]:
        eng.check(lib.kllm_seq_step(eng.handle, n, seqs, st["counts"], st["tokens"], st["n"], st["want"],
                                    st["logits"].data_ptr(), None))
    for i in range(n):
        eng.check(lib.kllm_seq_close(eng.handle, seqs[i]))
    return [st["logits"] for st in s["steps"]]


def proj_rows(case):
    H, KV, D = case["heads"], case["kv_heads"], case["dim"]
    return {"attention": (H + 2 * KV) * D, "latent": H * (D + D // 2) + 2 * D + D // 2, "linear": 4 * H * D}[case["mixer"]]


def work_engine(case):
    es = 2 if case["dtype"] == "bf16" else 4
    W, H, KV, D, F, E = (case[k] for k in ("width", "heads", "kv_heads", "dim", "ff_size", "experts"))
    ns = lengths(case)
    mixer = (proj_rows(case) + H * D) * W + (4 * H * D * D if case["mixer"] == "latent" else 0)
    cached = {"attention": 2 * KV * D, "latent": 2 * D + D // 2, "linear": 0}[case["mixer"]]
    state = H * D * D * 4 if case["mixer"] == "linear" else 0
    reach = (lambda p: min(p + 1, case["window"]) if case["window"] else p + 1) if case["mixer"] != "linear" else (lambda p: 0)
    pair = H * (4 * D if case["mixer"] != "latent" else 5 * D)  # scores and weighted values of one query and one key
    flops = bytes_ = 0
    for step in range(1 + case["steps"]):
        T = sum(ns) if step == 0 else case["entries"]
        rows = T if case["kind"] == "score" else case["entries"]
        first = [0] * len(ns) if step == 0 else [n + step - 1 for n in ns]
        last = ns if step == 0 else [n + step for n in ns]
        keys = sum(reach(p) for a, b in zip(first, last) for p in range(a, b))
        if case["ff"] == "dense":
            ff_read, ff_mul = 3 * F * W, 3 * F * W
        else:
            ff_read = E * (1 - (1 - case["top"] / E) ** T) * 3 * F * W + 6 * F * W + E * W * 4 / es
            ff_mul = (case["top"] * 3 * F + 6 * F + E) * W
        layer = 2 * T * (mixer + ff_mul) + pair * keys + (4 * T * H * D * D if state else 0)
        read = (mixer + ff_read) * es + sum(last) * cached * es + 2 * len(ns) * state
        flops += case["layers"] * layer + 2 * rows * case["vocab"] * W
        bytes_ += case["layers"] * read + case["vocab"] * W * es + T * W * es + rows * case["vocab"] * 4
    return {"bytes": bytes_, "flops": flops}


def exact_mixer(case, p, h, pos):
    H, KV, D = case["heads"], case["kv_heads"], case["dim"]
    t = h.shape[0]
    y = h @ p["w_in"].double().T
    if case["mixer"] == "attention":
        q, k, v = (m.reshape(t, -1, D) for m in y.split([H * D, KV * D, KV * D], 1))
        q, k = rms(q, p["q_norm"], EPS), rms(k, p["k_norm"], EPS)
        o = attend(rotate(q, pos, ROPE_BASE, D, False), rotate(k, pos, ROPE_BASE, D, False), v, D ** -0.5, case["window"])
    elif case["mixer"] == "latent":
        R = D // 2
        q, c, r = y.split([H * (D + R), 2 * D, R], 1)
        q = q.reshape(t, H, D + R)
        q = torch.cat([q[..., :D], rotate(q[..., D:], pos, ROPE_BASE, R, False)], -1)
        kv = rms(c, p["kv_norm"], EPS) @ p["w_ukv"].double().T
        r = rotate(r.reshape(t, 1, R), pos, ROPE_BASE, R, False).expand(t, H, R)
        k = torch.cat([kv[:, :H * D].reshape(t, H, D), r], -1)
        o = attend(q, k, kv[:, H * D:].reshape(t, H, D), (D + R) ** -0.5, case["window"])
    else:
        q, k, v, z = (m.reshape(t, H, D) for m in y.split(H * D, 1))
        q, k = rotate(q, pos, ROPE_BASE, D, False), rotate(k, pos, ROPE_BASE, D, False) * D ** -0.5
        ago = (pos[:, None] - pos[None, :]).double()
        o = torch.stack([(q[:, i] @ k[:, i].T * torch.where(ago >= 0, p["decay"][i].double() ** ago.clamp(min=0), 0.0)) @ v[:, i]
                         for i in range(H)], 1)
        o = rms(o, None, EPS) * torch.nn.functional.silu(z)
    return o.flatten(1) @ p["w_out"].double().T


def exact_ff(case, p, h):
    F = case["ff_size"]
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
    silu = torch.nn.functional.silu
    if case["ff"] == "dense":
        u = h @ p["up"].double().T
        return (gelu(u[:, :F]) * u[:, F:]) @ p["down"].double().T
    score = torch.softmax(h @ p["router"].double().T, -1)
    weight, chosen = score.topk(case["top"], -1)
    weight = weight / weight.sum(-1, keepdim=True)
    u = h @ p["shared_up"].double().T
    y = (silu(u[:, :2 * F]) * u[:, 2 * F:]) @ p["shared_down"].double().T * torch.sigmoid(h @ p["shared_gate"].double())[:, None]
    for e in range(case["experts"]):
        row, slot = torch.nonzero(chosen == e, as_tuple=True)
        if len(row):
            u = h[row] @ p["gate_up"][e].double().T
            y[row] += weight[row, slot][:, None] * ((silu(u[:, :F]) * u[:, F:]) @ p["expert_down"][e].double().T)
    return y


def exact_engine(case, seed):
    w = engine_weights(case, seed)
    plan = engine_plan(case, seed)
    out = [[None] * case["entries"] for _ in plan]
    for e in range(case["entries"]):
        ids = torch.tensor([t for step in plan for t in step[e]], device="cuda")
        pos = torch.arange(len(ids), device="cuda")
        x = w["embed"][ids].double()
        for p in w["layers"]:
            x = x + exact_mixer(case, p, rms(x, p["norm1"], EPS), pos)
            x = x + exact_ff(case, p, rms(x, p["norm2"], EPS))
        n = len(plan[0][e])
        rows = [slice(0, n) if case["kind"] == "score" else slice(n - 1, n)] + [slice(n + i, n + i + 1) for i in range(case["steps"])]
        for i, r in enumerate(rows):
            out[i][e] = rms(x[r], w["final"], EPS) @ w["head"].double().T
    return [torch.cat(o) for o in out]


# ---- what a measurement calls ----------------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] in ("decode", "prefill"):
        return prepare_decoder(case, seed)
    return prepare_product(case, seed) if case["kind"] == "product" else prepare_engine(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind in ("decode", "prefill"):
        return run_decoder(state)
    return run_product(state) if kind == "product" else run_engine(state)


def work(case):
    if case["kind"] in ("decode", "prefill"):
        return work_decoder(case)
    if case["kind"] == "product":
        t, k, n, es = case["tokens"], case["in_dim"], case["out_dim"], 2 if case["dtype"] == "bf16" else 4
        return {"bytes": (t * k + n * k) * es + t * n * 4, "flops": 2 * t * k * n}
    return work_engine(case)


def exact(case, seed):
    if case["kind"] in ("decode", "prefill"):
        return exact_decoder(case, seed)
    if case["kind"] == "product":
        a, w = product_inputs(case, seed)
        return a.double() @ w.double().T
    return exact_engine(case, seed)


def tolerance(case):
    """About four times the error against 64 bits that the paths show at their largest sizes."""
    if case["kind"] == "prefill":  # TF32 operands: ten bits of mantissa in every product of every layer
        return {"rel": 1.2e-2, "max": 0.15}
    if case["kind"] == "decode":  # fp32 sums, int8 rows as 24-bit fixed point: up to 6e-6
        return {"rel": 2.5e-5, "max": 2.5e-4}
    if case["kind"] == "product":  # operands are exact, sums are fp32: 4e-6 on the tensor cores' accumulators, 6e-7 in fp32
        return {"rel": 1.5e-5, "max": 1.5e-4} if case["dtype"] == "bf16" else {"rel": 3e-6, "max": 3e-5}
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 2e-4}
    # bf16 activations between the products; a router may turn over between experts that score alike
    if case["ff"] == "moe":
        return {"rel": 3e-2, "max": 0.9}
    return {"rel": 1e-2, "max": 0.15} if case["layers"] == 1 else {"rel": 3e-2, "max": 0.4}
