"""Performance cases of the batched decode step, through `Engine.step` as a serving or rollout loop calls it.

A case is one scheduler step of continuous batching (or a few in a row): decode rows over resident contexts of ragged
lengths, prompt chunks beside them or alone, or both. Shapes are those of the benchmark's workloads: the tiny CPU-runnable
decoder, the Llama-3-8B shape in Q4_K (whole) and in Q8_0, with LoRA adapters or over a quantised KV pool (cut to eight of its
32 layers: every layer costs the same), and the 20B-class mixture-of-experts shape with MXFP4 experts (cut to its first layers).
Weights are random (a model file is written once per machine and kept), prompts are uniform random token ids.

Fields of a case:
  model      key of MODELS                      adapters   LoRA adapters loaded (rows are spread over them by Zipf(1.1)), 0 = none
  kv         storage type of the KV pool        decode     decode rows of a step
  group      rows that share one prompt's KV    ctx_lo, ctx_hi   resident tokens of the rows, spread log-uniformly
  steps      decode steps in one pass           chunks     prompt chunks beside them: "n", or "n@p" after p resident tokens; a
  sampling   key of SAMPLING                               trailing "+" means that the prompt goes on, so nothing is sampled
  top        top log-probabilities asked for per sampled row
"""
import math
import os
import struct
import tempfile

import numpy as np

import retrograd_b200 as rb

SHAPE_8B = dict(arch="llama", d=4096, heads=32, kv_heads=8, ff=14336, vocab=128256)
MODELS = {
    "tiny_q8_0": dict(arch="llama", layers=2, d=256, heads=4, kv_heads=4, ff=688, vocab=4096, dtype="q8_0", seed=20261125),
    "8b_q4_k": dict(SHAPE_8B, layers=32, dtype="q4_k", seed=2),
    "8b_q4_k_8_layers": dict(SHAPE_8B, layers=8, dtype="q4_k", seed=2),
    "8b_q8_0_8_layers": dict(SHAPE_8B, layers=8, dtype="q8_0", seed=3),
    "moe_20b_mxfp4_4_layers": dict(arch="olmoe", layers=4, d=2880, heads=64, kv_heads=8, head_dim=64, ff=2880, vocab=201088, experts=32,
                                   experts_used=4, dtype="q8_0", expert_dtype="mxfp4", seed=5),
}
# n_ctx of an engine that holds a few cases' sequences at a time
CONTEXT = {"tiny_q8_0": 65536, "8b_q4_k": 400_000, "8b_q4_k_8_layers": 300_000, "8b_q8_0_8_layers": 400_000, "moe_20b_mxfp4_4_layers": 400_000}
# options of the sampled rows: greedy decoding; a chat server's truncated sampling; a rollout's temperature 1.0 over the likeliest tokens
SAMPLING = {
    "greedy": dict(top_k=1),
    "chat": dict(temperature=0.8, top_k=40, top_p=0.95, min_p=0.05),
    "rollout": dict(temperature=1.0, top_k=20),
}
N_BATCH, CHUNK, RANK, ALPHA = 2048, 512, 16, 32.0
WINDOW = 16     # passes decode at growing positions and go back to the first after this many


def _case(name, model, decode=0, ctx_lo=64, ctx_hi=64, chunks="", sampling="greedy", group=1, steps=1, adapters=0, kv="f16", top=0):
    return dict(name=name, model=model, decode=decode, ctx_lo=ctx_lo, ctx_hi=ctx_hi, chunks=chunks, sampling=sampling, group=group, steps=steps,
                adapters=adapters, kv=kv, top=top)


def listed():
    return [
        # the smallest call: one request of a tiny model, where launches and host work are everything
        _case("tiny_decode_1", "tiny_q8_0", decode=1, ctx_lo=100, ctx_hi=100, top=5),
        # one chat user of an 8B model: the weight stream at one token
        _case("chat_decode_1", "8b_q4_k", decode=1, ctx_lo=777, ctx_hi=777),
        # a lightly loaded server: four consecutive steps of eight users
        _case("serve_decode_8", "8b_q4_k", decode=8, ctx_lo=64, ctx_hi=2048, steps=4),
        # a medium load with a chat server's sampling options
        _case("serve_decode_30_chat", "8b_q4_k", decode=30, ctx_lo=64, ctx_hi=2048, sampling="chat"),
        # a full server between admissions: every slot decodes, contexts of all lengths
        _case("serve_decode_203", "8b_q4_k", decode=203, ctx_lo=64, ctx_hi=2048),
        # time to first token of one prompt, whole in one step
        _case("prompt_437", "8b_q4_k", chunks="437"),
        # the continuous-batching step under load: decode rows, full chunks at several depths, a ragged last chunk
        _case("serve_mixed_1781", "8b_q4_k", decode=128, ctx_lo=64, ctx_hi=1024, chunks="512+ 512@512+ 512@1024+ 117@512"),
        # a rollout batch: 40 prompts sampled in groups of eight that share the prompt's KV
        _case("rollout_decode_320", "8b_q8_0_8_layers", decode=320, group=8, ctx_lo=256, ctx_hi=1024, sampling="rollout"),
        # many adapters in one step: 96 decode rows over 16 adapters and a chunk of a new prompt
        _case("lora_decode_96", "8b_q4_k_8_layers", decode=96, ctx_lo=128, ctx_hi=1024, chunks="131", adapters=16),
        # long contexts over a quantised KV pool
        _case("kv_q8_0_decode_60", "8b_q4_k_8_layers", decode=60, ctx_lo=256, ctx_hi=4096, kv="q8_0"),
        # mixture of experts: a small decode batch (few tokens per expert), and a loaded mixed step
        _case("moe_decode_24", "moe_20b_mxfp4_4_layers", decode=24, ctx_lo=64, ctx_hi=2048, steps=2),
        _case("moe_mixed_1400", "moe_20b_mxfp4_4_layers", decode=256, ctx_lo=64, ctx_hi=512, chunks="512+ 512@512+ 120@200"),
    ]


def draw(rng):
    """One more case: any of the models, one to some hundred decode rows, up to three chunks of any length."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tiny", "dense", "dense", "dense", "rollout", "lora", "kv", "moe", "moe"])
    model = {"tiny": "tiny_q8_0", "dense": "8b_q4_k", "rollout": "8b_q8_0_8_layers", "lora": "8b_q4_k_8_layers", "kv": "8b_q4_k_8_layers",
             "moe": "moe_20b_mxfp4_4_layers"}[kind]
    most_rows = {"tiny": 12, "dense": 180, "rollout": 40, "lora": 120, "kv": 100, "moe": 300}[kind]
    decode = log_int(1, most_rows)
    ctx_hi = rng.choice([256, 700, 1024, 2048]) if kind != "tiny" else rng.choice([64, 160, 300])
    if decode > 80:
        ctx_hi = min(ctx_hi, 1024)
    group = 1
    if kind == "rollout":
        group, decode = 8, 8 * decode
    chunks = []
    if kind != "rollout" and rng.random() < 0.5:
        for _ in range(rng.randint(1, 3 if kind != "tiny" else 1)):
            n = log_int(9, CHUNK if kind != "tiny" else 100)
            chunks.append("%d%s%s" % (n, "@%d" % log_int(16, 1000) if kind != "tiny" and rng.random() < 0.5 else "", "+" if rng.random() < 0.5 else ""))
    if chunks and rng.random() < 0.25:
        decode = 0
        chunks[0] = chunks[0].rstrip("+")       # something is sampled in every pass
    sampling = "greedy"
    if decode >= 30 and rng.random() < 0.4:
        sampling = "chat" if kind != "rollout" else "rollout"
    c = _case("", model, decode=decode, ctx_lo=rng.choice([17, 64, 128]), ctx_hi=ctx_hi, chunks=" ".join(chunks), sampling=sampling, group=group,
              adapters=16 if kind == "lora" else 0, kv="q8_0" if kind == "kv" else "f16")
    del c["name"]
    return c


# ---- sizes that follow from a case

def _contexts(case):
    """Resident tokens of each prompt of the decode rows, spread evenly over the logarithm of the range."""
    lo, hi = math.log(case["ctx_lo"]), math.log(case["ctx_hi"])
    return [int(round(math.exp(lo + (hi - lo) * ((0.37 + 0.6180339887 * i) % 1.0)))) for i in range(-(-case["decode"] // case["group"]))]


def _chunks(case):
    """(tokens, resident tokens before them, whether the prompt ends with them)."""
    out = []
    for word in case["chunks"].split():
        n, _, at = word.rstrip("+").partition("@")
        out.append((int(n), int(at or 0), not word.endswith("+")))
    return out


def work(case):
    """Weights once per step as the file packs them, every context's K and V once, the new rows' K and V; two operations per
    weight and token, four per query element and context token."""
    sp = MODELS[case["model"]]
    bpw = {"q4_k": 144 / 256, "q8_0": 34 / 32, "mxfp4": 17 / 32}
    hd = sp.get("head_dim") or sp["d"] // sp["heads"]
    dq, dkv, d, ff = sp["heads"] * hd, sp["kv_heads"] * hd, sp["d"], sp["ff"]
    chunks, contexts = _chunks(case), _contexts(case)
    rows = case["decode"]
    tokens = rows + sum(n for n, _, _ in chunks)
    sampled = rows + sum(1 for c in chunks if c[2])
    attn_w = d * (dq + 2 * dkv) + dq * d
    if sp.get("experts"):
        used = min(sp["experts"], tokens * sp["experts_used"])
        layer_bytes = attn_w * bpw[sp["dtype"]] + used * 3 * d * ff * bpw[sp["expert_dtype"]] + 4 * d * sp["experts"]
        layer_w = attn_w + sp["experts_used"] * 3 * d * ff + d * sp["experts"]
    else:
        layer_bytes = (attn_w + 3 * d * ff) * bpw[sp["dtype"]]
        layer_w = attn_w + 3 * d * ff
    if case["adapters"]:
        factors = RANK * ((d + dq) + 2 * (d + dkv) + (dq + d) + 3 * (d + ff))
        layer_bytes += min(case["adapters"], rows + len(chunks)) * factors * 4
        layer_w += factors
    kv_row = 2 * dkv * {"f16": 2.0, "q8_0": 34 / 32}[case["kv"]]
    resident = sum(contexts) + sum(at for _, at, _ in chunks)
    pairs = sum(contexts[i // case["group"]] + 1 for i in range(rows)) + sum(n * at + n * (n + 1) // 2 for n, at, _ in chunks)
    head = d * sp["vocab"]
    nbytes = sp["layers"] * (layer_bytes + (resident + tokens) * kv_row) + head * bpw[sp["dtype"]] + tokens * d * bpw[sp["dtype"]]
    flops = sp["layers"] * (2 * tokens * layer_w + 4 * pairs * dq) + 2 * sampled * head
    return {"bytes": case["steps"] * nbytes, "flops": case["steps"] * flops}


def tolerance(case):
    """K and V are rounded to 16 bits (or quantised) when they are stored, so any difference in the last bits of an f32 sum comes
    back as a difference of one storage step in some of them: about 1e-3 of a log-probability. A sampled row whose draw falls
    that close to the border of two tokens takes the other one, with a log-probability of its own; so does an arg-max of two
    nearly equal logits, and an expert choice between two nearly equal probabilities changes a token's whole row."""
    if case["model"].startswith("moe") or case["sampling"] != "greedy":
        return {"rel": 1e-2, "max": 0.5, "differ": 0.01}
    return {"rel": 5e-3 if case["kv"] != "f16" else 1e-3, "differ": 0.01}


# ---- model and adapter files, engines

def _folder():
    base = "/dev/shm" if os.access("/dev/shm", os.W_OK) else tempfile.gettempdir()
    path = os.path.join(base, "retrograd_b200_cases")
    os.makedirs(path, exist_ok=True)
    if not os.access(path, os.W_OK):        # another user's: keep files of our own
        path = "%s_%d" % (path, os.getuid())
        os.makedirs(path, exist_ok=True)
    return path


def _file(name, write):
    """A file that is written once: under another name first, so that nobody sees half of it."""
    path = os.path.join(_folder(), name)
    if not os.path.exists(path):
        part = "%s.%d" % (path, os.getpid())
        write(part)
        os.replace(part, path)
    return path


def _write_adapter(path, sp, seed):
    """A LoRA adapter GGUF: A and B ~ N(0, 0.02) on the seven projections of every layer."""
    rng = np.random.default_rng(seed)
    hd = sp.get("head_dim") or sp["d"] // sp["heads"]
    d, dq, dkv, ff = sp["d"], sp["heads"] * hd, sp["kv_heads"] * hd, sp["ff"]
    shapes = {"attn_q": (d, dq), "attn_k": (d, dkv), "attn_v": (d, dkv), "attn_output": (dq, d), "ffn_gate": (d, ff), "ffn_up": (d, ff), "ffn_down": (ff, d)}
    tensors = []
    for layer in range(sp["layers"]):
        for target, (n_in, n_out) in shapes.items():
            tensors.append(("blk.%d.%s.weight.lora_a" % (layer, target), (n_in, RANK)))
            tensors.append(("blk.%d.%s.weight.lora_b" % (layer, target), (RANK, n_out)))

    def text(s):
        return struct.pack("<Q", len(s)) + s.encode()

    kv = b"".join(text(k) + struct.pack("<I", 8) + text(v) for k, v in
                  (("general.architecture", "llama"), ("general.type", "adapter"), ("adapter.type", "lora")))
    kv += text("adapter.lora.alpha") + struct.pack("<If", 6, ALPHA)
    head, at = b"GGUF" + struct.pack("<IQQ", 3, len(tensors), 4) + kv, 0
    for name, ne in tensors:
        head += text(name) + struct.pack("<IQQIQ", 2, ne[0], ne[1], 0, at)
        at += ne[0] * ne[1] * 4         # a multiple of the 32-byte alignment: RANK is 16
    with open(path, "wb") as f:
        f.write(head + b"\0" * (-len(head) % 32))
        for _, ne in tensors:
            (rng.standard_normal(ne[0] * ne[1], dtype=np.float32) * np.float32(0.02)).tofile(f)


class Server:
    """An engine with its adapters, and the slots and request ids that are free in it."""

    def __init__(self, model, adapters, kv):
        sp = MODELS[model]
        path = _file(model + ".gguf", lambda p: rb.synth_gguf(p, **sp))
        n_slots = 64 if model.startswith("tiny") else 1024
        self.engine = rb.Engine(path, rb.EngineConfig(n_ctx=CONTEXT[model], n_seq_max=n_slots, n_batch=N_BATCH, n_ubatch=N_BATCH,
                                                      kv_dtype={"f16": rb.KV_DTYPE_F16, "q8_0": rb.KV_DTYPE_Q8_0}[kv]))
        self.adapters = [self.engine.adapter_load(_file("%s_adapter_%d.gguf" % (model, a), lambda p, a=a: _write_adapter(p, sp, 7000 + a)))
                         for a in range(adapters)]
        self.free = list(range(n_slots))[::-1]
        self.next_request = 0


_servers = {}       # a program keeps its engine from one batch of requests to the next


def _server(case):
    key = (case["model"], case["adapters"], case["kv"])
    if key not in _servers:
        _servers[key] = Server(*key)
    return _servers[key]


class State:
    """The requests of a case, resident in the engine; they leave it with this object."""

    def __init__(self, case, seed):
        self.slots, self.requests, self.at = [], [], 0
        self.case, self.server = case, _server(case)
        self.engine = self.server.engine
        self.out = rb.StepOutput(0, case["top"])
        rng = np.random.default_rng(seed)
        vocab = MODELS[case["model"]]["vocab"]
        weights = 1.0 / np.arange(1, len(self.server.adapters) + 1) ** 1.1

        def adapter():
            return int(rng.choice(self.server.adapters, p=weights / weights.sum())) if self.server.adapters else 0

        def tokens(n):
            return rng.integers(3, vocab, n, dtype=np.int32)

        fill, share = [], []        # contexts to decode first, and whose they become
        self.decode = []            # (request, slot, tokens of the next positions, position, sampling, adapter)
        contexts = _contexts(case)
        for i in range(case["decode"]):
            slot, length = self.slot(), contexts[i // case["group"]]
            if i % case["group"] == 0:
                leader, its = slot, adapter()
                fill.append((slot, tokens(length), its))
            else:
                share.append((leader, slot))
            self.decode.append((self.request(), slot, tokens(WINDOW), length, self.sampling(seed, i), its))
        self.chunks = []            # (request, slot, tokens, position, whether to sample, sampling, adapter)
        for i, (n, at, final) in enumerate(_chunks(case)):
            slot, its = self.slot(), adapter()
            if at:
                fill.append((slot, tokens(at), its))
            self.chunks.append((self.request(), slot, tokens(n), at, final, self.sampling(seed, case["decode"] + i), its))
        self.prefill(fill)
        for leader, slot in share:
            self.engine.seq_cp(leader, slot)

    def slot(self):
        self.slots.append(self.server.free.pop())
        return self.slots[-1]

    def request(self):
        self.server.next_request += 1
        self.requests.append(self.server.next_request)
        return self.requests[-1]

    def sampling(self, seed, i):
        return rb.SamplingParamsV2(seed=(seed * 1009 + i) % 2**31, **SAMPLING[self.case["sampling"]])

    def prefill(self, pending):
        """Chunked, as a scheduler does it."""
        out, pos = rb.StepOutput(), {slot: 0 for slot, _, _ in pending}
        while pending:
            rows, left = [], N_BATCH
            for slot, toks, its in pending:
                n = min(CHUNK, left, len(toks) - pos[slot])
                if n > 0:
                    rows.append(rb.StepRow(-1, slot, toks[pos[slot] : pos[slot] + n], pos[slot], adapter=its))
                    pos[slot] += n
                    left -= n
                if not left:
                    break
            self.engine.step(rows, out)
            pending = [p for p in pending if pos[p[0]] < len(p[1])]

    def __del__(self):
        for request in self.requests:
            self.engine.request_free(request)
        for slot in self.slots:
            self.engine.seq_rm(slot)
        self.server.free.extend(self.slots)


def prepare(case, seed):
    return State(case, seed)


def run(state):
    engine, out, case = state.engine, state.out, state.case
    results = []
    for _ in range(case["steps"]):
        if state.at == WINDOW:          # the generation is taken back to where it began
            for _, slot, _, pos, _, _ in state.decode:
                engine.seq_rm(slot, pos)
            state.at = 0
        k, rows = state.at, []
        state.at += 1
        for request, slot, tokens, pos, sampling, adapter in state.decode:
            rows.append(rb.StepRow(request, slot, [int(tokens[k])], pos + k, True, sampling, case["top"], case["sampling"] != "greedy", adapter))
        for request, slot, tokens, pos, final, sampling, adapter in state.chunks:
            rows.append(rb.StepRow(request, slot, tokens, pos, final, sampling, case["top"] if final else 0, final and case["sampling"] != "greedy", adapter))
        engine.step(rows, out)
        got = out.rows()
        results.append({
            "rows": np.array([(r.token, r.n_top, r.forced, r.sampled) for r in got], dtype=np.int32),
            "logprobs": np.array([(r.logprob, r.sampled_logprob) for r in got], dtype=np.float32),
            "top": [out.top(i) for i, r in enumerate(got) if r.n_top],
        })
        for _, slot, _, pos, _, _, _ in state.chunks:       # the prompt's request is given up again
            engine.seq_rm(slot, pos if pos else -1)
    return {"rows": np.concatenate([r["rows"] for r in results]), "logprobs": np.concatenate([r["logprobs"] for r in results]),
            "top": [t for r in results for t in r["top"]]}
