"""Workloads whose speed is tracked: fine-tuning steps and cached generation as a program on this framework runs them.

Every case goes through the entry points that such a program calls: ``TrainingLoop`` for (Q)LoRA fine-tuning of packed documents,
``Generator`` for prompts and for decoding on the paged cache. Models are the presets of ``models/config.py`` with random weights;
the mixture of experts keeps 8 of its 48 layers, as ``bench/moe_serve.py --layers 8`` does, so that several copies fit one card.

A case's ``kind`` is ``train`` (one optimiser step), ``prefill`` (prompts to the logits of their last tokens) or ``decode``
(a few single-token steps of a batch with cached context)."""
import math

import torch

from pmetal_b200.core.config import LoraConfig, TrainingConfig
from pmetal_b200.data.dataloader import synthetic_documents
from pmetal_b200.data.packing import PackerConfig, SequencePacker, collate_packs
from pmetal_b200.lora import apply_lora
from pmetal_b200.lora.qlora import quantize_base
from pmetal_b200.models.config import preset
from pmetal_b200.models.decoder import DecoderLM
from pmetal_b200.models.generation import Generator
from pmetal_b200.models.sampling import Sampler, SamplingParams
from pmetal_b200.parallel.ep import shard_experts
from pmetal_b200.trainer.loop import TrainingLoop

DENSE, LARGE, MOE = "qwen3-0.6b", "qwen3-4b", "qwen3-30b-a3b"
MOE_LAYERS = 8
RANK, ALPHA = 16, 32.0
TARGETS = ["q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj"]
LR, WARMUP, TOTAL_STEPS, DECAY, CLIP = 2e-4, 100, 10_000, 0.01, 1.0
STEPS = 4           # decoded tokens of one pass


def _train(name, packs, pack_len, model=DENSE, quant="none", graph=True):
    return {"name": name, "kind": "train", "model": model, "packs": packs, "pack_len": pack_len, "quant": quant, "graph": graph}


def _prefill(name, seqs, tokens, model=DENSE):
    return {"name": name, "kind": "prefill", "model": model, "seqs": seqs, "tokens": tokens}


def _decode(name, batch, context, model=DENSE, kv="bf16"):
    return {"name": name, "kind": "decode", "model": model, "batch": batch, "context": context, "kv": kv}


def listed():
    return [
        # supervised fine-tuning at the size of the headline benchmark: 4 packs of 4096 tokens, the step replayed from a graph
        _train("lora 4x4096", 4, 4096),
        # the small batch that the published single-machine figures are quoted for: 4 x 512
        _train("lora 4x512", 4, 512),
        # a short ragged stream stepped without a graph, which is what ``train`` does by default
        _train("lora 1x1537 eager", 1, 1537, graph=False),
        # QLoRA of a larger model: packed NF4 base with double-quantised scales, 2 packs of 4096
        _train("qlora 4b 2x4096", 2, 4096, model=LARGE, quant="nf4"),
        # first answer to a short chat message
        _prefill("prefill 1x37", 1, 37),
        # several requests of ordinary, unequal lengths together
        _prefill("prefill 6x3001", 6, 3001),
        # one long document
        _prefill("prefill 1x12000", 1, 12000),
        # one user waiting for tokens
        _decode("decode 1", 1, 500),
        # a server with some load; a rollout group
        _decode("decode 16", 16, 700),
        # a loaded server
        _decode("decode 64", 64, 450),
        # long contexts on the 8-bit cache
        _decode("decode 8 int8", 8, 6000, kv="int8"),
        # mixture of experts under load
        _decode("decode moe 64", 64, 300, model=MOE),
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["lora", "lora", "lora", "qlora", "prefill", "prefill", "prefill", "decode", "decode", "decode", "int8", "moe"])
    if kind == "lora":
        case = _train("", rng.randint(1, 4), _spread(rng, 300, 4096), graph=rng.random() < 0.7)
    elif kind == "qlora":
        case = _train("", rng.randint(1, 2), _spread(rng, 500, 4096), model=LARGE, quant="nf4")
    elif kind == "prefill":
        seqs = _spread(rng, 1, 12)
        case = _prefill("", seqs, _spread(rng, 16 * seqs, 12000))
    elif kind == "moe":
        case = _decode("", _spread(rng, 4, 64), _spread(rng, 20, 400), model=MOE)
    else:
        batch = _spread(rng, 1, 64)
        case = _decode("", batch, _spread(rng, 30, min(6000, 48_000 // batch)), kv="int8" if kind == "int8" else "bf16")
    del case["name"]
    return case


# ------------------------------------------------------------------ what both sides start from
def _config(case):
    cfg = preset(case["model"])
    if case["model"] == MOE:
        cfg.num_hidden_layers = MOE_LAYERS
    return cfg


def _weights(cfg, seed):
    """bf16 tensors by checkpoint name: matrices N(0, 0.64 / sqrt(input width)), which is the usual 0.02 at a width of 1024, norm
    weights near one, routers that prefer few experts clearly as trained ones do. Expert stacks are returned whole as well."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    H, d, V = cfg.hidden_size, cfg.head_dim, cfg.vocab_size


    def mat(*shape, gain=0.64):
        return torch.empty(*shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, gain * shape[-1] ** -0.5, generator=g)

    def norm(n):
        return (1.0 + 0.1 * torch.randn(n, device="cuda", generator=g)).to(torch.bfloat16)
    sd, stacks = {"model.embed_tokens.weight": mat(V, H), "model.norm.weight": norm(H)}, {}
    if not cfg.tie_word_embeddings:
        sd["lm_head.weight"] = mat(V, H)
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        sd[p + "input_layernorm.weight"], sd[p + "post_attention_layernorm.weight"] = norm(H), norm(H)
        sd[p + "self_attn.q_norm.weight"], sd[p + "self_attn.k_norm.weight"] = norm(d), norm(d)
        for n, rows, cols in (("q", cfg.q_size, H), ("k", cfg.kv_size, H), ("v", cfg.kv_size, H), ("o", H, cfg.q_size)):
            sd[p + f"self_attn.{n}_proj.weight"] = mat(rows, cols)
        if cfg.is_moe_layer(i):
            E, I = cfg.num_experts, cfg.moe_intermediate_size
            sd[p + "mlp.gate.weight"] = mat(E, H, gain=3.0)
            gu, dn = mat(E, 2 * I, H), mat(E, H, I)
            stacks[i] = (gu, dn)
            for e in range(E):
                sd[p + f"mlp.experts.{e}.gate_proj.weight"], sd[p + f"mlp.experts.{e}.up_proj.weight"] = gu[e, :I], gu[e, I:]
                sd[p + f"mlp.experts.{e}.down_proj.weight"] = dn[e]
        else:
            I = cfg.intermediate_size
            sd[p + "mlp.gate_proj.weight"], sd[p + "mlp.up_proj.weight"] = mat(I, H), mat(I, H)
            sd[p + "mlp.down_proj.weight"] = mat(H, I)
    return sd, stacks


def _groups(cfg):
    """Projection groups of a layer: (name, input width, rows of each projection)."""
    H, I = cfg.hidden_size, cfg.intermediate_size
    return [("self_attn.qkv_proj", H, (cfg.q_size, cfg.kv_size, cfg.kv_size)), ("self_attn.o_proj", cfg.q_size, (H,)),
            ("mlp.gate_up_proj", H, (I, I)), ("mlp.down_proj", I, (H,))]


def _adapters(cfg, seed):
    """fp32 LoRA factors of an adapter that has trained for a while, in the order of the model's parameters."""
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    out = {}
    for i in range(cfg.num_hidden_layers):
        for name, width, rows in _groups(cfg):
            a = torch.empty(len(rows) * RANK, width, device="cuda")
            out[f"layers.{i}.{name}.lora_a"] = a.uniform_(-1, 1, generator=g).mul_(math.sqrt(3.0 / width))
            out[f"layers.{i}.{name}.lora_b"] = torch.randn(sum(rows), RANK, device="cuda", generator=g) * 0.01
    return out


def _batch(case, cfg, seed):
    n, length = case["packs"], case["pack_len"]
    longest = min(2048, length)
    docs = synthetic_documents(int(n * length / ((64 + longest) / 2) * 1.3) + 8, 64, longest, cfg.vocab_size, seed)
    packs = SequencePacker(PackerConfig(max_length=length, max_seq_length=length)).pack(docs)
    packs.sort(key=lambda p: -p.total_tokens())
    return collate_packs(packs[:n], length)


def _lengths(case):
    """Unequal lengths around the mean that add up to the case's tokens (prompts) or average its context (decode)."""
    n = case.get("seqs") or case["batch"]
    total = case["tokens"] if case["kind"] == "prefill" else case["batch"] * case["context"]
    lens = [max(1, int(total / n * (0.5 + (i * 7 % n + 0.5) / n))) for i in range(n)]
    lens[0] += max(total - sum(lens), 1 - lens[0])
    return lens


def _tokens(case, cfg, seed):
    g = torch.Generator().manual_seed(seed + 3)
    extra = STEPS if case["kind"] == "decode" else 0
    return [torch.randint(0, cfg.vocab_size, (n + extra,), generator=g).tolist() for n in _lengths(case)]


# ------------------------------------------------------------------ what a program has in hand
def _prepare_train(case, seed):
    cfg = _config(case)
    model = DecoderLM(cfg, torch.bfloat16, "cuda")
    model.load_hf_state_dict(_weights(cfg, seed)[0])
    for p in model.parameters():
        p.requires_grad_(False)
    if case["quant"] != "none":
        quantize_base(model, case["quant"], 64, True)
    apply_lora(model, LoraConfig(r=RANK, alpha=ALPHA, target_modules=TARGETS), seed=seed)
    values = _adapters(cfg, seed)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name in values:
                p.copy_(values[name])
    model.prepare_for_training()
    loop = TrainingLoop(model, TrainingConfig(learning_rate=LR, gradient_accumulation_steps=1, warmup_steps=WARMUP, max_grad_norm=CLIP,
                                              weight_decay=DECAY, lr_scheduler="cosine"), total_steps=TOTAL_STEPS)
    batch = _batch(case, cfg, seed).pin()
    # the first step runs at a learning rate of zero (warm-up): moments exist, the weights are as they were
    if case["graph"]:
        loop.enable_cuda_graph(batch)
    else:
        loop.train_step(batch.to("cuda"))
    return {"kind": "train", "loop": loop, "batch": batch, "graph": case["graph"]}


def _served(case, seed):
    cfg = _config(case)
    model = DecoderLM(cfg, torch.bfloat16, "cuda").eval()
    model.load_hf_state_dict(_weights(cfg, seed)[0])
    for p in model.parameters():
        p.requires_grad_(False)
    for layer in model.layers:
        if hasattr(layer.mlp, "router"):
            shard_experts(layer.mlp, None, max_tokens=2048)
            for name in ("gate_up", "down"):        # the engine holds them now
                setattr(layer.mlp, name, torch.nn.Parameter(torch.empty(0, dtype=torch.bfloat16, device="cuda"), requires_grad=False))
    return model, cfg


def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    model, cfg = _served(case, seed)
    prompts = _tokens(case, cfg, seed)
    blocks = sum(-(-len(p) // 64) + 1 for p in prompts) + 16
    quant = "int8" if case.get("kv") == "int8" else None
    gen = Generator(model, cache=model.new_cache(blocks, quant=quant))
    state = {"kind": case["kind"], "gen": gen, "prompts": prompts, "sampler": Sampler(SamplingParams.greedy(), "cuda")}
    if case["kind"] == "decode":
        seqs = [gen.new_seq() for _ in prompts]
        gen.prefill(seqs, [p[:-STEPS] for p in prompts])
        state["seqs"] = seqs
        state["next"] = [torch.tensor([p[len(p) - STEPS + k] for p in prompts]) for k in range(STEPS)]
    return state


def run(state):
    if state["kind"] == "train":
        loop, batch = state["loop"], state["batch"]
        loss, gnorm = loop.train_step_graphed(batch) if state["graph"] else loop.train_step(batch.to("cuda"))
        return {"loss": float(loss), "grad_norm": float(gnorm), "grad": loop.opt.flat_g, "param": loop.opt.flat_p}
    gen = state["gen"]
    if state["kind"] == "prefill":
        seqs = [gen.new_seq() for _ in state["prompts"]]
        logits = gen.prefill(seqs, state["prompts"])
        state["sampler"].sample(logits).tolist()                # the first token reaches the host
        for s in seqs:
            gen.cache.free_sequence(s)
        return logits
    out, seqs = [], state["seqs"]
    before = [gen.cache.length(s) for s in seqs]
    for ids in state["next"]:           # a recorded continuation; every step's choice is read back as a server does
        logits = gen.decode_step(seqs, ids)
        state["sampler"].sample(logits).tolist()
        out.append(logits)
    for s, n in zip(seqs, before):
        gen.cache.truncate(s, n)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _dense_weights(cfg):
    """(entries of the projections of all layers, entries a token meets)."""
    attn = cfg.hidden_size * (2 * cfg.q_size + 2 * cfg.kv_size)
    if cfg.num_experts:
        ex = 3 * cfg.hidden_size * cfg.moe_intermediate_size
        router = cfg.num_experts * cfg.hidden_size
        return (cfg.num_hidden_layers * (attn + router + cfg.num_experts * ex),
                cfg.num_hidden_layers * (attn + router + cfg.num_experts_per_tok * ex))
    n = cfg.num_hidden_layers * (attn + 3 * cfg.hidden_size * cfg.intermediate_size)
    return n, n


def work(case):
    cfg = _config(case)
    stored, met = _dense_weights(cfg)
    V, H, L, hq, d = cfg.vocab_size, cfg.hidden_size, cfg.num_hidden_layers, cfg.num_attention_heads, cfg.head_dim
    if case["kind"] == "train":
        T, longest = case["packs"] * case["pack_len"], min(2048, case["pack_len"])
        mean, square = (64 + longest) / 2, (64 * 64 + 64 * longest + longest * longest) / 3
        lora = L * RANK * sum(w * len(r) + sum(r) for _, w, r in _groups(cfg))
        # forward and input gradient of the frozen projections and the head, three products per adapter, two and five of attention
        flops = 4 * T * (met + V * H) + 6 * T * lora + 7 * L * hq * d * T * square / mean
        size = 0.5 + 1 / 64 if case["quant"] == "nf4" else 2
        return {"bytes": stored * size + V * H * 2 + lora * 4 * 8, "flops": flops}
    lens = _lengths(case)
    kv = 2 * L * cfg.kv_size * ((1 + 4 / 64) if case.get("kv") == "int8" else 2)
    if case["kind"] == "prefill":
        T = sum(lens)
        flops = 2 * T * met + 2 * len(lens) * V * H + 2 * L * hq * d * sum(n * n for n in lens)
        return {"bytes": 2 * (stored + V * H) + T * kv, "flops": flops}
    n = len(lens)
    read = stored
    if cfg.num_experts:          # the experts that a batch of this size is expected to reach
        share = 1 - (1 - cfg.num_experts_per_tok / cfg.num_experts) ** n
        read = (stored - L * cfg.num_experts * 3 * H * cfg.moe_intermediate_size * (1 - share))
    step_bytes = 2 * (read + V * H) + sum(lens) * kv + 2 * n * V
    step_flops = 2 * n * (met + V * H) + 4 * L * hq * d * sum(lens)
    return {"bytes": STEPS * step_bytes, "flops": STEPS * step_flops}


def tolerance(case):
    return {"rel": 0.03}


# ------------------------------------------------------------------ the same in 64 bits
NF4 = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334,
       -0.09105003625154495, 0.0, 0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224,
       0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0]


def _nf4(w):
    """What a weight stands for once it is stored as NF4 codes in blocks of 64 with 8-bit block maxima."""
    bins = torch.tensor(NF4, dtype=torch.float32, device=w.device)
    x = w.float().reshape(-1, 64)
    top = x.abs().amax(1).clamp_min(1e-10)
    codes = torch.bucketize((x / top[:, None]).clamp(-1, 1), (bins[1:] + bins[:-1]) / 2, right=True)
    lo = float(top.min())
    step = (float(top.max()) - lo) / 255.0
    top = torch.round((top - lo) / step).clamp(0, 255).double() * step + lo
    return (bins.double()[codes] * top[:, None]).reshape(w.shape)


def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rotate(x, cos, sin):
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, spans, rows):
    """Causal attention within the spans of a packed stream, ``rows`` query rows at a time. q [T, hq, d], k / v [T, hkv, d]."""
    rep, out = q.shape[1] // k.shape[1], []
    for s, e in spans:
        kk, vv = (t[s:e].transpose(0, 1).repeat_interleave(rep, 0) for t in (k, v))
        for a in range(s, e, rows):
            b = min(e, a + rows)
            sc = q[a:b].transpose(0, 1) @ kk[:, :b - s].transpose(1, 2) * q.shape[2] ** -0.5
            see = torch.arange(b - s, device=q.device)[None] <= torch.arange(a - s, b - s, device=q.device)[:, None]
            out.append((sc.masked_fill(~see, float("-inf")).softmax(-1) @ vv[:, :b - s]).transpose(0, 1))
    return torch.cat(out)


class _Exact:
    """The decoder in 64 bits on a packed stream."""

    def __init__(self, case, seed, positions, spans, rows=1 << 30):
        self.cfg = _config(case)
        self.sd, self.stacks = _weights(self.cfg, seed)
        self.quant = case.get("quant") == "nf4"
        self.spans, self.rows = spans, rows
        half = self.cfg.head_dim // 2
        freq = self.cfg.rope_theta ** (-torch.arange(half, dtype=torch.float64, device="cuda") / half)
        ang = positions.double()[:, None] * freq[None]
        self.cos, self.sin = ang.cos()[:, None], ang.sin()[:, None]

    def stacked(self, p, names):
        """Weight of a row-stacked group in 64 bits (quantised as one tensor where the base is)."""
        w = torch.cat([self.sd[p + n + ".weight"] for n in names]) if len(names) > 1 else self.sd[p + names[0] + ".weight"]
        return _nf4(w) if self.quant else w.double()

    def project(self, x, w, lora, rows):
        y = x @ w.t()
        if lora is None:
            return y
        a, b = lora
        t, parts, at = x @ a.t() * (ALPHA / RANK), [], 0
        for i, n in enumerate(rows):
            parts.append(t[:, i * RANK:(i + 1) * RANK] @ b[at:at + n].t())
            at += n
        return y + torch.cat(parts, -1)

    def layer(self, i, x, *lora):
        cfg, p = self.cfg, f"model.layers.{i}."
        pair = (lambda k: (lora[2 * k], lora[2 * k + 1])) if lora else (lambda k: None)
        g = [rows for _, _, rows in _groups(cfg)]
        T, hq, hkv, d, eps = x.shape[0], cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.rms_norm_eps
        h = _rms(x, self.sd[p + "input_layernorm.weight"], eps)
        qkv = self.project(h, self.stacked(p + "self_attn.", ["q_proj", "k_proj", "v_proj"]), pair(0), g[0]).view(T, -1, d)
        q, k, v = qkv.split([hq, hkv, hkv], 1)
        q = _rotate(_rms(q, self.sd[p + "self_attn.q_norm.weight"], eps), self.cos, self.sin)
        k = _rotate(_rms(k, self.sd[p + "self_attn.k_norm.weight"], eps), self.cos, self.sin)
        o = _attend(q, k, v, self.spans, self.rows).reshape(T, hq * d)
        x = x + self.project(o, self.stacked(p + "self_attn.", ["o_proj"]), pair(1), g[1])
        h = _rms(x, self.sd[p + "post_attention_layernorm.weight"], eps)
        if i in self.stacks:
            return x + self.experts(h, i)
        gate, up = self.project(h, self.stacked(p + "mlp.", ["gate_proj", "up_proj"]), pair(2), g[2]).chunk(2, -1)
        return x + self.project(torch.nn.functional.silu(gate) * up, self.stacked(p + "mlp.", ["down_proj"]), pair(3), g[3])

    def experts(self, h, i):
        cfg = self.cfg
        prob = (h @ self.sd[f"model.layers.{i}.mlp.gate.weight"].double().t()).softmax(-1)
        w, idx = prob.topk(cfg.num_experts_per_tok, -1)
        w = w / (w.sum(-1, keepdim=True) + 1e-8)
        gu, dn = self.stacks[i]
        out = torch.zeros_like(h)
        for e in range(cfg.num_experts):
            tok, slot = (idx == e).nonzero(as_tuple=True)
            if len(tok):
                gate, up = (h[tok] @ gu[e].double().t()).chunk(2, -1)
                out.index_add_(0, tok, (torch.nn.functional.silu(gate) * up) @ dn[e].double().t() * w[tok, slot, None])
        return out

    def hidden(self, ids, lora=None):
        from torch.utils.checkpoint import checkpoint
        x = self.sd["model.embed_tokens.weight"][ids].double()
        if lora is not None:
            x.requires_grad_(True)
        for i in range(self.cfg.num_hidden_layers):
            mine = lora[8 * i:8 * i + 8] if lora is not None else ()
            x = checkpoint(self.layer, i, x, *mine, use_reentrant=False) if lora is not None else self.layer(i, x)
        return x

    def head(self, x):
        w = self.sd.get("lm_head.weight", self.sd["model.embed_tokens.weight"])
        return _rms(x, self.sd["model.norm.weight"], self.cfg.rms_norm_eps) @ w.double().t()


def _exact_train(case, seed):
    from torch.utils.checkpoint import checkpoint
    cfg = _config(case)
    b = _batch(case, cfg, seed).to("cuda")
    cu = b.cu_seqlens.tolist()
    m = _Exact(case, seed, b.position_ids, list(zip(cu[:-1], cu[1:])))
    values = _adapters(cfg, seed)
    lora = [t.double().requires_grad_(True) for t in values.values()]
    x = m.hidden(b.input_ids, lora)
    target = torch.full_like(b.labels, -100)
    target[:-1] = b.labels[1:]
    n = int((target != -100).sum())

    def part(h, t):
        return torch.nn.functional.cross_entropy(m.head(h), t, ignore_index=-100, reduction="sum")
    loss = sum(checkpoint(part, x[s:s + 2048], target[s:s + 2048], use_reentrant=False) for s in range(0, x.shape[0], 2048)) / n
    loss.backward()

    def flat(ts):        # every tensor starts on a multiple of 1024 values
        return torch.cat([torch.nn.functional.pad(t.reshape(-1), (0, -t.numel() % 1024)) for t in ts])
    grad, param = flat([t.grad for t in lora]), flat([t.detach() for t in lora])
    norm = float(grad.norm())
    # moments of two steps on the same batch, bias-corrected: the (clipped) gradient and its square
    g, lr = grad * min(1.0, CLIP / (norm + 1e-6)), LR / WARMUP
    param = param - lr * g / (g.abs() + 1e-8)
    return {"loss": float(loss.detach()), "grad_norm": norm, "grad": grad, "param": param * (1 - lr * DECAY)}


@torch.no_grad()
def _exact_served(case, seed):
    tokens = _tokens(case, _config(case), seed)
    lens = [len(t) for t in tokens]
    ends = [sum(lens[:i + 1]) for i in range(len(lens))]
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    m = _Exact(case, seed, pos, [(e - n, e) for e, n in zip(ends, lens)], rows=1024)
    x = m.hidden(torch.tensor([t for ts in tokens for t in ts], device="cuda"))
    if case["kind"] == "prefill":
        return m.head(x[[e - 1 for e in ends]])
    return [m.head(x[[e - STEPS + k for e in ends]]) for k in range(STEPS)]


def exact(case, seed):
    return _exact_train(case, seed) if case["kind"] == "train" else _exact_served(case, seed)
