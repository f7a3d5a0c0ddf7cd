"""What a user has this framework do, as cases that can be timed and checked: training steps of the GPT (forward, reverse, Muon and
AdamW), its evaluation losses, and serving (a prompt, then token by token) of the GPT and of the decoders that list their layers.

`listed()` names cases over the range of sizes, `draw(rng)` gives others of the same ranges.  `prepare` builds what a program holds
before the call, `run` makes one pass through the public entry points, `exact` gives the results in 64 bits from plain torch."""
import math

import numpy as np
import torch

import femtochat_b200 as fb

# ---- models: the sizes of the benchmark, of its small configuration and of the introductory example -----------------------------------
GPTS = {
    "tiny": dict(sequence_len=4, max_document_tokens=64, vocab_size=16, n_layer=2, n_head=2, n_kv_head=1, n_embed=32, window_pattern="L"),
    "small": dict(max_document_tokens=512, vocab_size=4096, n_layer=4, n_head=4, n_kv_head=2, n_embed=512, window_pattern="SL"),
    "d12": dict(max_document_tokens=8192, vocab_size=65536, n_layer=12, n_head=6, n_kv_head=6, n_embed=768, window_pattern="L"),
    "d20": dict(max_document_tokens=8192, vocab_size=65536, n_layer=20, n_head=10, n_kv_head=5, n_embed=1280, window_pattern="SSSL"),
}
# short window and document mask as the benchmark sets them (0, False: the reference's defaults)
OPTIONS = {"tiny": (0, False), "small": (128, True), "d12": (0, False), "d20": (1024, True)}
DECODERS = {
    "d20": dict(width=1280, n_layer=20, ff=3456, heads=10, kv_heads=5, q_rank=768, kv_rank=512, vocab=65536),
    "w2560": dict(width=2560, n_layer=12, ff=6912, heads=20, kv_heads=10, q_rank=1536, kv_rank=512, vocab=65536),
}
VIROLORN = ("lightning", "channel_delta", "channel_delta", "latent_attention")
LR = dict(unembedding_lr=0.004, embedding_lr=0.2, matrix_lr=0.02, weight_decay=0.01, scalar_lr=0.5, smear_lr=0.2)   # the optimiser's defaults
STEP = dict(eta=1.0, mu=0.95, lam=0.01)
TRAINED = 100              # updates that the optimiser's moments have seen


def train(name, model, dtype, B, T):
    return dict(name=name, kind="train", model=model, dtype=dtype, B=B, T=T)


def serve(name, family, model, B, prompt, new):
    return dict(name=name, kind="serve", family=family, model=model, B=B, prompt=prompt, new=new)


def listed():
    return [
        # the introductory example's model, in the default type: a step is a few hundred launches of a few microseconds
        train("train tiny f32 2x4", "tiny", "float32", 2, 4),
        # the default type at a size that a test or a debugging session trains, a ragged length
        train("train small f32 3x200", "small", "float32", 3, 200),
        # a small model trained in bf16
        train("train d12 bf16 4x2048", "d12", "bfloat16", 4, 2048),
        # the benchmark's model at a quarter of its batch: documents, a short window
        train("train d20 bf16 8x2048", "d20", "bfloat16", 8, 2048),
        # evaluation: the loss of every token, a length that is no multiple of a tile
        dict(name="eval d12 bf16 5x1000", kind="eval", model="d12", dtype="bfloat16", B=5, T=1000),
        # a long prompt, of which only the last logits are wanted, as long as the user's text happens to be
        serve("GPT d20 prompt 1x1500", "GPT", "d20", 1, 1500, 0),
        # a conversation on a small model: short prompt, one token at a time
        serve("GPT d12 chat 1x24+32", "GPT", "d12", 1, 24, 32),
        # eight requests in step: decoding with a longer context
        serve("GPT d20 batch 8x512+32", "GPT", "d20", 8, 512, 32),
        # the same of the two other families: long prompts, and answers token by token
        serve("Virolorn prompt 1x4096", "Virolorn", "d20", 1, 4096, 0),
        serve("Virolorn chat 1x100+32", "Virolorn", "d20", 1, 100, 32),
        serve("Zurevik prompt 4x1777", "Zurevik", "d20", 4, 1777, 0),
        serve("Zurevik batch 4x300+32", "Zurevik", "d20", 4, 300, 32),
    ]


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(("train", "train", "eval", "serve", "serve", "serve", "serve"))
    if kind in ("train", "eval"):
        model, dtype = rng.choice((("tiny", "float32"), ("small", "float32"), ("small", "bfloat16"), ("d12", "bfloat16"), ("d20", "bfloat16")))
        if model == "tiny":
            B, T = log_int(rng, 1, 16), log_int(rng, 2, 32)
        elif model == "small":
            B, T = log_int(rng, 1, 8), log_int(rng, 64, 256)
        else:       # mostly whole tiles, as sequence lengths are chosen; ragged ones beside them
            ragged = rng.random() < 0.4
            T = log_int(rng, 130, 900) if ragged else 128 * log_int(rng, 2, 16)
            B = log_int(rng, 1, max(1, (2000 if ragged else 8192) // T))
        return dict(kind=kind, model=model, dtype=dtype, B=B, T=T)
    family = rng.choice(("GPT", "GPT", "Virolorn", "Zurevik"))
    model = rng.choice(("d12", "d20") if family == "GPT" else ("d20", "d20", "w2560"))
    B = log_int(rng, 1, 12)
    longest = min(4096, 8192 // B) if family != "GPT" else int((3e6 / B) ** 0.5)
    if rng.random() < 0.4:
        return dict(kind="serve", family=family, model=model, B=B, prompt=log_int(rng, 100, longest), new=0)
    return dict(kind="serve", family=family, model=model, B=B, prompt=log_int(rng, 4, min(1000, longest // 2)), new=log_int(rng, 8, 32 if model != "w2560" else 20))


# ---- what a program holds before the call ---------------------------------------------------------------------------------------------
def generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000 * seed + salt)


def gpt_config(case):
    fields = dict(GPTS[case["model"]])
    fields["sequence_len"] = case["T"] if case["kind"] != "serve" else 2048
    return fb.GPTConfig(**fields)


def gpt_theta(case, layout, seed):
    """Weights as `initialize_` draws them, every path carrying signal, with logits of a model that has seen some text."""
    theta = torch.empty(layout.nparams, device="cuda")
    fb.initialize_(theta, layout, seed=seed, all_nonzero=True)
    head = layout.lm_head
    theta[head.offset:head.offset + head.size].normal_(0.0, 0.6 * case_width(case) ** -0.5, generator=generator(seed, 1))
    return theta


def case_width(case):
    return (GPTS if case.get("family", "GPT") == "GPT" else DECODERS)[case["model"]]["n_embed" if case.get("family", "GPT") == "GPT" else "width"]


def packed(case, cfg, seed):
    batches = fb.PackedBatches(cfg.vocab_size, case["T"], case["B"], max_document_tokens=cfg.max_document_tokens,
                               mean_doc_len=min(512, max(3, case["T"] // 2)), seed=seed)
    return tuple(torch.from_numpy(x).cuda() for x in batches.next())


def moments(opt, seed):
    """Moments of a run that has been going on for a while."""
    g = generator(seed, 2)
    for a in opt.adamw:
        a.m.normal_(0.0, 3e-6, generator=g)
        a.v.uniform_(0.5e-10, 1.5e-10, generator=g)
    for m in opt.muon:
        m.m.normal_(0.0, 1e-4, generator=g)
        m.v.uniform_(0.5 / max(m.m.shape[1:]), 1.5 / max(m.m.shape[1:]), generator=g)
    opt.set_t([TRAINED] * len(opt.adamw))


def layer_list(case):
    s = DECODERS[case["model"]]
    layers = []
    for i in range(s["n_layer"]):
        if case["family"] == "Zurevik":
            kw = dict(mixer="attention", heads=s["heads"], kv_heads=s["kv_heads"], vdim=128, window=1024, ff=2 * s["width"], experts=8, top=2)
            if i % 4 < 2:       # the second reads the keys and values of the first
                layers.append(fb.LayerConfig(dim=128, scale=128 ** -0.5, qkv_bias=True, sink=True, gate="head", kv_from=i - 1 if i % 4 else None, **kw))
            else:
                layers.append(fb.LayerConfig(dim=64, scale=64 ** -0.5, maps=2, qk_norm=True, gate="element", diff=0.5, keep_first=4, **kw))
            continue
        lc = fb.LayerConfig(mixer=VIROLORN[i % 4], heads=s["heads"], dim=128, vdim=128, ff=s["ff"])
        if lc.mixer == "lightning":
            lc.decay = tuple(math.exp(-2.0 ** (-8.0 * (h + 1) / s["heads"])) for h in range(s["heads"]))
        elif lc.mixer == "channel_delta":
            lc.kv_heads, lc.conv, lc.decay_rank, lc.gate_rank = s["kv_heads"], 4, 128, 128
        else:
            lc.q_rank, lc.kv_rank, lc.rot_dim, lc.rot_dims, lc.rot_base, lc.scale = s["q_rank"], s["kv_rank"], 64, 64, 500000.0, 192 ** -0.5
        layers.append(lc)
    return layers


def decoder_config(case):
    s = DECODERS[case["model"]]
    if case["family"] == "Zurevik":
        return fb.DecoderConfig(vocab_size=s["vocab"], width=s["width"], norm_eps=1e-6, layers=layer_list(case), block="parallel", untied=True,
                                embed_scale=1.0, logit_softcap=15.0)
    return fb.DecoderConfig(vocab_size=s["vocab"], width=s["width"], norm_eps=1e-6, residual_mult=0.5, layers=layer_list(case))


def decoder_theta(layout, seed):
    theta = torch.zeros(max(s.offset + s.size for s in layout.values()) + 3 & ~3, device="cuda")
    g = generator(seed)
    for name, spec in layout.items():
        v, leaf = theta[spec.offset:spec.offset + spec.size], name.rsplit(".", 1)[-1]
        # a trained stream: every sublayer adds a little to what the token brought
        if leaf in ("norm1b", "norm2b"):
            v.fill_(0.3)
        elif leaf.startswith("norm"):
            v.fill_(1.0)
        elif leaf == "embed":
            v.normal_(0.0, 1.0, generator=g)
        elif "head" in layout and leaf in ("o", "down"):
            v.normal_(0.0, 0.1 * spec.shape[-1] ** -0.5, generator=g)
        elif leaf in ("sink", "b") and len(spec.shape) == 1 or leaf in ("lq1", "lk1", "lq2", "lk2"):
            v.normal_(0.0, 0.1, generator=g)
        elif leaf == "dt_bias":
            v.normal_(-3.0, 1.0, generator=g)
        elif leaf == "A_log":
            v.normal_(0.0, 0.5, generator=g)
        elif leaf == "router":       # a trained router is decided
            v.normal_(0.0, 4.0 * spec.shape[-1] ** -0.5, generator=g)
        else:
            v.normal_(0.0, spec.shape[-1] ** -0.5, generator=g)
    return theta


def request(case, vocab, base, seed):
    """The prompt, and the tokens that follow it one by one (int32, as sampling leaves them on the device)."""
    ids = torch.randint(base, vocab + base, (case["B"], case["prompt"] + case["new"]), generator=generator(seed, 3), device="cuda", dtype=torch.int32)
    return ids


def prepare(case, seed):
    if case["kind"] == "serve":
        if case["family"] == "GPT":
            cfg = gpt_config(case)
            layout = fb.parameter_layout(cfg)
            window, docs = OPTIONS[case["model"]]
            model = fb.GPT(fb.Params(gpt_theta(case, layout, seed), delta=False), cfg, layout, compute_type="bfloat16", short_window=window, doc_mask=docs)
        else:
            cfg = decoder_config(case)
            layout = fb.decoder_layout(cfg)
            model = fb.Decoder(fb.Params(decoder_theta(layout, seed), delta=False), cfg, layout, compute_type="bfloat16")
        ids = request(case, cfg.vocab_size, model.index_base, seed)
        cache = fb.KVCache(model.state(case["B"]), case["B"], case["prompt"] + case["new"])
        n = case["prompt"]
        return dict(kind="serve", model=model, cache=cache, prompt=ids[:, :n].contiguous(), steps=[ids[:, n + i].contiguous() for i in range(case["new"])])
    cfg = gpt_config(case)
    layout = fb.parameter_layout(cfg)
    window, docs = OPTIONS[case["model"]]
    options = dict(compute_type=case["dtype"], short_window=window, doc_mask=docs)
    tokens, targets, positions = packed(case, cfg, seed)
    theta = gpt_theta(case, layout, seed)
    if case["kind"] == "eval":
        model = fb.GPT(fb.Params(theta, delta=False), cfg, layout, **options)
        model.state(case["B"])
        return dict(kind="eval", model=model, batch=(tokens, targets, positions))
    params = fb.Params(theta)
    state = fb.gradient_state(params, cfg, layout, tokens, targets, positions, **options)
    opt = fb.MuonAdamW(params, layout, state, compute_type=case["dtype"], **LR)
    moments(opt, seed)
    return dict(kind="train", params=params, state=state, layout=layout, opt=opt, batch=(tokens, targets, positions), slots=float(tokens.numel()))


# ---- one pass ---------------------------------------------------------------------------------------------------------------------------
def parts(layout, vec):
    """A flat vector as views: the tables, each block's matrices, each block's value embeddings, and the gates and scalars at the end."""
    def view(first, last=None):
        last = last or first
        return vec[first.offset:last.offset + last.size]
    return dict(embedding=view(layout.embedding), lm_head=view(layout.lm_head), gates=view(layout.smear_gate, layout.lam_y),
                blocks=[view(b["wq"], b["proj"]) for b in layout.blocks],
                values=[view(b["ve_table"]) for b in layout.blocks if b["ve_table"] is not None])


def run(state):
    if state["kind"] == "train":
        loss, _ = fb.loss_and_gradient_(state["params"], state["state"], state["layout"], *state["batch"], reduction="sum", sync=False)
        state["opt"].step(Nt=state["slots"], **STEP)
        return dict(loss=loss, delta=parts(state["layout"], state["params"].delta), theta=state["params"].theta)
    if state["kind"] == "eval":
        return state["model"](*state["batch"], reduction="none")
    out = [fb.prefill(state["model"], state["cache"], state["prompt"])]
    for tokens in state["steps"]:
        out.append(fb.decode_step(state["model"], state["cache"], tokens))
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------------------------------------
def gpt_sizes(case):
    c = GPTS[case["model"]]
    d, L, V = c["n_embed"], c["n_layer"], c["vocab_size"]
    kv = d * c["n_kv_head"] // c["n_head"]
    block = 2 * d * d + 2 * d * kv + 8 * d * d
    return dict(d=d, L=L, V=V, kv=kv, block=block, matrices=L * block, head=d * V, tables=d * V + (L + 1) // 2 * kv * V)


def gpt_windows(case, T):
    c, (short, _) = GPTS[case["model"]], OPTIONS[case["model"]]
    S = min(T, short) if short else min(T, -(-T // 512) * 128)
    left = [S if c["window_pattern"][i % len(c["window_pattern"])] == "S" else T for i in range(c["n_layer"])]
    left[-1] = T
    return left


def seen(first, T, window):
    """(query, key) pairs of T tokens at positions first ..., each with at most `window` keys."""
    return sum(min(t + 1, window) for t in range(first, first + T))


def decoder_sizes(case):
    """Weights of the products of one token (two experts of each mixture), all weights, and bytes of state per column that a token reads."""
    s = DECODERS[case["model"]]
    w, H, G, used, held = s["width"], s["heads"], s["kv_heads"], 0, 0
    for lc in layer_list(case):
        if lc.mixer == "attention":
            q, k = H * lc.maps * lc.dim, 0 if lc.kv_from is not None else G * (lc.maps * lc.dim + lc.vdim)
            n = w * (q + k + (H * 128 if lc.gate == "element" else H)) + w * H * 128 + 8 * w
            used, held = used + n + 2 * 2 * w * lc.ff, held + n + 8 * 2 * w * lc.ff
            continue
        if lc.mixer == "lightning":
            n = 5 * w * H * 128
        elif lc.mixer == "channel_delta":
            n = w * (2 * G * 128 + 2 * H * 128 + H + 256) + 2 * H * 128 * 128
        else:
            n = w * (s["q_rank"] + s["kv_rank"] + 64 + H + H * 128) + s["q_rank"] * H * 192 + s["kv_rank"] * H * 256
        n += 3 * w * lc.ff
        used, held = used + n, held + n
    return used, held


def work(case):
    if case["kind"] == "serve":
        B, P, new = case["B"], case["prompt"], case["new"]
        if case["family"] == "GPT":
            z = gpt_sizes(case)
            head, used, held, per_key, per_pair = z["head"], z["matrices"], z["matrices"], 2 * 2 * z["kv"], 4 * z["d"]
            windows = [w + 1 for w in gpt_windows(case, 2048)]
            width, V = z["d"], z["V"]
        else:
            s = DECODERS[case["model"]]
            used, held = decoder_sizes(case)
            width, V = s["width"], s["vocab"]
            head = width * V
            if case["family"] == "Zurevik":
                windows, per_key, per_pair = [1024] * s["n_layer"], 2 * s["kv_heads"] * 256, 4 * s["heads"] * 128
            else:
                windows, per_key, per_pair = [1 << 30] * (s["n_layer"] // 4), 2 * (s["kv_rank"] + 64), 2 * s["heads"] * 320
        flops = 2.0 * B * (P * used + head) + per_pair * B * sum(seen(0, P, w) for w in windows)
        bytes_ = 2.0 * (held + head) + B * P * (2 * width + len(windows) * per_key) + 4 * B * V
        for t in range(P, P + new):
            flops += 2.0 * B * (used + head) + per_pair * B * sum(min(t + 1, w) for w in windows)
            bytes_ += 2.0 * (min(held, B * used) + head) + B * per_key * sum(min(t + 1, w) for w in windows) + 4 * B * V
        return dict(bytes=bytes_, flops=flops)
    z, N = gpt_sizes(case), case["B"] * case["T"]
    docs = OPTIONS[case["model"]][1]
    pairs = case["B"] * sum(seen(0, case["T"], min(w + 1, 512) if docs else w + 1) for w in gpt_windows(case, case["T"]))
    flops = 2.0 * N * (z["matrices"] + z["head"]) + 4.0 * z["d"] * pairs
    if case["kind"] == "eval":
        return dict(bytes=(2.0 if case["dtype"] == "bfloat16" else 4.0) * (z["matrices"] + z["head"]) + 16.0 * N, flops=flops)
    d, kv = z["d"], z["kv"]
    iteration = sum(4.0 * min(m, n) ** 2 * max(m, n) + 2.0 * min(m, n) ** 3 for m, n in ((d, d), (d, kv), (d, kv), (d, d), (d, 4 * d), (d, 4 * d)))
    # Θ, both moments (Muon: one) read and written, δ written
    return dict(bytes=28.0 * (z["tables"] + z["head"]) + 20.0 * z["matrices"] + 12.0 * N, flops=3 * flops + 5 * z["L"] * iteration)


def tolerance(case):
    """About four times what the results were measured to be off the same in 64 bits: fp32 steps 1e-6 (gradients) to 6e-6 (updated weights),
    bf16 steps 0.5 %, the mean over a token's losses 0.06 %, logits after 20 layers 1.3 % (a mixture's choice between two nearly equal
    experts can add to that)."""
    if case["kind"] == "serve":
        return dict(rel=3e-2, max=0.9)
    if case["dtype"] == "float32":
        return dict(rel=5e-5, max=1e-2)
    return dict(rel=2e-2, max=0.9) if case["kind"] == "train" else dict(rel=3e-3, max=0.12)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------------------------
def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def turn(x, angle, sign):
    """Half-split rotation of the last axis; angle [T, half]."""
    half = x.shape[-1] // 2
    c, s = torch.cos(angle)[:, None], sign * torch.sin(angle)[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c + b * s, b * c - a * s], -1)


def attend(q, k, v, mask, scale, sink=None):
    """q [T, H, D] on k [N, G, D], v [N, G, E]; mask [T, N]."""
    out, per = [], q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // per].T) * scale
        s = s.masked_fill(~mask, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(len(s), 1)], 1)
        p = torch.softmax(s, -1)
        out.append((p if sink is None else p[:, :-1]) @ v[:, h // per])
    return torch.stack(out, 1)


class Gpt64:
    """The GPT of the reference (its layout, its arithmetic) on one column, differentiable."""

    def __init__(self, case, seed, grad):
        self.cfg, (self.short, self.docs) = gpt_config(case), OPTIONS[case["model"]]
        self.layout, self.case = fb.parameter_layout(self.cfg), case
        self.theta = gpt_theta(case, self.layout, seed)
        self.eps = 2.0 ** -7 if case.get("dtype", "bfloat16") == "bfloat16" else 2.0 ** -23
        self.leaf = {}
        for name, spec in self.layout.named():
            t = self.theta[spec.offset:spec.offset + spec.size].double()
            self.leaf[name] = (t.view(spec.shape[1], spec.shape[0]) if len(spec.shape) == 2 else t).requires_grad_(grad)

    def hidden(self, tok, pos, T_of_windows):
        c, w, eps = self.cfg, self.leaf, self.eps
        T, d, H, G = len(tok), c.n_embed, c.n_head, c.n_kv_head
        hd = d // H
        angle = pos.double()[:, None] * torch.pow(100000.0, -torch.arange(0, hd, 2, device="cuda").double() / hd)[None]
        xe = rms(w["wte"][tok], eps)
        gate = w["lam_s"] * torch.sigmoid(xe[1:, :24] @ w["smear_gate"])
        x0 = torch.cat([xe[:1], xe[1:] + gate * xe[:-1]])
        t = torch.arange(T, device="cuda")
        x, kept = x0, None
        for i, left in enumerate(gpt_windows(self.case, T_of_windows)):
            p = f"l{i}."
            mask = (t[None] <= t[:, None]) & (t[:, None] - t[None] <= left)
            if self.docs:
                mask = mask & (t[None] >= (t - pos).clamp(min=0)[:, None])
            xm = w[p + "lam_b"] * x + w[p + "lam_x0"] * x0
            h = rms(xm, eps)
            q, k, v = ((h @ w[p + n]).view(T, -1, hd) for n in ("wq", "wk", "wv"))
            if p + "ve_table" in w:
                v = v + 3.0 * torch.sigmoid(h[:, :12] @ w[p + "ve_gate"])[..., None] * w[p + "ve_table"][tok].view(T, G, hd)
            q, k = (1.2 * rms(turn(y, angle, 1.0), eps) for y in (q, k))
            xa = xm + attend(q, k, v, mask, hd ** -0.5).reshape(T, d) @ w[p + "wo"]
            x = xa + torch.clamp(rms(xa, eps) @ w[p + "fc"], min=0) ** 2 @ w[p + "proj"]
            if i == c.n_layer // 2:
                kept = x
        return rms(x - w["lam_y"] * kept, eps)

    def logits(self, h):
        return 15.0 * torch.tanh(h @ self.leaf["lm_head"][:, :self.cfg.vocab_size] / 15.0)

    def losses(self, tokens, targets, positions):
        z = self.logits(self.hidden(tokens.long() - 1, positions.long(), self.case["T"]))
        return torch.nn.functional.cross_entropy(z, torch.where(targets > 0, targets - 1, -100).long(), reduction="none", ignore_index=-100)


POLAR = ((8.156554524902461, -22.48329292557795, 15.878769915207462), (4.042929935166739, -2.808917465908714, 0.5000178451051316),
         (3.8916678022926607, -2.772484153217685, 0.5060648178503393), (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
         (2.3465413258596377, -1.7097828382687081, 0.42323551169305323))


def muon64(W, G, m, v):
    """The new weights of one matrix; all as [out, in]."""
    mu, (rows, cols) = STEP["mu"], W.shape
    m = mu * m + (1 - mu) * G
    X = (1 - mu) * G + mu * m
    norm = lambda t: torch.sqrt((t * t).sum())  # noqa: E731
    X = X * (norm(X) / rows ** 0.5) / torch.sqrt((X * X).sum(1, keepdim=True)).clamp(min=1e-6)
    X = X / (1.01 * norm(X) + 1e-6)
    X = X.T if rows > cols else X
    for a, b, c in POLAR:
        A = X @ X.T
        X = a * X + (b * A + c * (A @ A)) @ X
    X = X.T if rows > cols else X
    X = X * (min(rows, cols) ** 0.5 / norm(X).clamp(min=1e-6))
    axis = 1 if rows >= cols else 0
    mean = (X * X).mean(axis, keepdim=True)
    v = 0.9 * v.view(mean.shape) + 0.1 * mean
    size = 1.0 / torch.sqrt(v.clamp(min=1e-10))
    X = X * (size * norm(X) / torch.sqrt((X.shape[axis] * mean * size ** 2).sum()).clamp(min=1e-10))
    rate = STEP["eta"] * LR["matrix_lr"] * max(1.0, rows / cols) ** 0.5
    return W - rate * X - rate * STEP["lam"] * W * (X * W >= 0)


def adam_groups(layout):
    """(tensor, rate, beta1, beta2, decay) in the optimiser's order."""
    s = (768.0 / layout.embedding.shape[0]) ** 0.5
    yield layout.lm_head, LR["unembedding_lr"] * s, 0.8, 0.96, 0.01
    yield layout.embedding, LR["embedding_lr"] * s, 0.8, 0.995, 0.001
    for b in layout.blocks:
        if b["ve_table"] is not None:
            yield b["ve_table"], 0.5 * LR["embedding_lr"] * s, 0.8, 0.995, 0.01
        yield b["lam_b"], 0.01 * LR["scalar_lr"], 0.8, 0.95, 0.05
        yield b["lam_x0"], LR["scalar_lr"], 0.96, 0.95, 0.0
    for spec in (layout.smear_gate, layout.lam_s, layout.lam_y):
        yield spec, LR["smear_lr"], 0.8, 0.95, 0.0


class Moments:
    """The optimiser's buffers as `moments` fills them, without an optimiser."""

    class Group:
        def __init__(self, m, v, specs):
            self.m, self.v, self.specs = m, v, specs

    def __init__(self, layout):
        new = lambda *n: torch.zeros(*n, device="cuda")  # noqa: E731
        self.adamw = [self.Group(new(s.size), new(s.size), [s]) for s, *_ in adam_groups(layout)]
        shapes = {}
        for b in layout.blocks:
            for n in ("wq", "wk", "wv", "wo", "fc", "proj", "ve_gate"):
                if b[n] is not None:
                    shapes.setdefault(b[n].shape, []).append(b[n])
        self.muon = [self.Group(new(len(s), c, r), new(len(s), r if r >= c else c), s) for (r, c), s in shapes.items()]

    def set_t(self, ts):
        pass


def exact_train(case, seed):
    g = Gpt64(case, seed, True)
    cfg, layout = g.cfg, g.layout
    batch, total = packed(case, cfg, seed), 0.0
    for b in range(case["B"]):
        loss = g.losses(*(x[b] for x in batch)).sum()
        loss.backward()
        total += loss.detach()
    delta, theta = (torch.zeros(layout.nparams, device="cuda", dtype=torch.float64) for _ in range(2))
    for name, spec in layout.named():
        delta[spec.offset:spec.offset + spec.size] = g.leaf[name].grad.reshape(-1)
        theta[spec.offset:spec.offset + spec.size] = g.leaf[name].detach().reshape(-1)
    held, slots = Moments(layout), float(batch[0].numel())
    g.leaf = None
    moments(held, seed)
    t = TRAINED + 1
    for group, (spec, rate, b1, b2, decay) in zip(held.adamw, adam_groups(layout)):
        at, rate = slice(spec.offset, spec.offset + spec.size), rate * STEP["eta"]
        x = delta[at] / slots
        m, v = b1 * group.m.double() + (1 - b1) * x, b2 * group.v.double() + (1 - b2) * x * x
        theta[at] = theta[at] * (1 - rate * decay) - rate * (m / (1 - b1 ** t)) / (torch.sqrt(v / (1 - b2 ** t)) + 1e-10)
    for group in held.muon:
        for k, spec in enumerate(group.specs):
            at, (r, c) = slice(spec.offset, spec.offset + spec.size), spec.shape
            new = muon64(theta[at].view(c, r).T, delta[at].view(c, r).T / slots, group.m[k].double().T, group.v[k].double())
            theta[at] = new.T.reshape(-1)
    return dict(loss=total.reshape(1), delta=parts(layout, delta), theta=theta)


def swish(x):
    return x * torch.sigmoid(x)


class Decoder64:
    """The decoders that list their layers, one column, from their equations."""

    def __init__(self, case, seed):
        self.cfg = decoder_config(case)
        layout = fb.decoder_layout(self.cfg)
        theta = decoder_theta(layout, seed)
        self.w = {n: theta[s.offset:s.offset + s.size].view(s.shape) for n, s in layout.items()}

    def get(self, name):
        return self.w[name].double()

    def lightning(self, h, p, lc):
        T, H = len(h), lc.heads
        q, k, v = (swish(h @ self.get(p + n).T).view(T, H, -1) for n in "qkv")
        decay = torch.tensor(lc.decay, device="cuda", dtype=torch.float64)
        S, out, at = torch.zeros(H, lc.dim, lc.vdim, device="cuda", dtype=torch.float64), [], 64
        for t0 in range(0, T, at):      # by blocks: what came before through the state, the block itself directly
            a, b, c = q[t0:t0 + at], k[t0:t0 + at], v[t0:t0 + at]
            n = torch.arange(len(a), device="cuda", dtype=torch.float64)
            gap = n[:, None] - n[None]
            fall = torch.where(gap >= 0, decay[:, None, None] ** gap.clamp(min=0), 0.0)
            out.append(torch.einsum("thd,hde,ht->the", a, S, decay[:, None] ** (n + 1)) + torch.einsum("thd,shd,hts,she->the", a, b, fall, c))
            S = decay[:, None, None] ** len(a) * S + torch.einsum("shd,hs,she->hde", b, decay[:, None] ** (len(a) - 1 - n), c)
        o = rms(torch.cat(out).reshape(T, -1), self.cfg.norm_eps) * self.get(p + "norm")
        return (o * torch.sigmoid(h @ self.get(p + "g").T)) @ self.get(p + "o").T

    def channel_delta(self, h, p, lc):
        T, H, G = len(h), lc.heads, lc.kv_heads
        x = {}
        for n in "qkv":
            y, taps = h @ self.get(p + n).T, self.get(p + n + ".conv")
            y = torch.cat([y.new_zeros(lc.conv - 1, y.shape[1]), y])
            x[n] = swish(sum(y[i:i + T] * taps[:, i] for i in range(lc.conv)))
        unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q = (unit(x["q"].view(T, G, -1)) * lc.dim ** -0.5).repeat_interleave(H // G, 1)
        k = unit(x["k"].view(T, G, -1)).repeat_interleave(H // G, 1)
        v, beta = x["v"].view(T, H, -1), torch.sigmoid(h @ self.get(p + "b").T)
        rate = torch.nn.functional.softplus((h @ self.get(p + "a1").T) @ self.get(p + "a2").T + self.get(p + "dt_bias"), threshold=700).view(T, H, -1)
        g = torch.exp(-torch.exp(self.get(p + "A_log"))[:, None] * rate)
        S, o = torch.zeros(H, lc.dim, lc.vdim, device="cuda", dtype=torch.float64), torch.empty_like(v)
        for t in range(T):
            S = S * g[t][:, :, None]
            u = beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0])
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o[t] = (q[t][:, None] @ S)[:, 0]
        o = rms(o, self.cfg.norm_eps) * self.get(p + "norm") * torch.sigmoid((h @ self.get(p + "g1").T) @ self.get(p + "g2").T).view(T, H, -1)
        return o.reshape(T, -1) @ self.get(p + "o").T

    def latent_attention(self, h, p, lc):
        T, H, eps = len(h), lc.heads, self.cfg.norm_eps
        t = torch.arange(T, device="cuda")
        angle = t.double()[:, None] * torch.pow(lc.rot_base, -torch.arange(0, lc.rot_dims, 2, device="cuda").double() / lc.rot_dims)[None]
        q = ((rms(h @ self.get(p + "dq").T, eps) * self.get(p + "dq.norm")) @ self.get(p + "uq").T).view(T, H, -1)
        q = torch.cat([q[..., :lc.dim], turn(q[..., lc.dim:], angle, -1.0)], -1)
        c = h @ self.get(p + "dkv").T
        r = turn(c[:, None, lc.kv_rank:], angle, -1.0)
        c = rms(c[:, :lc.kv_rank], eps) * self.get(p + "dkv.norm")
        k = torch.cat([(c @ self.get(p + "uk").T).view(T, H, -1), r.expand(T, H, -1)], -1)
        o = attend(q, k, (c @ self.get(p + "uv").T).view(T, H, -1), t[None] <= t[:, None], lc.scale)
        return (o * torch.sigmoid(h @ self.get(p + "g").T)[..., None]).reshape(T, -1) @ self.get(p + "o").T

    def attention(self, h, p, lc, i):
        T, H, G, eps = len(h), lc.heads, lc.kv_heads, self.cfg.norm_eps
        t = torch.arange(T, device="cuda")
        mask = (t[None] <= t[:, None]) & ((t[:, None] - t[None] < lc.window) | (t[None] < lc.keep_first))
        bias = lambda n: self.get(p + n + ".b") if lc.qkv_bias else 0.0  # noqa: E731
        q = (h @ self.get(p + "q").T + bias("q")).view(T, H, lc.maps, -1)
        if lc.kv_from is None:
            k = (h @ self.get(p + "k").T + bias("k")).view(T, G, lc.maps, -1)
            k = rms(k, eps) * self.get(p + "k.norm") if lc.qk_norm else k
            self.kv[i] = k, (h @ self.get(p + "v").T + bias("v")).view(T, G, -1)
        k, v = self.kv[i if lc.kv_from is None else lc.kv_from]
        q = rms(q, eps) * self.get(p + "q.norm") if lc.qk_norm else q
        a = [attend(q[:, :, m], k[:, :, m], v, mask, lc.scale, self.get(p + "sink") if lc.sink else None) for m in range(lc.maps)]
        if lc.maps == 2:
            e = lambda n: torch.exp((self.get(p + "lq" + n) * self.get(p + "lk" + n)).sum())  # noqa: E731
            a[0] = rms(a[0] - (e("1") - e("2") + lc.diff) * a[1], eps) * (1.0 - lc.diff)
        gate = torch.sigmoid(h @ self.get(p + "g").T)
        o = a[0] * (gate[..., None] if lc.gate == "head" else gate.view(T, H, -1))
        return o.reshape(T, -1) @ self.get(p + "o").T

    def experts(self, h, p, lc):
        best = torch.topk(h @ self.get(p + "router").T + self.get(p + "router.b"), lc.top)
        share, out = torch.softmax(best.values, -1), torch.zeros_like(h)
        for e in range(lc.experts):
            row, k = torch.nonzero(best.indices == e, as_tuple=True)
            out.index_add_(0, row, share[row, k][:, None] * (torch.clamp(h[row] @ self.get(p + f"e{e}.up").T, min=0) ** 2 @ self.get(p + f"e{e}.down").T))
        return out

    def logits(self, tokens, first):
        """Of positions first .. len(tokens) - 1."""
        c, self.kv = self.cfg, {}
        norm = lambda x, n: rms(x, c.norm_eps) * self.get(n)  # noqa: E731
        x = c.embed_scale * self.get("embed")[tokens.long()]
        for i, lc in enumerate(c.layers):
            p = f"l{i}."
            if c.block == "parallel":
                x = x + self.attention(norm(x, p + "norm1"), p + "mix.", lc, i) + self.experts(norm(x, p + "norm2"), p + "mlp.", lc)
                continue
            x = x + c.residual_mult * norm(getattr(self, lc.mixer)(norm(x, p + "norm1"), p + "mix.", lc), p + "norm1b")
            h = norm(x, p + "norm2")
            y = (swish(h @ self.get(p + "mlp.gate").T) * (h @ self.get(p + "mlp.up").T)) @ self.get(p + "mlp.down").T
            x = x + c.residual_mult * norm(y, p + "norm2b")
        z = norm(x[first:], "final.norm") @ self.get("head" if c.untied else "embed").T
        return c.logit_softcap * torch.tanh(z / c.logit_softcap) if c.logit_softcap else z


def exact(case, seed):
    if case["kind"] == "train":
        return exact_train(case, seed)
    if case["kind"] == "eval":
        g = Gpt64(case, seed, False)
        batch = packed(case, g.cfg, seed)
        return torch.stack([g.losses(*(x[b] for x in batch)) for b in range(case["B"])])
    P, new, B, out = case["prompt"], case["new"], case["B"], []
    if case["family"] == "Virolorn" and B * (P + new) > 8000:      # token by token: too long
        return None
    if case["family"] == "GPT":
        g = Gpt64(case, seed, False)
        ids = request(case, g.cfg.vocab_size, 1, seed)
        pos = torch.arange(P + new, device="cuda")
        out = [g.logits(g.hidden(ids[b].long() - 1, pos, 2048)[P - 1:]) for b in range(B)]
    else:
        d = Decoder64(case, seed)
        ids = request(case, d.cfg.vocab_size, 0, seed)
        out = [d.logits(ids[b], P - 1) for b in range(B)]
    return [torch.stack([z[i] for z in out]) for i in range(new + 1)]
