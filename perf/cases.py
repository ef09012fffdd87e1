"""The work by which this engine's speed is measured: decode and prefill steps of its model families at their own widths.

Every case is one engine step of a slice of a preset: a few whole layers (one period where the layers differ) with the vocabulary cut in
about the same proportion, so that the head keeps its share of the step.  The weights go through the checkpoint loader, the step
through the engine's runner: ``forward`` of a :class:`ForwardBatch` (a replayed CUDA graph for decode steps where the engine captures
them) and the logits of every sequence's last row.  Outputs are the hidden states, the logits, the paged cache and the recurrent states.

=========  ==========================================================================================================
family     slice
=========  ==========================================================================================================
dense      ``llama3-8b``: 4 of 32 layers; FP8 128 x 128 block-scaled weights
moe        ``qwen3-30b-a3b``: 4 of 48 layers; bf16 attention, 128 NVFP4 experts
hybrid     ``qwen3-next-80b``: 4 of 48 layers (three of Gated DeltaNet, one of attention); FP8, 512 experts and a shared one
mamba      ``nemotron-h-8b``: Mamba-2, MLP, Mamba-2, attention, MLP, Mamba-2, MLP out of 52 blocks; bf16
=========  ==========================================================================================================

Sizes: ``seqs`` sequences with ``ctx`` tokens in the cache and ``rows`` new ones each; with ``ragged`` these are the largest and the
others fall off to a quarter.  ``rows`` 0 stands for decode (one new token).  ``kv``: the cache's data type.
"""
import dataclasses
import math

import torch
import torch.nn.functional as F

BLOCK = 16
OPEN = 64            # channels of the residual stream that only the embedding writes; the routers read these


def listed():
    return [
        # one user's stream: what sets the time per token of an interactive session
        dict(name="dense-decode-1", family="dense", seqs=1, rows=0, ctx=1100, ragged=False, kv="fp8"),
        # a full server, requests at different places of their answers
        dict(name="dense-decode-128", family="dense", seqs=128, rows=0, ctx=1280, ragged=True, kv="fp8"),
        # a short chat prompt
        dict(name="dense-prefill-77", family="dense", seqs=1, rows=77, ctx=0, ragged=False, kv="fp8"),
        # a full prefill step: eight prompts of 1024 tokens
        dict(name="dense-prefill-8x1024", family="dense", seqs=8, rows=1024, ctx=0, ragged=False, kv="fp8"),
        # a few users of a mixture of experts: every row takes other experts
        dict(name="moe-decode-12", family="moe", seqs=12, rows=0, ctx=2300, ragged=True, kv="fp8"),
        # three prompts of different lengths in one step
        dict(name="moe-prefill-3x2001", family="moe", seqs=3, rows=2001, ctx=0, ragged=True, kv="fp8"),
        # one user of the hybrid model at a long context
        dict(name="hybrid-decode-1", family="hybrid", seqs=1, rows=0, ctx=8500, ragged=False, kv="fp8"),
        # its server load
        dict(name="hybrid-decode-48", family="hybrid", seqs=48, rows=0, ctx=3000, ragged=True, kv="fp8"),
        # a long prompt
        dict(name="hybrid-prefill-8192", family="hybrid", seqs=1, rows=8192, ctx=0, ragged=False, kv="fp8"),
        # the rest of a prompt whose first 4096 tokens came from the prefix cache
        dict(name="hybrid-prefill-517+4096", family="hybrid", seqs=1, rows=517, ctx=4096, ragged=False, kv="fp8"),
        # prompts and server load of a Mamba-2 model in 16 bits
        dict(name="mamba-prefill-4x1500", family="mamba", seqs=4, rows=1500, ctx=0, ragged=True, kv="bf16"),
        dict(name="mamba-decode-32", family="mamba", seqs=32, rows=0, ctx=2048, ragged=False, kv="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["dense", "dense", "moe", "hybrid", "hybrid", "mamba"])
    kv = "fp8" if rng.random() < 0.7 else "bf16"
    if rng.random() < 0.5:
        seqs = _log(rng, 1, 128)
        return dict(family=family, seqs=seqs, rows=0, ctx=_log(rng, 40, min(8192, 131072 // seqs)), ragged=seqs > 1, kv=kv)
    total = _log(rng, 16, 8000)
    seqs = rng.randint(1, min(8, total // 8))
    ctx = _log(rng, 16, 4096) if seqs < 4 and total < 2048 and rng.random() < 0.4 else 0
    return dict(family=family, seqs=seqs, rows=total // seqs, ctx=ctx, ragged=seqs > 1 and rng.random() < 0.7, kv=kv)


def _falling(n, most, ragged):
    """``n`` lengths from ``most`` down to about a quarter of it."""
    return [max(1, most - (3 * most // 4) * i // n) if ragged else most for i in range(n)]


def _lengths(case):
    """New rows and cached tokens of every sequence."""
    n = case["seqs"]
    if case["rows"] == 0:
        return [1] * n, _falling(n, case["ctx"], case["ragged"])
    return _falling(n, case["rows"], case["ragged"]), [case["ctx"]] * n


# ----------------------------------------------------------------------------- the models
def _config(case):
    from atlas_b200.config import PRESETS
    family, cut = case["family"], {}
    if family == "dense":
        cfg, cut = PRESETS["llama3-8b"](), dict(num_hidden_layers=4, vocab_size=16032)
    elif family == "moe":
        cfg, cut = PRESETS["qwen3-30b-a3b"](), dict(num_hidden_layers=4, vocab_size=12672)
    elif family == "hybrid":
        cfg, cut = PRESETS["qwen3-next-80b"](), dict(num_hidden_layers=4, vocab_size=12672, mtp_num_layers=0)
    else:
        kinds = ["mamba", "mlp", "mamba", "attention", "mlp", "mamba", "mlp"]
        cfg, cut = PRESETS["nemotron-h-8b"](), dict(num_hidden_layers=len(kinds), vocab_size=17664, block_types=kinds)
    return dataclasses.replace(cfg, **cut)


class _Maker:
    """Random checkpoint tensors.  Values that the loader quantises to FP8 are representable exactly (e4m3 times a power of two, with
    the largest code in every block), so that the loaded model is the one these tensors say."""

    def __init__(self, cfg, seed):
        self.cfg, self.fp8 = cfg, cfg.quant.method == "fp8_block"
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.gen, device="cuda") * std).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=self.gen, device="cuda") * (hi - lo) + lo

    def weight(self, *shape, out=False):
        """N(0, 0.02), rounded; ``out``: a projection back to the residual stream, an eighth of that as initialisations of deep models
        have it, that writes no open channel."""
        w = torch.randn(*shape, generator=self.gen, device="cuda", dtype=torch.bfloat16)
        if self.fp8:
            w = (w.mul_(164.0)).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn).to(torch.bfloat16).mul_(2.0 ** -13)
        else:
            w.mul_(0.02)
        if out:
            w.mul_(0.125)[..., -OPEN:, :] = 0
        return w

    def packed(self, *shape, out=False):
        """NVFP4: codes, a scale per 16 and one for all."""
        codes = torch.randint(0, 256, shape[:-1] + (shape[-1] // 2,), generator=self.gen, device="cuda", dtype=torch.uint8)
        if out:
            codes[..., -OPEN:, :] = 0
        scale = self.uniform(*shape[:-1], shape[-1] // 16, lo=0.5, hi=1.5).to(torch.float8_e4m3fn)
        return codes, scale, torch.full((1,), 0.02 / 2.926 / (8 if out else 1), device="cuda")

    def router(self):
        w = torch.zeros(self.cfg.num_experts, self.cfg.hidden_size, device="cuda")
        w[:, -OPEN:] = torch.randn(self.cfg.num_experts, OPEN, generator=self.gen, device="cuda") * 0.15
        return w.to(torch.bfloat16)

    def norm(self, n):
        return self.normal(n, std=0.1, dtype=torch.float32).add_(0.0 if self.cfg.norm_plus_one else 1.0).to(torch.bfloat16)

    def steps(self, n):
        """Step-size biases of a trained recurrence: softplus of them lies between 0.001 and 0.1."""
        dt = torch.exp(self.uniform(n, lo=math.log(1e-3), hi=math.log(0.1)))
        return dt + torch.log(-torch.expm1(-dt))


def _attention(m, pre, norms):
    c, d = m.cfg, m.cfg.head_dim
    t = {f"{pre}.q_proj.weight": m.weight(c.q_size * (2 if c.attn_output_gate else 1), c.hidden_size), f"{pre}.k_proj.weight": m.weight(c.kv_size, c.hidden_size),
         f"{pre}.v_proj.weight": m.weight(c.kv_size, c.hidden_size), f"{pre}.o_proj.weight": m.weight(c.hidden_size, c.q_size, out=True)}
    if norms:
        t[f"{pre}.q_norm.weight"], t[f"{pre}.k_norm.weight"] = m.norm(d), m.norm(d)
    return t


def _checkpoint(case, seed):
    """Named tensors as a checkpoint has them; expert stacks under one name each, ``...experts.<projection>``."""
    c = _config(case)
    m, t, H = _Maker(c, seed), {}, c.hidden_size
    if case["family"] == "mamba":
        t["backbone.embeddings.weight"] = m.normal(c.vocab_size, H)
        di, gn, nh = c.mamba_num_heads * c.mamba_head_dim, c.mamba_n_groups * c.ssm_state_size, c.mamba_num_heads
        for i, kind in enumerate(c.block_types):
            pre = f"backbone.layers.{i}.mixer"
            t[f"backbone.layers.{i}.norm.weight"] = m.norm(H)
            if kind == "mamba":
                t[f"{pre}.in_proj.weight"] = m.weight(2 * di + 2 * gn + nh, H)
                t[f"{pre}.conv1d.weight"], t[f"{pre}.conv1d.bias"] = m.normal(di + 2 * gn, 1, 4, std=0.3), m.normal(di + 2 * gn, std=0.1)
                t[f"{pre}.dt_bias"], t[f"{pre}.A_log"], t[f"{pre}.D"] = m.steps(nh), torch.log(m.uniform(nh, lo=1.0, hi=16.0)), torch.ones(nh, device="cuda")
                t[f"{pre}.norm.weight"], t[f"{pre}.out_proj.weight"] = m.norm(di), m.weight(H, di, out=True)
            elif kind == "attention":
                t.update(_attention(m, pre, False))
            else:
                t[f"{pre}.up_proj.weight"], t[f"{pre}.down_proj.weight"] = m.weight(c.intermediate_size, H), m.weight(H, c.intermediate_size, out=True)
        t["backbone.norm_f.weight"], t["lm_head.weight"] = m.norm(H), m.normal(c.vocab_size, H, std=0.02)
        return t
    t["model.embed_tokens.weight"] = m.normal(c.vocab_size, H)
    for i in range(c.num_hidden_layers):
        pre = f"model.layers.{i}"
        t[f"{pre}.input_layernorm.weight"], t[f"{pre}.post_attention_layernorm.weight"] = m.norm(H), m.norm(H)
        if c.layer_kind(i) == "attention":
            t.update(_attention(m, f"{pre}.self_attn", c.qk_norm))
        else:
            g = f"{pre}.linear_attn"
            kd, nv = c.linear_num_key_heads * c.linear_key_head_dim, c.linear_num_value_heads
            vd = nv * c.linear_value_head_dim
            t[f"{g}.in_proj_qkv.weight"], t[f"{g}.in_proj_z.weight"] = m.weight(2 * kd + vd, H), m.weight(vd, H)
            t[f"{g}.in_proj_b.weight"], t[f"{g}.in_proj_a.weight"] = m.weight(nv, H), m.weight(nv, H)
            t[f"{g}.conv1d.weight"] = m.normal(2 * kd + vd, 1, 4, std=0.3)
            t[f"{g}.dt_bias"], t[f"{g}.A_log"] = m.steps(nv), torch.log(m.uniform(nv, lo=0.5, hi=16.0))
            t[f"{g}.norm.weight"] = m.normal(c.linear_value_head_dim, std=0.1, dtype=torch.float32).add_(1.0).to(torch.bfloat16)
            t[f"{g}.out_proj.weight"] = m.weight(H, vd, out=True)
        if c.num_experts:
            e, n = c.moe_intermediate_size, c.num_experts
            make = m.packed if c.quant.method == "nvfp4" else m.weight
            t[f"{pre}.mlp.gate.weight"] = m.router()
            t[f"{pre}.mlp.experts.gate_proj"], t[f"{pre}.mlp.experts.up_proj"] = make(n, e, H), make(n, e, H)
            t[f"{pre}.mlp.experts.down_proj"] = make(n, H, e, out=True)
        width, name = (c.shared_expert_intermediate_size, "mlp.shared_expert") if c.num_experts else (c.intermediate_size, "mlp")
        if width:
            t[f"{pre}.{name}.gate_proj.weight"], t[f"{pre}.{name}.up_proj.weight"] = m.weight(width, H), m.weight(width, H)
            t[f"{pre}.{name}.down_proj.weight"] = m.weight(H, width, out=True)
            if c.num_experts:
                t[f"{pre}.mlp.shared_expert_gate.weight"] = m.normal(1, H, std=0.02)
    t["model.norm.weight"], t["lm_head.weight"] = m.norm(H), m.normal(c.vocab_size, H, std=0.02)
    return t


class _Shards:
    """A checkpoint that is in memory already, as ``load_weights`` reads one."""

    def __init__(self, tensors):
        self.t = tensors

    def keys(self):
        return self.t.keys()

    def has(self, name):
        return name in self.t

    def get(self, name):
        return self.t[name]

    def maybe(self, name):
        return self.t.get(name)

    def linear(self, prefix):
        from atlas_b200.loader import QTensor
        if prefix + ".weight" in self.t:
            return QTensor("dense", self.t[prefix + ".weight"])
        root, expert, leaf = prefix.rsplit(".", 2)
        w, e = self.t[f"{root}.{leaf}"], int(expert)
        return QTensor("nvfp4", w[0][e], w[1][e], w[2]) if isinstance(w, tuple) else QTensor("dense", w[e])

    def close(self):
        pass


# ----------------------------------------------------------------------------- inputs
def _inputs(case, seed):
    """Token ids, and for sequences with a past the contents of cache and states."""
    c = _config(case)
    rows, ctx = _lengths(case)
    gen = torch.Generator(device="cuda").manual_seed(seed * 2 + 1)
    ids = [torch.randint(0, c.vocab_size, (n,), generator=gen, device="cuda") for n in rows]
    normal = lambda *s, std: torch.randn(*s, generator=gen, device="cuda", dtype=torch.bfloat16) * std
    cached = torch.float8_e4m3fn if case["kv"] == "fp8" else torch.bfloat16
    kv, states = {}, {}
    spread = 1.0 if c.qk_norm else 1.28
    for i in range(c.num_hidden_layers):
        kind = c.layer_kind(i)
        if kind == "attention" and max(ctx):
            kv[i] = [tuple(normal(n, c.num_key_value_heads, c.head_dim, std=spread).to(cached) for _ in "kv") for n in ctx]
        elif kind in ("gdn", "mamba2") and max(ctx):
            if kind == "gdn":
                h = (c.linear_num_value_heads, c.linear_key_head_dim, c.linear_value_head_dim)
                conv = 2 * c.linear_num_key_heads * c.linear_key_head_dim + c.linear_num_value_heads * c.linear_value_head_dim
            else:
                h = (c.mamba_num_heads, c.mamba_head_dim, c.ssm_state_size)
                conv = c.mamba_num_heads * c.mamba_head_dim + 2 * c.mamba_n_groups * c.ssm_state_size
            states[i] = (torch.randn(len(rows), *h, generator=gen, device="cuda") * 0.1, normal(len(rows), conv, 3, std=0.9))
    return ids, kv, states


def _pages(case):
    """Block tables: the sequences' pages in turn, as requests that grow side by side get them."""
    rows, ctx = _lengths(case)
    need = [(n + p + BLOCK) // BLOCK for n, p in zip(rows, ctx)]
    tables, page = [[] for _ in need], 0
    for k in range(max(need)):
        for i, n in enumerate(need):
            if k < n:
                tables[i].append(page)
                page += 1
    return tables, page


def _slots(table, lo, hi):
    p = torch.arange(lo, hi, device="cuda")
    return torch.tensor(table, device="cuda")[p // BLOCK] * BLOCK + p % BLOCK


def prepare(case, seed):
    from atlas_b200.config import EngineConfig
    from atlas_b200.engine import LLMEngine
    from atlas_b200.loader import load_weights
    from atlas_b200.models import ForwardBatch, build_model
    from atlas_b200.ops import cuda
    c = _config(case)
    # models of several sizes in one process: the shared workspace of decode attention is reserved for the largest before any graph
    cuda.reserve_scratch("attn_part_o", 64 << 20, torch.device("cuda"))
    cuda.reserve_scratch("attn_part_ml", 4 << 20, torch.device("cuda"))
    most = 32768 if case["family"] == "hybrid" else 8192 + 1024
    model = build_model(c, device="cuda")
    load_weights(model, _Shards(_checkpoint(case, seed)))
    model.finalize(most)
    rows, ctx = _lengths(case)
    tables, pages = _pages(case)
    eng = LLMEngine(model, EngineConfig(max_seq_len=most, block_size=BLOCK, kv_cache_dtype=case["kv"], num_kv_blocks=pages + 1, max_num_seqs=len(rows),
                                        max_batch_size=len(rows), max_prefill_tokens=8192, enable_prefix_caching=False))
    ids, kv, states = _inputs(case, seed)
    for i, parts in kv.items():
        for table, n, pair in zip(tables, ctx, parts):
            s = _slots(table, 0, n)
            for pool, x in zip(eng.cache.kv[i], pair):
                if x.dtype == torch.float8_e4m3fn:
                    pool, x = pool.view(torch.uint8), x.view(torch.uint8)
                pool[s // BLOCK, s % BLOCK] = x
    for i, (h, conv) in states.items():
        eng.cache.states[i]["h"][:len(rows)] = h
        eng.cache.states[i]["conv"][:len(rows)] = conv
    hybrid = case["family"] in ("hybrid", "mamba")
    batch = ForwardBatch.build([t.tolist() for t in ids], ctx, tables, BLOCK, device="cuda", state_slots=list(range(len(rows))) if hybrid else None,
                               has_state=[n > 0 for n in ctx] if hybrid else None)
    last = torch.tensor(rows).cumsum(0).sub(1).tolist()
    return dict(engine=eng, batch=batch, last=last)


def run(state):
    eng = state["engine"]
    with torch.inference_mode():
        hidden = eng.runner.forward(state["batch"])
        logits = eng.runner.logits(hidden, state["last"])
    n = state["batch"].num_seqs
    return dict(logits=logits, hidden=hidden, kv={str(i): tuple(p) for i, p in eng.cache.kv.items()},
                states={str(i): [s["h"][:n], s["conv"][:n]] for i, s in eng.cache.states.items()})


# ----------------------------------------------------------------------------- what a step cannot do without
def work(case):
    c = _config(case)
    rows, ctx = _lengths(case)
    T, H = sum(rows), c.hidden_size
    pairs = sum(n * p + n * (n + 1) // 2 for n, p in zip(rows, ctx))
    wb = 1.0 if c.quant.method == "fp8_block" else 2.0
    eb = {"nvfp4": 9.0 / 16.0, "fp8_block": 1.0}.get(c.quant.method, 2.0)
    kb = 1.0 if case["kv"] == "fp8" else 2.0
    nbytes = T * H * 2 * 2 + len(rows) * c.vocab_size * 2 + c.vocab_size * H * 2
    flops = 2.0 * len(rows) * c.vocab_size * H
    for i in range(c.num_hidden_layers):
        kind, dense = c.layer_kind(i), 0
        if kind == "attention":
            dense += H * (c.q_size * (2 if c.attn_output_gate else 1) + 2 * c.kv_size) + H * c.q_size
            nbytes += 2 * c.kv_size * kb * (sum(ctx) + T)
            flops += 4.0 * pairs * c.q_size
        elif kind == "gdn":
            kd, vd = c.linear_num_key_heads * c.linear_key_head_dim, c.linear_num_value_heads * c.linear_value_head_dim
            dense += H * (2 * kd + 2 * vd + 2 * c.linear_num_value_heads) + H * vd
            nbytes += len(rows) * vd * c.linear_key_head_dim * 4 * (2 if max(ctx) else 1)
            flops += 6.0 * T * vd * c.linear_key_head_dim
        elif kind == "mamba2":
            di, gn = c.mamba_num_heads * c.mamba_head_dim, c.mamba_n_groups * c.ssm_state_size
            dense += H * (2 * di + 2 * gn + c.mamba_num_heads) + H * di
            nbytes += len(rows) * di * c.ssm_state_size * 4 * (2 if max(ctx) else 1)
            flops += 5.0 * T * di * c.ssm_state_size
        if c.num_experts:
            one = 3 * H * c.moe_intermediate_size
            hit = c.num_experts * (1.0 - (1.0 - c.num_experts_per_tok / c.num_experts) ** T)
            nbytes += hit * one * eb + c.num_experts * H * 2
            flops += 2.0 * T * (c.num_experts_per_tok * one + c.num_experts * H)
            dense += 3 * H * c.shared_expert_intermediate_size
        elif not c.block_types:
            dense += 3 * H * c.intermediate_size
        elif c.block_types[i] == "mlp":
            dense += 2 * H * c.intermediate_size
        nbytes += dense * wb
        flops += 2.0 * T * dense
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    # activations are rounded to FP8 (in groups of 128) or bf16 between the products: another order of the sums turns some roundings
    if case["family"] == "mamba":
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 2e-2, "max": 0.99}


# ----------------------------------------------------------------------------- the same in 64 bits
def _value(w, e=None):
    """Weight in 64 bits; of expert ``e``."""
    if not isinstance(w, tuple):
        return (w if e is None else w[e]).double()
    codes, scale, g = w[0][e], w[1][e], w[2]
    lut = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6], dtype=torch.float64, device="cuda")
    lut = torch.cat([lut, -lut])
    v = torch.stack([lut[(codes & 15).long()], lut[(codes >> 4).long()]], -1).flatten(1)
    return v * scale.double().repeat_interleave(16, 1) * g.double()


def _rms(x, w, c):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + c.rms_norm_eps)
    return y * (w.double() + (1.0 if c.norm_plus_one else 0.0))


def _turn(x, pos, c):
    n = int(c.head_dim * c.partial_rotary_factor)
    if n == 0:
        return x
    f = c.rope_theta ** (-torch.arange(0, n // 2, device="cuda", dtype=torch.float64) * 2 / n)
    a = (pos.double()[:, None] * f)[:, None]
    u, v = x[..., :n // 2], x[..., n // 2:n]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin(), x[..., n:]], -1)


def _attend(x, t, pre, c, rows, ctx, past):
    """Attention of every sequence, and its new keys and values."""
    d, out, new, r0 = c.head_dim, [], [], 0
    q = x @ _value(t[f"{pre}.q_proj.weight"]).t()
    k = (x @ _value(t[f"{pre}.k_proj.weight"]).t()).view(len(x), -1, d)
    v = (x @ _value(t[f"{pre}.v_proj.weight"]).t()).view(len(x), -1, d)
    gate = None
    q = q.view(len(x), c.num_attention_heads, -1)
    if c.attn_output_gate:
        q, gate = q[..., :d], q[..., d:]
    if f"{pre}.q_norm.weight" in t:
        q, k = _rms(q, t[f"{pre}.q_norm.weight"], c), _rms(k, t[f"{pre}.k_norm.weight"], c)
    for i, (n, p) in enumerate(zip(rows, ctx)):
        pos = torch.arange(p, p + n, device="cuda")
        qi, ki, vi = _turn(q[r0:r0 + n], pos, c), _turn(k[r0:r0 + n], pos, c), v[r0:r0 + n]
        new.append((ki, vi))
        if p:
            ki, vi = torch.cat([past[i][0].double(), ki]), torch.cat([past[i][1].double(), vi])
        rep = c.num_attention_heads // c.num_key_value_heads
        o = torch.empty(n, c.num_attention_heads, d, dtype=torch.float64, device="cuda")
        for h in range(c.num_attention_heads):
            s = qi[:, h] @ ki[:, h // rep].t() * d ** -0.5
            s.masked_fill_(torch.arange(p + n, device="cuda")[None] > pos[:, None], -math.inf)
            o[:, h] = s.softmax(-1) @ vi[:, h // rep]
        out.append(o)
        r0 += n
    o = torch.cat(out)
    if gate is not None:
        o = o * torch.sigmoid(gate)
    return o.flatten(1) @ _value(t[f"{pre}.o_proj.weight"]).t(), new


def _convolve(x, w, bias, window):
    """Short convolution with silu over one sequence, and the window behind it."""
    full = torch.cat([window.double().t(), x])
    y = (full.unfold(0, w.shape[-1], 1) * w.double().flatten(1)).sum(-1)
    return F.silu(y if bias is None else y + bias.double()), full[-(w.shape[-1] - 1):].t()


def _spans(rows):
    r0 = 0
    for n in rows:
        yield r0, r0 + n
        r0 += n


def _delta_net(x, t, pre, c, rows, state):
    kd, dk, dv = c.linear_num_key_heads * c.linear_key_head_dim, c.linear_key_head_dim, c.linear_value_head_dim
    nv, rep = c.linear_num_value_heads, c.linear_num_value_heads // c.linear_num_key_heads
    mixed, z, b, a = (x @ _value(t[f"{pre}.in_proj_{n}.weight"]).t() for n in ("qkv", "z", "b", "a"))
    decay = torch.exp(-t[f"{pre}.A_log"].double().exp() * F.softplus(a + t[f"{pre}.dt_bias"].double()))
    beta, out, hs, windows = torch.sigmoid(b), [], [], []
    unit = lambda u: u * torch.rsqrt(u.square().sum(-1, keepdim=True) + 1e-6)
    for i, (lo, hi) in enumerate(_spans(rows)):
        window = state[1][i] if state else torch.zeros(2 * kd + nv * dv, 3, device="cuda")
        y, after = _convolve(mixed[lo:hi], t[f"{pre}.conv1d.weight"], None, window)
        q = (unit(y[:, :kd].view(hi - lo, -1, dk)) * dk ** -0.5).repeat_interleave(rep, 1)
        k = unit(y[:, kd:2 * kd].view(hi - lo, -1, dk)).repeat_interleave(rep, 1)
        v = y[:, 2 * kd:].view(hi - lo, nv, dv)
        h = state[0][i].double() if state else torch.zeros(nv, dk, dv, dtype=torch.float64, device="cuda")
        o = torch.empty(hi - lo, nv, 1, dv, dtype=torch.float64, device="cuda")
        for r in range(hi - lo):
            h = h * decay[lo + r][:, None, None]
            u = (v[r][:, None] - k[r][:, None] @ h) * beta[lo + r][:, None, None]
            h = torch.baddbmm(h, k[r][:, :, None], u)
            torch.bmm(q[r][:, None], h, out=o[r])
        out.append(o[:, :, 0])
        hs.append(h)
        windows.append(after)
    o = torch.cat(out)
    o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + c.rms_norm_eps) * t[f"{pre}.norm.weight"].double() * F.silu(z.view(len(x), nv, dv))
    return o.flatten(1) @ _value(t[f"{pre}.out_proj.weight"]).t(), [torch.stack(hs), torch.stack(windows)]


def _mamba(x, t, pre, c, rows, state):
    nh, hd, ns = c.mamba_num_heads, c.mamba_head_dim, c.ssm_state_size
    di, gn = nh * hd, c.mamba_n_groups * ns
    z, xbc, raw = (x @ _value(t[f"{pre}.in_proj.weight"]).t()).split([di, di + 2 * gn, nh], 1)
    step = F.softplus(raw + t[f"{pre}.dt_bias"].double()).clamp_min(c.mamba_dt_min)
    decay, out, hs, windows = torch.exp(-step * t[f"{pre}.A_log"].double().exp()), [], [], []
    for i, (lo, hi) in enumerate(_spans(rows)):
        window = state[1][i] if state else torch.zeros(di + 2 * gn, 3, device="cuda")
        y, after = _convolve(xbc[lo:hi], t[f"{pre}.conv1d.weight"], t[f"{pre}.conv1d.bias"], window)
        u = y[:, :di].view(hi - lo, nh, hd)
        b, g = (p.view(hi - lo, -1, ns).repeat_interleave(nh // c.mamba_n_groups, 1) for p in y[:, di:].split(gn, 1))
        h = state[0][i].double() if state else torch.zeros(nh, hd, ns, dtype=torch.float64, device="cuda")
        o = torch.empty(hi - lo, nh, hd, 1, dtype=torch.float64, device="cuda")
        fed = u * step[lo:hi, :, None]
        for r in range(hi - lo):
            h = torch.baddbmm(h * decay[lo + r][:, None, None], fed[r][:, :, None], b[r][:, None])
            torch.bmm(h, g[r][:, :, None], out=o[r])
        out.append((o[..., 0] + u * t[f"{pre}.D"].double()[:, None]).flatten(1))
        hs.append(h)
        windows.append(after)
    y = (torch.cat(out) * F.silu(z)).view(len(x), c.mamba_n_groups, -1)
    y = (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + c.rms_norm_eps)).flatten(1) * t[f"{pre}.norm.weight"].double()
    return y @ _value(t[f"{pre}.out_proj.weight"]).t(), [torch.stack(hs), torch.stack(windows)]


def _gated(x, t, pre, e=None):
    """Gated unit; of expert ``e`` of a stack."""
    w = [t.get(f"{pre}.{n}_proj.weight", t.get(f"{pre}.{n}_proj")) for n in ("gate", "up", "down")]
    g, u, d = (_value(p, e) for p in w)
    return (F.silu(x @ g.t()) * (x @ u.t())) @ d.t()


def _experts(x, t, pre, c):
    p = (x @ _value(t[f"{pre}.gate.weight"]).t()).softmax(-1)
    w, ids = p.topk(c.num_experts_per_tok, -1)
    w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in ids.unique().tolist():
        r, k = (ids == e).nonzero(as_tuple=True)
        y.index_add_(0, r, _gated(x[r], t, f"{pre}.experts", e) * w[r, k][:, None])
    if f"{pre}.shared_expert_gate.weight" in t:
        y += _gated(x, t, f"{pre}.shared_expert") * torch.sigmoid(x @ _value(t[f"{pre}.shared_expert_gate.weight"]).t())
    return y


def exact(case, seed):
    """As :func:`run`; the cache is returned only by the new keys' and values' influence on the other outputs."""
    c = _config(case)
    t, (ids, past, had) = _checkpoint(case, seed), _inputs(case, seed)
    rows, ctx = _lengths(case)
    single = case["family"] == "mamba"
    x = t["backbone.embeddings.weight" if single else "model.embed_tokens.weight"][torch.cat(ids)].double()
    states, kv = {}, {}
    for i in range(c.num_hidden_layers):
        kind = c.layer_kind(i)
        pre = f"backbone.layers.{i}" if single else f"model.layers.{i}"
        h = _rms(x, t[f"{pre}.norm.weight" if single else f"{pre}.input_layernorm.weight"], c)
        mixer = f"{pre}.mixer" if single else f"{pre}.self_attn" if kind == "attention" else f"{pre}.linear_attn"
        if kind == "attention":
            y, _ = _attend(h, t, mixer, c, rows, ctx, past.get(i))
            kv[str(i)] = (None, None)
        elif kind == "gdn":
            y, states[str(i)] = _delta_net(h, t, mixer, c, rows, had.get(i))
        elif kind == "mamba2":
            y, states[str(i)] = _mamba(h, t, mixer, c, rows, had.get(i))
        else:
            y = (h @ _value(t[f"{mixer}.up_proj.weight"]).t()).relu().square() @ _value(t[f"{mixer}.down_proj.weight"]).t()
        x = x + y
        if not single:
            h = _rms(x, t[f"{pre}.post_attention_layernorm.weight"], c)
            x = x + (_experts(h, t, f"{pre}.mlp", c) if c.num_experts else _gated(h, t, f"{pre}.mlp"))
    hidden = _rms(x, t["backbone.norm_f.weight" if single else "model.norm.weight"], c)
    last = torch.tensor(rows, device="cuda").cumsum(0) - 1
    return dict(logits=hidden[last] @ _value(t["lm_head.weight"]).t(), hidden=hidden, kv=kv, states=states)
