"""What the engine is timed on: steps of whole models through the step function, and the sampling behind them.

A case is one step as a serving program runs it: some requests that decode one token behind the context they hold
(``decoders``, ``context``; ``ragged``: contexts from an eighth of ``context`` up to it), a portion of a prompt
(``portion`` rows behind ``past`` earlier tokens), or both side by side.  The models are the Qwen3 sizes of the
benchmarks, and the layer sizes that ``bench.py`` gives the Sagelorn design (attention over a window and over a latent,
retention) and the Kedavik design (selective scans; attention in chunks beside a delta rule), with feed-forwards for
every token: with routed experts, two correct implementations may choose another expert for the same row.  The engine
is warm, as a serving process is: the step's shape has been run and captured.  Weights are random (N(0, 0.02) and the
like, by tensor name), tokens uniform; a Qwen3 context is keys of N(0, 1), which is what normed keys are, and values
that share half their variance a channel, as the values of one text do; the other designs' contexts are prompts that the
engine itself has run.
"""
import math

import numpy as np
import torch

PAGE = 64
QWEN3 = {
    "0.6b": dict(hidden_size=1024, intermediate_size=3072, num_hidden_layers=28, num_attention_heads=16),
    "1.7b": dict(hidden_size=2048, intermediate_size=6144, num_hidden_layers=28, num_attention_heads=16),
}
DESIGN_LAYERS = 4            # one round of a design's mixers, or two
VOCAB = 151936
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}


def _step(name, model, decoders=0, context=0, portion=0, past=0, ragged=False, dtype="bf16", width=1024):
    case = {"kind": "step", "model": model, "width": width, "dtype": dtype, "decoders": decoders, "context": context,
            "ragged": ragged, "portion": portion, "past": past}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user's chat: a token at a time, where the launches and the latency of every kernel count
        _step("decode 1 0.6b", "0.6b", decoders=1, context=700),
        # the headline of bench.py: eight requests with contexts of 2048 tokens
        _step("decode 8 0.6b", "0.6b", decoders=8, context=2048),
        # a busy server at the larger size: requests of all ages
        _step("decode 64 ragged 1.7b", "1.7b", decoders=64, context=2304, ragged=True),
        # a long prompt in one step
        _step("prompt 2048 0.6b", "0.6b", portion=2048),
        # a question of a sentence or two: the time to its first token
        _step("prompt 129 0.6b", "0.6b", portion=129),
        # continuous batching under a budget of 512 rows: a portion of a prompt beside the others' decode tokens
        _step("mixed 512 1.7b", "1.7b", decoders=31, context=1500, ragged=True, portion=481, past=512),
        # the true 32-bit path, with which a user checks what the 16-bit one says
        _step("prompt 200 0.6b f32", "0.6b", portion=200, dtype="f32"),
        # the other designs: a prompt, and a decode step of a small batch
        _step("prompt 2048 sagelorn", "sagelorn", portion=2048),
        _step("decode 8 sagelorn", "sagelorn", decoders=8, context=1500),
        _step("prompt 1531 kedavik", "kedavik", portion=1531),
        _step("decode 16 kedavik", "kedavik", decoders=16, context=900),
        # a token for every row of a batch of 32: greedy, temperature, top-k and top-p side by side
        {"name": "sample 32", "kind": "sample", "rows": 32, "vocab": VOCAB},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(case):
    """Seconds that a pass cannot do without, roughly: what bounds the size of a drawn case."""
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / (1.2e15 if case.get("dtype") != "f32" else 6e13))


def _drawn(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "f32", "design", "design", "design", "sample"])
    if kind == "sample":
        return {"kind": "sample", "rows": _log_int(rng, 1, 64), "vocab": rng.choice([32768, VOCAB])}
    size = rng.choice(sorted(QWEN3))
    if kind == "decode":
        return _step(None, size, decoders=_log_int(rng, 1, 64), context=_log_int(rng, 16, 4096), ragged=rng.random() < 0.5)
    if kind == "prompt":
        past = 0 if rng.random() < 0.7 else _log_int(rng, 16, 2048)
        return _step(None, size, portion=_log_int(rng, 16, 2048), past=past)
    if kind == "mixed":
        return _step(None, size, decoders=_log_int(rng, 1, 32), context=_log_int(rng, 64, 2048), ragged=True,
                     portion=_log_int(rng, 16, 1024), past=rng.choice([0, 64, 512, 777]))
    if kind == "f32":
        if rng.random() < 0.5:
            return _step(None, "0.6b", decoders=_log_int(rng, 1, 8), context=_log_int(rng, 16, 1024), dtype="f32")
        return _step(None, "0.6b", portion=_log_int(rng, 16, 256), dtype="f32")
    design, width = rng.choice(["sagelorn", "kedavik"]), rng.choice([1024, 1024, 2048])
    if rng.random() < 0.5:
        return _step(None, design, portion=_log_int(rng, 16, 2048), width=width)
    return _step(None, design, decoders=_log_int(rng, 1, 32), context=_log_int(rng, 16, 2048), width=width)


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        case = _drawn(rng)
        if _cost(case) <= largest and case.get("decoders", 0) * case.get("context", 0) <= 65536:
            return case


# -- models -------------------------------------------------------------------------------------------------------------
def _config(case):
    """The config.json of the case's model."""
    width = case["width"]
    if case["model"] in QWEN3:
        return dict(QWEN3[case["model"]], architectures=["Qwen3ForCausalLM"], model_type="qwen3", torch_dtype="bfloat16",
                    hidden_act="silu", use_cache=True, tie_word_embeddings=True, num_key_value_heads=8, head_dim=128,
                    vocab_size=VOCAB, max_position_embeddings=40960, rope_theta=1000000.0, rms_norm_eps=1e-6,
                    bos_token_id=151643, eos_token_id=151645, attention_bias=False)
    heads = width // 128
    if case["model"] == "sagelorn":
        rot = {"dims": 64, "base": 1e6, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 2048}}
        decay = [1.0 - 2.0 ** (-5 - 5 * h / max(1, heads - 1)) for h in range(heads)]
        mixers = {"attention": {"heads": 2 * heads, "kv_heads": heads, "dim": 128, "vdim": 128, "rot": rot,
                                "scale": 128 ** -0.5, "mask": {"size": 1024}},
                  "latent_attention": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": width // 4 - 64,
                                       "q_rank": width // 2, "rot": {"dims": 64, "base": 1e4}, "scale": 192 ** -0.5,
                                       "mask": {"size": 1024}},
                  "retention": {"heads": heads, "dim": 128, "vdim": 128, "decay": decay}}
        kinds = ("attention", "latent_attention", "attention", "retention")
        layers = []
        for i in range(DESIGN_LAYERS):
            mixer = dict(mixers[kinds[i % 4]])
            if i % 4 == 2:                                  # every second attention layer reads the keys of the one before
                mixer["kv_from"] = i - 2
            layers.append({"type": kinds[i % 4], "mixer": mixer, "mlp": {"kind": "dense", "ff": 3 * width}})
        return {"architecture": "Sagelorn", "vocab": 32768, "width": width, "norm": {"eps": 1e-6}, "logit_scale": 0.5,
                "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 17}}, "layers": layers}
    mixers = {"mamba1": {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4},
              "parallel": {"left": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                    "rot": {"dims": 128, "base": 1e6}, "mask": {"size": 1024}},
                           "right": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4,
                                     "decay_rank": 128, "gate_rank": 128}, "left_scale": 0.8, "right_scale": 0.6}}
    return {"architecture": "Kedavik", "vocab": 32768, "width": width, "norm": {"eps": 1e-6}, "embedding": {"scale": 0.5},
            "residual_mult": 0.4,
            "layers": [{"type": kind, "mixer": mixers[kind], "mlp": {"kind": "dense", "ff": 4 * width} if kind == "parallel" else None}
                       for kind in [("mamba1", "parallel")[i % 2] for i in range(DESIGN_LAYERS)]]}


def _spec(case):
    from pih_b200.config import config_from_dict
    return config_from_dict(_config(case)).model_spec()


def _weights(case, seed):
    """Every tensor of the model by name, on the GPU, in the case's data type.  Matrices are N(0, 0.02) at a width of 1024
    and shrink with its root, the Qwen3 sub-layers' output matrices by the root of the number of sub-layers too, as models
    of their width and depth begin: otherwise rounding errors grow from layer to layer as no trained model lets them."""
    from pih_b200.models import expected_tensors
    config = _config(case)
    layers, sigma = config.get("num_hidden_layers"), 0.02 * math.sqrt(1024 / config.get("hidden_size", case["width"]))
    gen = torch.Generator("cuda").manual_seed(seed * 1000003 + 17)
    out = {}
    for name, info in expected_tensors(_spec(case)).items():
        t = torch.empty(tuple(info.shape), device="cuda", dtype=DTYPES[case["dtype"]])
        if info.init in ("conv", "unit_normal"):
            t.normal_(0.0, 0.5, generator=gen)
        elif info.init == "one_plus_normal":
            t.normal_(1.0, 0.02, generator=gen)
        else:
            last = name.endswith(("o_proj.weight", "down_proj.weight"))
            t.normal_(0.0, sigma / math.sqrt(2 * layers) if last else sigma, generator=gen)
        out[name] = t
    return out


def _requests(case):
    """(earlier tokens, rows of this step) of every request: the decoding ones, then the portion."""
    n, context = case["decoders"], case["context"]
    out = []
    for r in range(n):
        held = context
        if case["ragged"] and n > 1:
            held = max(1, int(context * (1.0 - 0.875 * r / (n - 1))) - (r * 37) % 61)
        out.append((held, 1))
    if case["portion"]:
        out.append((case["past"], case["portion"]))
    return out


def _tokens(case, seed):
    """Token ids of every request, the earlier ones and this step's."""
    rng = np.random.RandomState(seed % (1 << 31))
    vocab = VOCAB if case["model"] in QWEN3 else 32768
    return [rng.randint(0, vocab, past + rows).tolist() for past, rows in _requests(case)]


def _held_pages(case, seed, request, past):
    """Keys and values of a Qwen3 request's earlier tokens, a page after the other: [layers, pages, 2, kv heads, PAGE, 128]."""
    gen = torch.Generator("cuda").manual_seed(seed * 1000003 + 1000 + request)
    layers, like = QWEN3[case["model"]]["num_hidden_layers"], {"device": "cuda", "dtype": DTYPES[case["dtype"]]}
    pages = torch.empty(layers, -(-past // PAGE), 2, 8, PAGE, 128, **like).normal_(0.0, 1.0, generator=gen)
    pages[:, :, 1] += torch.empty(layers, 1, 8, 1, 128, **like).normal_(0.0, 1.0, generator=gen)
    pages[:, :, 1] *= 0.5
    return pages


# -- the passes -----------------------------------------------------------------------------------------------------------
def _prepare_sample(case, seed):
    from pih_b200.kernels import get_ops
    from pih_b200.sampling import SamplingParams
    from pih_b200.sampling.sampler import Sampler
    gen = torch.Generator("cuda").manual_seed(seed)
    rows, vocab, dev = case["rows"], case["vocab"], torch.device("cuda:0")
    logits = torch.empty(rows, vocab, device=dev).normal_(0.0, 2.5, generator=gen)
    kinds = [dict(temperature=0.7), dict(temperature=1.0, top_p=0.9), dict(temperature=0.8, top_k=40), dict(temperature=0.0),
             dict(temperature=0.7, top_k=200, top_p=0.95)]
    params = [SamplingParams(seed=seed % 9973 + r, **kinds[r % len(kinds)]) for r in range(rows)]
    return {"sampler": Sampler(get_ops(dev), vocab, dev), "logits": logits, "params": params,
            "ordinals": [5 + r for r in range(rows)], "suppressed": [[] for _ in range(rows)]}


def prepare(case, seed):
    if case["kind"] == "sample":
        return _prepare_sample(case, seed)
    from pih_b200.config import config_from_dict
    from pih_b200.engine import StepEntry
    from pih_b200.engine.factory import runner_for
    from pih_b200.kernels import get_ops
    from pih_b200.models import CausalLM
    from pih_b200.parts import Runtime

    dev = torch.device("cuda:0")
    model = CausalLM(config_from_dict(_config(case)).model_spec(), _weights(case, seed),
                     Runtime(dev, DTYPES[case["dtype"]], get_ops(dev)))
    requests, tokens = _requests(case), _tokens(case, seed)
    pages = sum(-(-(past + rows) // PAGE) for past, rows in requests)
    cache, runner = runner_for(model, page_size=PAGE, max_cache_tokens=pages * PAGE, max_requests=len(requests),
                               cuda_graphs=True)
    entries = []
    for r, (past, rows) in enumerate(requests):
        if past and case["model"] in QWEN3:
            cache.add_request(r)
            cache.append(r, past)
            cache.commit(r)
            table = np.empty((1, -(-past // PAGE)), dtype=np.int32)
            cache.fill_block_table(0, [r], table)
            cache.groups[0].kv[:, torch.from_numpy(table[0]).long().to(dev)] = _held_pages(case, seed, r, past)
        elif past:
            runner.step([StepEntry(r, tokens[r][:past], [])])
        entries.append(StepEntry(r, tokens[r][past:], [rows - 1]))
    state = {"runner": runner, "entries": entries, "held": [r for r, (past, _) in enumerate(requests) if past],
             "new": [r for r, (past, _) in enumerate(requests) if not past]}
    for _ in range(2):                                       # the step's shape is run and captured, as a warm engine has it
        run(state)
    return state


def run(state):
    """One step: its wanted rows' logits (or the sampled ids).  The requests stay as they were before it: a step whose
    tokens are not kept, as when several continuations of one context are scored; a prompt's request ends with it."""
    if "sampler" in state:
        return state["sampler"].sample_on_device(state["logits"], state["params"], state["ordinals"], state["suppressed"])
    runner = state["runner"]
    logits = runner.step(state["entries"], confirm=False)
    runner.discard(state["held"])
    for rid in state["new"]:
        runner.finish(rid)
    return logits


# -- what a pass cannot do without ------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 2.0 * case["rows"] * case["vocab"]}
    from pih_b200.models import expected_tensors
    size = 2 if case["dtype"] == "bf16" else 4
    requests = _requests(case)
    rows = sum(n for _, n in requests)
    shapes = {name: tuple(info.shape) for name, info in expected_tensors(_spec(case)).items()}
    table = "model.embed_tokens.weight" if case["model"] in QWEN3 else "embed"
    head = shapes[table]
    body = sum(math.prod(s) for name, s in shapes.items() if name not in (table, "head", "bigram"))
    nbytes = size * (body + math.prod(head) + rows * head[1]) + 4.0 * len(requests) * head[0]
    flops = 2.0 * rows * body + 2.0 * len(requests) * math.prod(head)

    def seen(window):
        """(keys read, scores formed) over all requests, for attention over the last ``window`` keys."""
        keys = scores = 0
        for past, n in requests:
            lens = np.minimum(np.arange(past + 1, past + n + 1), window or 1 << 40)
            keys += min(past + n, (window or 1 << 40) + n - 1)
            scores += int(lens.sum())
        return keys, scores

    def attention(heads, key, value, cached, window=0):
        keys, scores = seen(window)
        return size * keys * cached, 2.0 * scores * heads * (key + value)

    extra = []
    config = _config(case)
    if case["model"] in QWEN3:
        extra += [attention(16, 128, 128, 2 * 8 * 128)] * config["num_hidden_layers"]
    for layer in config.get("layers", ()):
        m = layer["mixer"]
        if layer["type"] == "attention":
            extra.append(attention(m["heads"], 128, 128, 2 * 128 * m["kv_heads"], 1024))
        elif layer["type"] == "latent_attention":
            extra.append(attention(m["heads"], 192, 128, m["kv_rank"] + 64, 1024))
        elif layer["type"] == "retention":
            extra.append((8.0 * len(requests) * m["heads"] * 128 * 128, 4.0 * rows * m["heads"] * 128 * 128))
        elif layer["type"] == "mamba1":
            extra.append((8.0 * len(requests) * m["inner"] * 16, 6.0 * rows * m["inner"] * 16))
        else:
            extra.append(attention(m["left"]["heads"], 128, 128, 2 * 128 * m["left"]["kv_heads"], 1024))
            extra.append((8.0 * len(requests) * m["right"]["heads"] * 128 * 128, 8.0 * rows * m["right"]["heads"] * 128 * 128))
    return {"bytes": nbytes + sum(b for b, _ in extra), "flops": flops + sum(f for _, f in extra)}


def tolerance(case):
    # the ids that exact masses and a counter-based generator give are the same whatever the order of the sums
    if case["kind"] == "sample":
        return "exact"
    # 32-bit: sums of 1024 to 3072 terms over 28 layers, about 1e-6 off the exact ones
    if case["dtype"] == "f32":
        return {"rel": 2e-5, "max": 2e-4}
    # 16-bit activations rounded at every operation of 8 or 28 layers: 0.6 to 1.2 % off the exact logits
    return {"rel": 0.03, "max": 0.3}


# -- the same in 64 bits, plainly -----------------------------------------------------------------------------------------
def _unit(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, positions, f, neighbours=False):
    """Rotates the first 2 * len(f) columns of x [T, ..., d] by positions * f: halves, or neighbouring columns, are pairs."""
    ang = (positions.double()[:, None] * f).reshape([x.shape[0]] + [1] * (x.dim() - 2) + [len(f)])
    c, s, n = torch.cos(ang), torch.sin(ang), 2 * len(f)
    u, v = (x[..., 0:n:2], x[..., 1:n:2]) if neighbours else (x[..., :n // 2], x[..., n // 2:n])
    both = (u * c - v * s, v * c + u * s)
    return torch.cat([torch.stack(both, -1).flatten(-2) if neighbours else torch.cat(both, -1), x[..., n:]], -1)


def _waves(rot):
    f = torch.tensor(rot["base"], dtype=torch.float64) ** (-torch.arange(0, rot["dims"], 2, dtype=torch.float64) / rot["dims"])
    if rot.get("scaling"):                                   # long waves are made longer, a blend of the two in between
        sc = rot["scaling"]
        t = ((sc["original"] * f / (2 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        f = (1 - t) * f / sc["factor"] + t * f
    return f.cuda()


def _attend(q, k, v, scale, pos, lo, sink=None):
    """q [T, H, d] at places ``pos`` over keys and values [K, G, d] of the places from lo[t] to pos[t]."""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device="cuda")
    at = torch.arange(k.shape[0], device="cuda")
    hidden = (at[None] > pos[:, None]) | (at[None] < lo[:, None])
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        out[:, h] = torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, h * G // H]
    return out.flatten(1)


def _qwen3(case, seed, w, tokens):
    c = _config(case)
    H, silu = c["num_attention_heads"], torch.nn.functional.silu
    f = _waves({"dims": 128, "base": c["rope_theta"]})
    out = []
    for r, (past, rows) in enumerate(_requests(case)):
        pos = torch.arange(past, past + rows, device="cuda")
        held = _held_pages(case, seed, r, past) if past else None
        x = w["model.embed_tokens.weight"][torch.tensor(tokens[r][past:], device="cuda")].double()
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            m = lambda t, name: t @ w[p + name + ".weight"].double().T  # noqa: E731
            n = _unit(x) * w[p + "input_layernorm.weight"].double()
            q = _turn(_unit(m(n, "self_attn.q_proj").view(rows, H, 128)) * w[p + "self_attn.q_norm.weight"].double(), pos, f)
            k = _turn(_unit(m(n, "self_attn.k_proj").view(rows, 8, 128)) * w[p + "self_attn.k_norm.weight"].double(), pos, f)
            v = m(n, "self_attn.v_proj").view(rows, 8, 128)
            if past:
                old = held[i].permute(1, 0, 3, 2, 4).reshape(2, -1, 8, 128)[:, :past].double()
                k, v = torch.cat([old[0], k]), torch.cat([old[1], v])
            if rows == 1:                                    # (one row: all heads at once)
                s = torch.einsum("gpd,kgd->gpk", q.view(8, H // 8, 128), k) * 128 ** -0.5
                a = torch.einsum("gpk,kgd->gpd", torch.softmax(s, -1), v).reshape(1, -1)
            else:
                a = _attend(q, k, v, 128 ** -0.5, pos, torch.zeros_like(pos))
            x = x + m(a, "self_attn.o_proj")
            n = _unit(x) * w[p + "post_attention_layernorm.weight"].double()
            x = x + m(silu(m(n, "mlp.gate_proj")) * m(n, "mlp.up_proj"), "mlp.down_proj")
        out.append(_unit(x[-1:]) * w["model.norm.weight"].double())
    return torch.cat(out) @ w["model.embed_tokens.weight"].double().T


def _sagelorn(case, w, rows_of):
    c, silu = _config(case), torch.nn.functional.silu
    b, out = c["embedding"]["bigram"], []
    for tokens in rows_of:
        t = torch.tensor(tokens, device="cuda")
        T, pos = len(tokens), torch.arange(len(tokens), device="cuda")
        pair = torch.cat([torch.tensor([b["buckets"]], device="cuda"), (t[:-1] * b["mul_prev"] + t[1:] * b["mul_cur"]) % b["buckets"]])
        x, kept = w["embed"][t] + w["bigram"][pair], {}
        for i, layer in enumerate(c["layers"]):
            m, H = layer["mixer"], layer["mixer"]["heads"]
            p = lambda t, name: t @ w[f"l{i}.mix.{name}"].T  # noqa: E731
            vec = lambda name: w[f"l{i}.mix.{name}"]  # noqa: E731
            if layer["type"] == "retention":
                q, k, v = (p(x, n).view(T, H, 128) for n in "qkv")
                decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")
                ages = (pos[:, None] - pos[None]).double()
                o = torch.empty(T, H, 128, dtype=torch.float64, device="cuda")
                for h in range(H):
                    far = torch.where(ages >= 0, decay[h] ** ages.clamp(min=0), 0.0)
                    o[:, h] = (q[:, h] @ k[:, h].T * 128 ** -0.5 * far) @ v[:, h]
                y = p(_unit(o).flatten(1) * silu(p(x, "g")), "o")
            elif layer["type"] == "latent_attention":
                f, R = _waves(m["rot"]), m["kv_rank"]
                down = p(x, "dkv")
                latent, turned = _unit(down[:, :R]) * vec("dkv.norm"), _turn(down[:, R:], pos, f, neighbours=True)
                q = p(_unit(p(x, "dq")) * vec("dq.norm"), "uq").view(T, H, 192)
                q = torch.cat([q[..., :128], _turn(q[..., 128:], pos, f, neighbours=True)], -1)
                k = torch.cat([p(latent, "uk").view(T, H, 128), turned[:, None].expand(T, H, 64)], -1)
                a = _attend(q, k, p(latent, "uv").view(T, H, 128), m["scale"], pos, pos - 1023)
                y = p(a * torch.sigmoid(p(x, "g")), "o")
            else:
                f = _waves(m["rot"])
                if "kv_from" not in m:
                    k = _turn((_unit(p(x, "k")) * vec("k.norm")).view(T, -1, 128), pos, f)
                    kept[i] = (k, p(x, "v").view(T, -1, 128))
                q = _turn((_unit(p(x, "q")) * vec("q.norm")).view(T, H, 128), pos, f)
                k, v = kept[m.get("kv_from", i)]
                y = p(_attend(q, k, v, m["scale"], pos, pos - 1023, vec("sink")), "o")
            x = x + _unit(y) * (1.0 + w[f"l{i}.norm1"])
            ff = lambda t, name: t @ w[f"l{i}.mlp.{name}"].T  # noqa: E731
            x = x + _unit(ff(silu(ff(x, "gate")) * ff(x, "up"), "down")) * (1.0 + w[f"l{i}.norm2"])
        out.append(_unit(x[-1:]) * (1.0 + w["final.norm"]))
    return torch.cat(out) @ w["head"].T * c["logit_scale"]


def _conv(x, taps, bias=None):
    """Causal convolution a channel of x [B, T, C], taps [C, n], then SiLU."""
    n = taps.shape[1]
    y = (torch.nn.functional.pad(x, (0, 0, n - 1, 0)).unfold(1, n, 1) * taps).sum(-1)
    return torch.nn.functional.silu(y if bias is None else y + bias)


def _kedavik(case, w, rows_of):
    c, silu, softplus = _config(case), torch.nn.functional.silu, torch.nn.functional.softplus
    t = torch.tensor(rows_of, device="cuda")                 # [B, T]: all requests hold as much
    B, T = t.shape
    pos = torch.arange(T, device="cuda")
    x = w["embed"][t] * c["embedding"]["scale"]
    for i, layer in enumerate(c["layers"]):
        n = _unit(x) * w[f"l{i}.norm1"]
        if layer["type"] == "mamba1":
            m = layer["mixer"]
            p = lambda a, name: a @ w[f"l{i}.mix.{name}"].T  # noqa: E731
            u, z = p(n, "in").split(m["inner"], -1)
            u = _conv(u, w[f"l{i}.mix.conv"], w[f"l{i}.mix.conv.b"])
            d, Bs, Cs = p(u, "x").split([m["dt_rank"], 16, 16], -1)
            d = softplus(p(d, "dt") + w[f"l{i}.mix.dt.b"])
            A, S = -torch.exp(w[f"l{i}.mix.A_log"]), torch.zeros(B, m["inner"], 16, dtype=torch.float64, device="cuda")
            y = torch.empty_like(u)
            for s in range(T):
                S = torch.exp(d[:, s, :, None] * A) * S + (d[:, s] * u[:, s])[..., None] * Bs[:, s, None]
                y[:, s] = (S @ Cs[:, s, :, None])[..., 0]
            y = p((y + w[f"l{i}.mix.D"] * u) * silu(z), "o")
        else:
            m = layer["mixer"]["left"]
            H, G, f = m["heads"], m["kv_heads"], _waves(m["rot"])
            p = lambda a, name: a @ w[f"l{i}.mix.left.{name}"].T  # noqa: E731
            att = torch.stack([_attend(_turn(p(r, "q").view(T, H, 128), pos, f), _turn(p(r, "k").view(T, G, 128), pos, f),
                                       p(r, "v").view(T, G, 128), m["scale"], pos, pos - pos % 1024) for r in n])
            att = att.view(B, T, H, 128) * torch.sigmoid(p(n, "g"))[..., None]
            y = layer["mixer"]["left_scale"] * p(att.flatten(2), "o")
            p = lambda a, name: a @ w[f"l{i}.mix.right.{name}"].T  # noqa: E731
            q, k, v = (_conv(p(n, r), w[f"l{i}.mix.right.{r}.conv"]).view(B, T, -1, 128) for r in "qkv")
            q, k = (a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
            q, k = (a.repeat_interleave(H // G, 2) for a in (q * 128 ** -0.5, k))
            g = softplus(p(p(n, "a1"), "a2") + w[f"l{i}.mix.right.dt_bias"]).view(B, T, H, 128)
            g, beta = torch.exp(-torch.exp(w[f"l{i}.mix.right.A_log"])[:, None] * g), torch.sigmoid(p(n, "b"))
            S, o = torch.zeros(B, H, 128, 128, dtype=torch.float64, device="cuda"), torch.empty_like(v)
            for s in range(T):
                S = g[:, s, ..., None] * S
                u = beta[:, s, :, None] * (v[:, s] - (k[:, s, :, None] @ S)[..., 0, :])
                S = S + k[:, s, ..., None] * u[..., None, :]
                o[:, s] = (q[:, s, :, None] @ S)[..., 0, :]
            o = (_unit(o) * w[f"l{i}.mix.right.norm"]).flatten(2) * torch.sigmoid(p(p(n, "g1"), "g2"))
            y = y + layer["mixer"]["right_scale"] * p(o, "o")
        x = x + c["residual_mult"] * y
        if layer["mlp"]:
            h = (_unit(x) * w[f"l{i}.norm2"]) @ w[f"l{i}.mlp.up"].T + w[f"l{i}.mlp.up.b"]
            x = x + c["residual_mult"] * (torch.nn.functional.gelu(h) @ w[f"l{i}.mlp.down"].T + w[f"l{i}.mlp.down.b"])
    return (_unit(x[:, -1]) * w["final.norm"]) @ w["head"].T


def exact(case, seed):
    if case["kind"] == "sample":
        return None                                          # ids
    w, tokens = _weights(case, seed), _tokens(case, seed)
    if case["model"] in QWEN3:
        return _qwen3(case, seed, w, tokens)
    w = {name: t.double() for name, t in w.items()}
    return (_sagelorn if case["model"] == "sagelorn" else _kedavik)(case, w, tokens)
