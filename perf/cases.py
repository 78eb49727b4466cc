"""The work this engine is used for, as cases that can be timed and checked.

A case is a dict of plain values.  All but the sampling cases are *served requests*: prompts go in, every request then
decodes a number of tokens, and what comes back are the 32-bit logits of every position whose next token a caller would
sample.  The tokens that follow a prompt are given (as in trace replay), so that two builds walk the same sequences.  A
pass goes the way generation goes: pages are reserved, a step of single decoded tokens runs through
``ModelRunner.decode_step`` and every other one through ``ModelRunner.step``, prompts are cut to the step budget and
join the tokens of the requests that already decode, and a request that is done gives its pages back.  A pass leaves
the engine as it found it, so it can be repeated.

Fields of a served case: ``design`` and ``dtype`` (which model), ``requests``, ``prompt_min``/``prompt_max`` (prompt
lengths, spread between the two), ``outputs`` (logits rows per request: the prompt's last position and ``outputs - 1``
decoded tokens), ``stagger`` (steps between two arrivals; 0: all at once) and ``max_len`` (the longest context the
Qwen3 model is configured for).  Fields of a sampling case: ``rows``, ``vocab``, ``temperature``, ``top_k``, ``top_p``.
"""
from __future__ import annotations

import math
import random
import shutil
import tempfile
from typing import Dict, List, Tuple

import torch

from cuinfer_b200 import SamplingParams
from cuinfer_b200.bench_designs import SIZES, bilolorn_config, neburax_config
from cuinfer_b200.config import EngineConfig, load_model_config
from cuinfer_b200.engine.runner import ModelRunner, StepEntry
from cuinfer_b200.parts import DecoderModel
from cuinfer_b200.sampling import Sampler
from cuinfer_b200.weights import open_weight_store, write_random_model

DEVICE = "cuda:0"
STEP_BUDGET = 8192        # tokens of one step, the engine's default
PAGE = 16                 # tokens of one cache page, the engine's default
VOCAB = 151936

# The benchmark's layer sizes; the 8B ones with eight of their 36 layers, so that preparing stays quick.
QWEN3 = {
    "qwen3_0.6b": dict(num_hidden_layers=28, hidden_size=1024, num_attention_heads=16, num_key_value_heads=8, head_dim=128,
                       intermediate_size=3072, vocab_size=VOCAB, tie_word_embeddings=True),
    "qwen3_8b": dict(num_hidden_layers=8, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                     intermediate_size=12288, vocab_size=VOCAB, tie_word_embeddings=False),
}


def _served(name, design, requests, prompt_min, prompt_max, outputs, stagger=0, dtype="bfloat16", max_len=4096):
    return {"name": name, "design": design, "dtype": dtype, "requests": requests, "prompt_min": prompt_min, "prompt_max": prompt_max,
            "outputs": outputs, "stagger": stagger, "max_len": max_len}


def listed() -> List[dict]:
    return [
        # one user, a short question and a short answer: a chain of small kernels, latency and launches
        _served("one_short", "qwen3_0.6b", 1, 37, 37, 24),
        # the reference's serving workload (1 024-token prompts) with eight requests in flight: mostly decode steps
        _served("eight_chats", "qwen3_0.6b", 8, 1024, 1024, 64),
        # long contexts at batch 8, the benchmark's headline batch: decode attention is half of a step
        _served("eight_long", "qwen3_0.6b", 8, 3900, 4000, 64),
        # a busy server: many requests of one size; decode steps of 64 rows, prompt steps at the full budget
        _served("many_chats", "qwen3_0.6b", 64, 1024, 1024, 32),
        # ragged requests that arrive one after the other: prompt portions beside decoded tokens in most steps, odd sizes
        _served("ragged_arrivals", "qwen3_0.6b", 27, 100, 1400, 40, stagger=2),
        # one prompt of the benchmark's prefill length, only the next token wanted (scoring, classification)
        _served("one_prompt", "qwen3_0.6b", 1, 2048, 2048, 1),
        # a long document in portions of the step budget, then an answer: attention over many keys in both directions
        _served("one_document", "qwen3_0.6b", 1, 11111, 11111, 24, max_len=16384),
        # the 8B layer sizes: large matrices, prompts and decode steps of a few requests
        _served("wide_layers", "qwen3_8b", 6, 300, 900, 24),
        # the 32-bit path (trace replay against another implementation): ragged prompts and decode steps
        _served("exact_32bit", "qwen3_0.6b", 3, 60, 300, 12, dtype="float32"),
        # attention over a cached latent and experts chosen by the token's id
        _served("latent_experts", "bilolorn", 8, 500, 700, 32),
        # state-space and gated linear recurrences: state instead of keys and values
        _served("recurrent", "neburax", 8, 500, 700, 32),
        # sampling with temperature and a nucleus over a large vocabulary, a row for each request of a step
        {"name": "nucleus", "design": "sampler", "rows": 32, "vocab": VOCAB, "temperature": 0.8, "top_k": 0, "top_p": 0.9},
    ]


def _log_uniform(rng: random.Random, low: int, high: int) -> int:
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng: random.Random) -> dict:
    """Another case of the same ranges: a design by how much it is used, 1 to 64 requests (fewer where the model is wide
    or 32-bit), prompts from a few tokens to the longest context, 1 to 48 outputs, arrivals at once or one by one."""
    kind = rng.choices(["qwen3_0.6b", "qwen3_8b", "float32", "bilolorn", "neburax", "sampler"], [6, 2, 1, 1, 1, 1])[0]
    if kind == "sampler":
        return {"design": "sampler", "rows": _log_uniform(rng, 1, 128), "vocab": rng.choice([VOCAB, 32768, 50257]),
                "temperature": round(rng.uniform(0.3, 1.2), 2), "top_k": rng.choice([0, 0, 20, 50]), "top_p": round(rng.uniform(0.8, 1.0), 3)}
    most_requests, most_tokens, most_prompt = {"qwen3_0.6b": (64, 49152, 4000), "qwen3_8b": (16, 6144, 2048), "float32": (8, 700, 400),
                                               "bilolorn": (16, 6144, 2048), "neburax": (16, 6144, 2048)}[kind]
    requests = _log_uniform(rng, 1, most_requests)
    longest = _log_uniform(rng, 16, min(most_prompt, most_tokens // requests))
    shortest = max(5, int(longest * rng.choice([1.0, 0.8, 0.3])))
    case = _served("", "qwen3_0.6b" if kind == "float32" else kind, requests, shortest, longest,
                   _log_uniform(rng, 1, 12 if kind == "float32" else 48), rng.choice([0, 0, 1, 2]),
                   "float32" if kind == "float32" else "bfloat16")
    if kind == "qwen3_0.6b" and requests == 1 and rng.random() < 0.3:
        case.update(prompt_min=4001, prompt_max=_log_uniform(rng, 4001, 11000), max_len=16384)
        case["prompt_min"] = case["prompt_max"]
    del case["name"]
    return case


# ---- what a case does, from its fields alone ----------------------------------------------------------------------------
def _prompt_lengths(case: dict) -> List[int]:
    rng = random.Random(f"{case['requests']}:{case['prompt_min']}:{case['prompt_max']}")
    return [rng.randint(case["prompt_min"], case["prompt_max"]) for _ in range(case["requests"])]


def _plan(case: dict) -> List[List[Tuple[int, int, int, bool]]]:
    """The steps of a pass: per step ``(request, first token, tokens, wants its last position's logits)``.  The requests
    that decode come first, then prompts in order of arrival, cut to what is left of the step budget."""
    lengths, outputs = _prompt_lengths(case), case["outputs"]
    ends = [n + outputs - 1 for n in lengths]
    done = [0] * len(lengths)
    steps, now = [], 0
    while any(d < e for d, e in zip(done, ends)):
        left, step = STEP_BUDGET, []
        for prompts in (False, True):
            for r, (d, e) in enumerate(zip(done, ends)):
                if d >= e or (d < lengths[r]) != prompts or r * case["stagger"] > now or left <= 0:
                    continue
                n = min(lengths[r] - d, left) if prompts else 1
                step.append((r, d, n, d + n >= lengths[r]))
                left -= n
        for r, d, n, _ in step:
            done[r] = d + n
        now += 1
        if step:
            steps.append(step)
    return steps


def _config(case: dict) -> dict:
    if case["design"] in QWEN3:
        return dict(QWEN3[case["design"]], architectures=["Qwen3ForCausalLM"], rope_theta=1000000.0, rms_norm_eps=1e-6,
                    max_position_embeddings=case["max_len"], torch_dtype=case["dtype"])
    if case["design"] == "bilolorn":
        return bilolorn_config(SIZES["large"])
    # Neburax with a dense feed-forward in every layer: a learned router's near-ties would make one rounding choose
    # other experts than the next
    config = neburax_config(SIZES["large"])
    for layer in config["layers"]:
        layer["mlp"] = {"kind": "dense", "ff": SIZES["large"]["ff"]}
    return config


def _write_model(case: dict, seed: int) -> str:
    """A model folder without tensors: the weights are drawn on the device while they are loaded."""
    gains = {"embed": 50.0} if case["design"] == "neburax" else None
    return write_random_model(tempfile.mkdtemp(prefix="cuinfer_b200_case_"), _config(case), seed, std=0.02, gain_std=0.05,
                              dtype=case["dtype"], gains=gains, generator="counter", materialize=False)


def _tokens(case: dict, seed: int) -> List[List[int]]:
    gen = torch.Generator().manual_seed(1000003 * seed + 17)
    vocab = VOCAB if case["design"] in QWEN3 else SIZES["large"]["vocab"]
    return [torch.randint(0, vocab, (n + case["outputs"] - 1,), generator=gen).tolist() for n in _prompt_lengths(case)]


def _sampling_inputs(case: dict, seed: int):
    """Logits as a trained model has them: a broad floor and a few likely tokens a row."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    logits = torch.randn((case["rows"], case["vocab"]), generator=gen, device=DEVICE) * 2.0
    at = torch.randint(0, case["vocab"], (case["rows"], 64), generator=gen, device=DEVICE)
    logits.scatter_add_(1, at, torch.rand((case["rows"], 64), generator=gen, device=DEVICE) * 10.0)
    return logits


class _Served:
    def __init__(self, case: dict, seed: int) -> None:
        lengths = _prompt_lengths(case)
        pages = sum((n + case["outputs"] + PAGE) // PAGE + 1 for n in lengths) + 8
        folder = _write_model(case, seed)
        try:
            self.runner = ModelRunner(folder, EngineConfig(
                model_path=folder, block_size=PAGE, dtype=case["dtype"], num_blocks=pages, max_num_seqs=max(8, case["requests"]),
                max_num_scheduled_tokens=STEP_BUDGET, device=DEVICE))
        finally:
            shutil.rmtree(folder, ignore_errors=True)
        tokens = _tokens(case, seed)
        last = [n + case["outputs"] - 1 for n in lengths]
        self.steps = []
        self.rows = 0
        for step in _plan(case):
            entries = [StepEntry(r, tokens[r][d:d + n], [n - 1] if wanted else []) for r, d, n, wanted in step]
            single = all(n == 1 and wanted for _, _, n, wanted in step)
            self.steps.append((entries, single, [r for r, d, n, _ in step if d + n == last[r]]))
            self.rows += sum(len(e.want) for e in entries)


def prepare(case: dict, seed: int):
    """A loaded model with its cache pool and the requests' tokens on the host; as a server that has run this kind of
    work before, it has recorded the CUDA graphs of its step sizes."""
    if case["design"] == "sampler":
        params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=seed)] * case["rows"]
        return Sampler(seed, torch.device(DEVICE), case["rows"]), _sampling_inputs(case, seed), params, list(range(case["rows"]))
    state = _Served(case, seed)
    run(state)
    run(state)
    return state


def run(state):
    if not isinstance(state, _Served):
        sampler, logits, params, keys = state
        return sampler.sample(logits, params, keys, keys)
    runner = state.runner
    out = torch.empty((state.rows, runner.vocab_size), dtype=torch.float32, device=DEVICE)
    at = 0
    for entries, single, finished in state.steps:
        for e in entries:
            if not runner.reserve(e.request_id, len(e.tokens)):
                raise RuntimeError("the cache pool is too small for the case")
        logits = runner.decode_step(entries) if single and runner.can_use_graph(entries) else runner.step(entries)
        out[at:at + logits.shape[0]].copy_(logits)          # the next step writes over a step's logits
        at += logits.shape[0]
        for r in finished:
            runner.release(r)
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _model(case: dict) -> DecoderModel:
    folder = _write_model(case, 0)
    try:
        architecture, config = load_model_config(folder)
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    return DecoderModel(architecture.spec(config), torch.float32 if case["dtype"] == "float32" else torch.bfloat16)


def work(case: dict) -> Dict[str, float]:
    """Per step: the weights once (of the experts those that its tokens choose), the keys and values of every request's
    context once, the new ones written, the wanted logits written."""
    if case["design"] == "sampler":
        return {"bytes": 4.0 * case["rows"] * (case["vocab"] + 1), "flops": 0.0}
    width = 4 if case["dtype"] == "float32" else 2
    matrices, experts, table = 0, 0, 0
    model = _model(case)
    for spec in model.tensors():
        n = math.prod(spec.shape)
        if spec.integer:
            continue
        if spec.name == model.spec.embedding_name:
            table = n
        elif ".mlp.e" in spec.name:
            experts += n
        else:
            matrices += n
    head = table if model.tied else 0
    lm_head = model.vocab_size * model.hidden_size
    chosen = 0.0
    if case["design"] in QWEN3:
        q = QWEN3[case["design"]]
        layers, heads, qk, v = q["num_hidden_layers"], q["num_attention_heads"], q["head_dim"], q["head_dim"]
        kv_row = 2 * layers * q["num_key_value_heads"] * q["head_dim"] * width
        chunk = 0
    else:
        s = SIZES["large"]
        heads = s["heads"]
        if case["design"] == "bilolorn":
            layers, qk, v, chunk = s["layers"], s["kv_rank"] + s["rot_dim"], s["kv_rank"], 0
            kv_row = layers * qk * width
            chosen = s["top"] / s["experts"]
        else:
            layers, qk, v, chunk = s["layers"] // 4, s["head_dim"], s["head_dim"], s["window"]
            kv_row = 2 * layers * s["kv_heads"] * s["head_dim"] * width
    nbytes = flops = 0.0
    for step in _plan(case):
        tokens, rows = sum(n for _, _, n, _ in step), sum(w for *_, w in step)
        touched = experts * (1.0 - (1.0 - chosen) ** tokens)
        nbytes += (matrices - (0 if model.tied or rows else lm_head) + (head if rows else 0) + touched) * width
        nbytes += 4.0 * rows * model.vocab_size + tokens * model.hidden_size * width
        flops += 2.0 * tokens * (matrices - (0 if model.tied else lm_head) + experts * chosen) + 2.0 * rows * lm_head
        for _, first, n, _ in step:
            begin = first // chunk * chunk if chunk else 0
            pairs = sum(min(p + 1, p % chunk + 1) for p in range(first, first + n)) if chunk else n * first + n * (n + 1) / 2
            nbytes += (first + n - begin + n) * kv_row
            flops += 2.0 * pairs * heads * (qk + v) * layers
            if case["design"] == "neburax":          # the recurrences' state, read and written
                inner, state = 2 * s["width"], 128
                nbytes += 2 * 4.0 * (s["layers"] - layers) * inner * state
                flops += 5.0 * n * (s["layers"] - layers) * inner * state
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict):
    """Relative to the result's 2-norm.  The models in bfloat16 round every projection's output, the softmax weights and
    the cached rows to eight bits of mantissa in every layer; the sums are 32-bit.  About four times what the same path
    differs by when other kernels compute it (library products for own ones, another attention): 0.6B sizes 0.6 %, 8B
    sizes 1.4 %, Bilolorn 0.8 %, Neburax 0.6 %; the 32-bit path is 7e-7 from the result in 64 bits."""
    if case["design"] == "sampler":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.36} if case["design"] == "qwen3_8b" else {"rel": 0.025, "max": 0.16}


# ---- the same in 64 bits, plainly ---------------------------------------------------------------------------------------
def _weights(case: dict, seed: int) -> Tuple[dict, Dict[str, torch.Tensor]]:
    model = _model(case)
    folder = _write_model(case, seed)
    store = open_weight_store(folder, model.dtype, torch.device(DEVICE))
    try:
        specs = model.tensors()
        store.check(specs)
        return _config(case), {s.name: store.get(s) if s.integer else store.get(s).double() for s in specs}
    finally:
        store.close()
        shutil.rmtree(folder, ignore_errors=True)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w + b


def _silu(x):
    return x * torch.sigmoid(x)


def _angles(T: int, base: float, dims: int):
    """32-bit frequencies and angles, as the engine's tables have them; cosine and sine in 64 bits."""
    exponent = torch.arange(dims // 2, dtype=torch.float32) * 2.0 / float(dims)
    freq = 1.0 / torch.pow(torch.tensor(float(base), dtype=torch.float32), exponent)
    angle = (torch.arange(T, dtype=torch.float32)[:, None] * freq[None, :]).to(DEVICE).double()
    return torch.cos(angle), torch.sin(angle)


def _attend(q, k, v, scale, chunk=0, sink=None):
    """q [T, H, d], k and v [T, G, *]; causal, inside chunks if given; ``sink [H]`` joins the denominator."""
    T, H, _ = q.shape
    share = H // k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for a in range(0, T, 2048):
        b = min(T, a + 2048)
        i, j = torch.arange(a, b, device=q.device)[:, None], torch.arange(b, device=q.device)[None, :]
        hidden = (j > i) | ((j // chunk != i // chunk) if chunk else False)
        for h in range(H):
            s = (q[a:b, h] @ k[:b, h // share].T * scale).masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], 1)
            out[a:b, h] = torch.softmax(s, -1)[:, :b] @ v[:b, h // share]
    return out


def _qwen3(cfg, t, ids):
    H, G, d, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    T = len(ids)
    c, s = (z[:, None, :] for z in _angles(T, cfg["rope_theta"], d))

    def rotate(u):
        a, b = u[..., :d // 2], u[..., d // 2:]
        return torch.cat((a * c - b * s, b * c + a * s), -1)

    x = t["model.embed_tokens.weight"][ids]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * t[p + "input_layernorm.weight"]
        q = rotate(_rms((h @ t[p + "self_attn.q_proj.weight"].T).view(T, H, d), eps) * t[p + "self_attn.q_norm.weight"])
        k = rotate(_rms((h @ t[p + "self_attn.k_proj.weight"].T).view(T, G, d), eps) * t[p + "self_attn.k_norm.weight"])
        v = (h @ t[p + "self_attn.v_proj.weight"].T).view(T, G, d)
        x = x + _attend(q, k, v, d ** -0.5).reshape(T, H * d) @ t[p + "self_attn.o_proj.weight"].T
        h = _rms(x, eps) * t[p + "post_attention_layernorm.weight"]
        x = x + (_silu(h @ t[p + "mlp.gate_proj.weight"].T) * (h @ t[p + "mlp.up_proj.weight"].T)) @ t[p + "mlp.down_proj.weight"].T
    return _rms(x, eps) * t["model.norm.weight"], t["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]


def _bilolorn(cfg, t, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = t["embed"][ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.", layer["mixer"], layer["mlp"]
        H, dn, dr, dv, rk = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        c, s = _angles(T, m["rot"]["base"], m["rot"]["dims"])

        def rotate(u):                        # neighbours pair up; u [T, heads, dr], all of it rotated
            a, b, cc, ss = u[..., 0::2], u[..., 1::2], c[:, None], s[:, None]
            return torch.stack((a * cc - b * ss, b * cc + a * ss), -1).flatten(-2)

        h = _layer_norm(x, t[p + "norm1"], t[p + "norm1.b"], eps)
        w = {k[len(p) + 4:]: v for k, v in t.items() if k.startswith(p + "mix.")}
        q = ((_rms(h @ w["dq"].T, eps) * w["dq.norm"]) @ w["uq"].T).view(T, H, dn + dr)
        down = h @ w["dkv"].T
        latent = _rms(down[:, :rk], eps) * w["dkv.norm"]
        k_rot = rotate(down[:, None, rk:]).expand(T, H, dr)
        k = torch.cat(((latent @ w["uk"].T).view(T, H, dn), k_rot), -1)
        q = torch.cat((q[..., :dn], rotate(q[..., dn:])), -1)
        y = _attend(q, k, (latent @ w["uv"].T).view(T, H, dv), m["scale"], sink=w["sink"]).reshape(T, H * dv)
        y = (y * torch.sigmoid(h @ w["g"].T)) @ w["o"].T
        x = x + _layer_norm(y, t[p + "norm1b"], t[p + "norm1b.b"], eps)
        h = _layer_norm(x, t[p + "norm2"], t[p + "norm2.b"], eps)
        p += "mlp."
        if f["kind"] == "dense":
            y = torch.relu(h @ t[p + "up"].T) ** 2 @ t[p + "down"].T
        else:
            def expert(rows, e):
                return (_silu(rows @ t[p + e + "gate"].T) * (rows @ t[p + e + "up"].T)) @ t[p + e + "down"].T

            y = expert(h, "shared.")
            chosen, top = t[p + "table"][ids].long(), f["router"]["top"]
            for e in range(f["router"]["experts"]):
                rows = (chosen == e).any(1).nonzero()[:, 0]
                if rows.numel():
                    y[rows] += expert(h[rows], f"e{e}.") / top
        x = x + _layer_norm(y, t[f"l{i}.norm2b"], t[f"l{i}.norm2b.b"], eps)
    return _layer_norm(x, t["final.norm"], t["final.norm.b"], eps), t["head"]


def _causal_conv(x, taps, bias):
    T, K = x.shape[0], taps.shape[1]
    y = bias.expand_as(x).clone()
    for j in range(min(K, T)):
        y[j:] += taps[:, K - 1 - j] * x[:T - j]
    return y


def _softplus(x):
    return torch.clamp_min(x, 0.0) + torch.log1p(torch.exp(-x.abs()))


def _state_space(h, w, m, eps):
    T, H, P, N, G = h.shape[0], m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    z, xbc, dt = torch.split(h @ w["in"].T, [inner, inner + 2 * G * N, H], dim=1)
    x, B, C = torch.split(_silu(_causal_conv(xbc, w["conv"], w["conv.b"])), [inner, G * N, G * N], dim=1)
    x, B, C, dt = x.reshape(T, H, P), B.reshape(T, G, N), C.reshape(T, G, N), _softplus(dt + w["dt_bias"])
    total = torch.cumsum(-torch.exp(w["A_log"]) * dt, 0)              # log of the decay from the start to each token
    later = torch.ones((T, T), dtype=torch.bool, device=h.device).triu(1)
    y = torch.empty_like(x)
    products = [C[:, g] @ B[:, g].T for g in range(G)]
    for a in range(H):
        decay = torch.exp((total[:, None, a] - total[None, :, a]).masked_fill_(later, -math.inf))
        y[:, a] = (products[a // (H // G)] * decay) @ (dt[:, a, None] * x[:, a]) + w["D"][a] * x[:, a]
    y = (y.reshape(T, inner) * _silu(z)).view(T, m["norm_groups"], -1)
    return (_rms(y, eps).reshape(T, inner) * w["norm"]) @ w["o"].T


def _linear_recurrence(h, w):
    y = h @ w["y"].T + w["y.b"]
    y = 0.5 * y * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (y + 0.044715 * y ** 3)))
    u = _causal_conv(h @ w["x"].T + w["x.b"], w["conv"], w["conv.b"])
    n, b = w["ra.b"].shape

    def gate(name):
        return torch.sigmoid(torch.cat([u[:, i * b:(i + 1) * b] @ w[name][i].T + w[name + ".b"][i] for i in range(n)], 1))

    log_a = -8.0 * gate("ra") * _softplus(w["lam"])
    a, step = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * gate("ri") * u
    s, out = torch.zeros_like(u[0]), torch.empty_like(u)
    for i in range(u.shape[0]):
        s = a[i] * s + step[i]
        out[i] = s
    return (out * y) @ w["o"].T


def _neburax(cfg, t, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = t["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        w = {k[len(p) + 4:]: v for k, v in t.items() if k.startswith(p + "mix.")}
        if layer["type"] == "mamba2":
            y = _state_space(x, w, m, eps)
        else:
            left = m["left"]
            q = (_rms(x @ w["left.q"].T, eps) * w["left.q.norm"]).view(T, left["heads"], left["dim"])
            k = (_rms(x @ w["left.k"].T, eps) * w["left.k.norm"]).view(T, left["kv_heads"], left["dim"])
            v = (x @ w["left.v"].T).view(T, left["kv_heads"], left["vdim"])
            y = _attend(q, k, v, left["scale"], chunk=left["mask"]["size"]).reshape(T, -1) @ w["left.o"].T
            right = {k[6:]: v for k, v in w.items() if k.startswith("right.")}
            y = m["left_scale"] * y + m["right_scale"] * _linear_recurrence(x, right)
        x = x + _rms(y, eps) * t[p + "norm1"]
        y = torch.relu(x @ t[p + "mlp.up"].T + t[p + "mlp.up.b"]) ** 2 @ t[p + "mlp.down"].T + t[p + "mlp.down.b"]
        x = x + _rms(y, eps) * t[p + "norm2"]
    return _rms(x, eps) * t["final.norm"], t["embed"]


def exact(case: dict, seed: int):
    """The logits in 64 bits: every request's whole sequence at once, without cache, batch or steps."""
    if case["design"] == "sampler":
        return None
    cfg, t = _weights(case, seed)
    forward = {"bilolorn": _bilolorn, "neburax": _neburax}.get(case["design"], _qwen3)
    lengths = _prompt_lengths(case)
    rows = []
    for r, ids in enumerate(_tokens(case, seed)):
        hidden, head = forward(cfg, t, torch.tensor(ids, device=DEVICE))
        rows.append((hidden[lengths[r] - 1:], head))
    at, out = [0] * len(rows), []
    for step in _plan(case):
        for r, _, _, wanted in step:
            if wanted:
                out.append(rows[r][0][at[r]])
                at[r] += 1
    return torch.stack(out) @ rows[0][1].T
