"""What serving costs: the workloads that the speed of this package is judged by.

A pass is what a serving program does with a batch of requests that arrive together: it admits them, brings their prompts
in portions of ``chunk`` tokens under a budget of ``budget`` tokens a step (prompt portions beside the decoded rows of the
requests that are further on, as the scheduler builds its steps), decodes ``new`` tokens for each and lets them go.  Steps go
through :meth:`Stepper.step` with the :class:`Sampler`, and steps of decoded rows alone through :meth:`Stepper.launch_decode`,
launched one ahead of the read-back of their tokens.  The continuations are given (every request decodes tokens that the seed
draws, as in scoring), so that two correct builds run the same rows; the logits of every decoded place come back beside the
tokens that the sampler chose there.

The models have the layer sizes that ``bench.py`` uses and random weights, drawn once for a model and kept as a server keeps
them: Llama at the 1B sizes (the headline), at the 8B sizes with 8 of 32 layers, and in 32-bit; and two of the other designs,
Kazodra and Tibivik, which between them run latent, two-map, windowed and chunked attention and all four matrix-state
recurrences.  (Designs that route rows to experts are left out: where two experts score nearly alike, two correct builds choose
differently, and their logits cannot be held against each other.)
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

# ----------------------------------------------------------------------------- models

LLAMA = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_act": "silu", "torch_dtype": "bfloat16",
    "attention_bias": False, "mlp_bias": False, "num_hidden_layers": 16, "hidden_size": 2048, "num_attention_heads": 32,
    "num_key_value_heads": 8, "head_dim": 64, "intermediate_size": 8192, "vocab_size": 128256,
    "max_position_embeddings": 131072, "rope_theta": 500000.0,
    "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                     "original_max_position_embeddings": 8192},
    "rms_norm_eps": 1e-5, "tie_word_embeddings": True, "bos_token_id": 128000, "eos_token_id": [128001],
}
LLAMA_8B = dict(LLAMA, hidden_size=4096, head_dim=128, intermediate_size=14336, tie_word_embeddings=False,
                rope_scaling=dict(LLAMA["rope_scaling"], factor=8.0))
VOCAB = 32768                                   # of the two other designs, as in their benchmark


def kazodra_config():
    """Linear attention with a decay twice, attention with two score maps, attention over a latent under a window, and over
    again; ten stored layers, the middle six walked twice."""
    light = {"type": "lightning", "mixer": {"heads": 16, "dim": 128, "vdim": 128,
                                            "decay": [1.0 - 2.0 ** (-5.0 - 3.0 * h / 15) for h in range(16)]}}
    maps = {"type": "attention", "mixer": {
        "heads": 16, "kv_heads": 4, "dim": 64, "vdim": 128, "diff": 0.8, "scale": 64 ** -0.5,
        "rot": {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    latent = {"type": "latent_attention", "mixer": {
        "heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "mask": {"size": 512}, "scale": 192 ** -0.5,
        "rot": {"dims": 64, "base": 10000.0}}}
    order = [light, light, maps, latent]
    return {"architecture": "Kazodra", "torch_dtype": "bfloat16", "width": 2048, "vocab": VOCAB, "norm": {"eps": 1e-5},
            "token_side": {"dim": 128}, "loop": {"start": 2, "stop": 8, "times": 2},
            "layers": [dict(order[i % 4], mlp={"kind": "dense", "ff": 8192}) for i in range(10)]}


def tibivik_config():
    """State-space layers in turn with layers of two sides: chunked attention beside the gated delta rule, window attention
    beside a matrix memory; ten stored layers, the middle six walked twice; four copies of the stream."""
    space = {"type": "mamba2", "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}}
    left = {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "scale": 64 ** -0.5, "mask": {"size": 512}}
    chunked = {"type": "parallel_2", "mixer": {
        "left": left, "right": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4},
        "left_scale": 1.0, "right_scale": 1.0}}
    windowed = {"type": "parallel", "mixer": {
        "left": dict(left, rot={"dims": 32, "base": 500000.0}),
        "right": {"heads": 16, "dim": 128, "vdim": 128, "gate_cap": 15.0}, "left_scale": 1.0, "right_scale": 1.0}}
    order = [space, chunked, space, windowed]
    return {"architecture": "Tibivik", "torch_dtype": "bfloat16", "width": 2048, "vocab": VOCAB, "streams": 4,
            "norm": {"eps": 1e-5}, "embedding": {"bigram": {"buckets": 65536, "mul_prev": 31, "mul_cur": 7}},
            "loop": {"start": 2, "stop": 8, "times": 2},
            "layers": [dict(order[i % 4], mlp={"kind": "dense", "ff": 8192}) for i in range(10)]}


def config_of(case):
    if case["model"] == "llama-1b":
        return dict(LLAMA)
    if case["model"] == "llama-8b":
        return dict(LLAMA_8B, num_hidden_layers=8)
    return {"kazodra-1b": kazodra_config, "tibivik-1b": tibivik_config}[case["model"]]()


def vocabulary(config):
    return config.get("vocab_size") or config["vocab"]


# ----------------------------------------------------------------------------- cases


def listed():
    def case(name, model, requests, shortest, longest, new, chunk, dtype="bfloat16"):
        return {"name": name, "model": model, "dtype": dtype, "requests": requests, "shortest": shortest, "longest": longest,
                "new": new, "chunk": chunk, "budget": 4096}

    return [
        # the time to the first token of one short question: the smallest call, launches and latency alone
        case("first_token", "llama-1b", 1, 23, 23, 1, 512),
        # eight short questions at once, as a chat server meets them: one ragged step of prompts, then decoding
        case("chat_8", "llama-1b", 8, 20, 25, 24, 512),
        # one user at a time: decoding a single row
        case("single", "llama-1b", 1, 180, 180, 32, 512),
        # the headline shape: a batch of eight behind prompts of about two thousand tokens
        case("decode_8_at_2k", "llama-1b", 8, 1900, 2048, 64, 2048),
        # a busy server: 64 ragged prompts come in beside the rows that decode already
        case("busy_64", "llama-1b", 64, 40, 300, 24, 512),
        # a prompt of 2,048 tokens in one step
        case("prompt_2048", "llama-1b", 1, 2048, 2048, 1, 2048),
        # a long document at the 8B layer sizes, an odd length, in portions of 2,048
        case("document_8b", "llama-8b", 1, 12345, 12345, 8, 2048),
        # the 32-bit path, for users who check a model exactly
        case("exact_f32", "llama-1b", 4, 60, 130, 8, 512, "float32"),
        # Kazodra: a long prompt; a small batch that decodes
        case("kazodra_prompt", "kazodra-1b", 1, 2000, 2000, 1, 2048),
        case("kazodra_decode_8", "kazodra-1b", 8, 200, 300, 24, 512),
        # Tibivik: a long prompt; a larger batch that decodes
        case("tibivik_prompt", "tibivik-1b", 1, 2048, 2048, 1, 2048),
        case("tibivik_decode_32", "tibivik-1b", 32, 30, 120, 24, 512),
    ]


def draw(rng):
    def log_int(low, high):
        return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))

    model, dtype = rng.choice([("llama-1b", "bfloat16")] * 4 + [("llama-8b", "bfloat16"), ("llama-1b", "float32"),
                                                                ("kazodra-1b", "bfloat16"), ("kazodra-1b", "bfloat16"),
                                                                ("tibivik-1b", "bfloat16"), ("tibivik-1b", "bfloat16")])
    most = 16 if dtype == "float32" else 64
    requests = log_int(1, most)
    rows = {"float32": 500}.get(dtype, 12000 if model.startswith("llama") else 4000)     # prompt tokens in all
    longest = log_int(8, max(16, min(8000 if model.startswith("llama") else 2500, rows // requests)))
    return {"model": model, "dtype": dtype, "requests": requests, "shortest": rng.randint(1, longest), "longest": longest,
            "new": log_int(1, 8 if dtype == "float32" else 24), "chunk": rng.choice([512, 512, 2048]), "budget": 4096}


def lengths_of(case):
    """The requests' prompt lengths: part of the case, whatever the seed."""
    rng = random.Random("%(requests)d %(shortest)d %(longest)d" % case)
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]


def schedule(case):
    """The steps of a pass, each a list of ``(request, first token, tokens)``: prompt portions first, full ones ahead, then the
    decoded rows.  ``tokens`` counts from the prompt's start on into the continuation."""
    prompts, steps = lengths_of(case), []
    done = [0] * len(prompts)
    while True:
        budget, rows, portions = case["budget"], [], []
        for r, p in enumerate(prompts):
            if p <= done[r] < p + case["new"] - 1 and budget:
                rows.append((r, done[r], 1))
                budget -= 1
        for r, p in enumerate(prompts):
            if done[r] < p and budget:
                count = min(p - done[r], case["chunk"], budget)
                portions.append((r, done[r], count))
                budget -= count
        portions.sort(key=lambda part: part[2] != case["chunk"])
        step = portions + rows
        if not step:
            return steps
        for r, _, count in step:
            done[r] += count
        steps.append(step)


def wants(case, prompts, part):
    r, first, count = part
    return first + count >= prompts[r]


# ----------------------------------------------------------------------------- the engine, kept as a server keeps it

_ENGINE = {}                                   # the engine in use; another model or another set of options replaces it


def weights_of(case):
    """``(spec, {name: tensor})`` on the GPU: the distributions of the package's random-weights writer, from the model alone.
    Llama's embedding has numbers of unit size and its output matrices shrink with the depth, as trained ones do, so that the
    largest logit stands clear of the others; Tibivik's copies of the stream mix little and its output matrices are smaller,
    without which a stack of random layers multiplies any rounding until nothing of the result is left."""
    import tesseract_b200.models  # noqa: F401  (registers the architectures)
    from tesseract_b200.config.registry import resolve_architecture
    from tesseract_b200.models.decoder import tensor_roles

    config = config_of(case)
    architecture = resolve_architecture(config)
    typed = architecture.read_config(config)
    spec = architecture.build_spec(typed)
    generator = torch.Generator(device="cuda")
    generator.manual_seed(20)
    tensors = {}
    with torch.device("cuda"):
        for cls, part, role, name, want in tensor_roles(spec):
            value = cls.random_tensor(part, role, tuple(want.shape), generator)
            if name in ("model.embed_tokens.weight", "lm_head.weight"):
                value = value * 50.0
            elif name.endswith(("o_proj.weight", "down_proj.weight")):
                value = value * (2 * config["num_hidden_layers"]) ** -0.5
            elif case["model"].startswith("tibivik"):
                if name.endswith((".o", ".down")):
                    value = value * 0.4
                elif name.endswith(("hc1.mix", "hc2.mix")):
                    value = torch.eye(value.shape[0]) + (value - 0.8 * torch.eye(value.shape[0])) / 3
            tensors[name] = value.to(torch.bfloat16)
    if "lm_head.weight" in tensors:            # an untied head near the embedding, for the same reason
        tensors["lm_head.weight"] = tensors["model.embed_tokens.weight"] + 0.25 * tensors["lm_head.weight"]
    return architecture, typed, spec, tensors


def engine_of(case):
    """The stepper and the sampler of a serving process for this model, with graphs as ``LLM`` sets them up."""
    from tesseract_b200 import kernels
    from tesseract_b200.engine.loading import make_stepper, parse_dtype, require_cuda
    from tesseract_b200.models.decoder import DecoderModel
    from tesseract_b200.parts.base import Runtime
    from tesseract_b200.sampling.sampler import Sampler

    tokens = sum(-(-(n + case["new"]) // 16) * 16 for n in lengths_of(case))
    key = (case["model"], case["dtype"], case["requests"], case["chunk"], case["budget"], tokens)
    if key not in _ENGINE:
        _ENGINE.clear()
        device = require_cuda(0)
        dtype = parse_dtype(case["dtype"])
        architecture, typed, spec, tensors = weights_of(case)
        libraries = architecture.kernel_libraries
        kernels.prepare(dtype, None if libraries is None else list(libraries(typed, case["dtype"])))
        model = DecoderModel(spec, tensors, Runtime(dtype, device))
        stepper = make_stepper(model, capacity_tokens=max(tokens, 16 * case["requests"]), page_size=16,
                               max_requests=case["requests"], max_step_tokens=case["chunk"])
        stepper.enable_graphs(case["requests"], chunk_rows=case["chunk"], max_sequence_length=131072,
                              max_batch_tokens=case["budget"])
        _ENGINE[key] = {"stepper": stepper, "sampler": Sampler(device), "warm": set()}
    return _ENGINE[key]


def inputs_of(case, seed):
    """Every request's prompt and given continuation, as lists of token ids."""
    rng = np.random.default_rng(seed)
    vocab = vocabulary(config_of(case))
    return [rng.integers(0, vocab, n + case["new"]).tolist() for n in lengths_of(case)]


def prepare(case, seed):
    engine = engine_of(case)
    prompts = lengths_of(case)
    steps = schedule(case)
    rows = sum(wants(case, prompts, part) for step in steps for part in step)
    state = {"case": case, "engine": engine, "prompts": prompts, "steps": steps, "tokens": inputs_of(case, seed),
             "logits": torch.empty((rows, vocabulary(config_of(case))), dtype=torch.float32, device="cuda")}
    warm = (case["shortest"], case["longest"], case["new"])
    if warm not in engine["warm"]:             # a serving process has met its shapes before (graphs are captured once)
        engine["warm"].add(warm)
        run(dict(state, logits=torch.empty_like(state["logits"])))
    return state


def run(state):
    from tesseract_b200.engine.step import StepEntry

    stepper, sampler = state["engine"]["stepper"], state["engine"]["sampler"]
    cache, prompts, case = stepper.cache, state["prompts"], state["case"]
    for r, n in enumerate(prompts):
        if not cache.admit(r, reserve_tokens=n + case["new"]):
            raise RuntimeError("the cache is too small for the requests")
    chosen, at, in_flight = [], 0, None
    for step in state["steps"]:
        entries, wanted = [], 0
        for part in step:
            r, first, count = part
            want = [count - 1] if wants(case, prompts, part) else []
            entries.append(StepEntry(r, state["tokens"][r][first:first + count], want))
            wanted += len(want)
        zeros = [0.0] * wanted
        if all(count == 1 and first >= prompts[r] for r, first, count in step) and stepper.can_launch_decode(wanted, [1.0] * wanted):
            launch = stepper.launch_decode(entries, zeros, zeros)
            state["logits"][at:at + wanted].copy_(launch.graph.logits[:wanted])
            if in_flight is not None:
                chosen += in_flight.tokens()
            in_flight = launch
        else:
            if in_flight is not None:
                chosen += in_flight.tokens()
                in_flight = None
            logits = stepper.step(entries)
            if wanted:
                state["logits"][at:at + wanted].copy_(logits)
                chosen += sampler.sample(logits, zeros, [1.0] * wanted, zeros)
        at += wanted
    if in_flight is not None:
        chosen += in_flight.tokens()
    for r in range(len(prompts)):
        cache.release(r)
    return {"logits": state["logits"], "tokens": np.asarray(chosen, dtype=np.int64)}


# ----------------------------------------------------------------------------- what a pass cannot do without


def work(case):
    """Per step: every matrix read once, the cached tokens of every request read once for its rows, states read and written
    once, the wanted logits written; the products of every row and the attention of every row over what it sees."""
    config, prompts = config_of(case), lengths_of(case)
    size = 4 if case["dtype"] == "float32" else 2
    vocab = vocabulary(config)
    stored = runs = 0                          # numbers in the layers' matrices; multiply-adds of a row through all runs
    paged = []                                 # per run with attention: (numbers cached a token, multiply-adds a seen token, reach)
    state, recurrent = 0, 0                    # 32-bit numbers of state a request; multiply-adds of a row against it
    if "architectures" in config:
        width, layers = config["hidden_size"], config["num_hidden_layers"]
        heads, kv, d = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"]
        stored = runs = layers * width * (2 * heads * d + 2 * kv * d + 3 * config["intermediate_size"])
        paged = [(2 * kv * d, 2 * heads * d, None)] * layers
    else:
        width, loop = config["width"], config["loop"]
        for index, layer in enumerate(config["layers"]):
            walks = loop["times"] if loop["start"] <= index < loop["stop"] else 1
            m, own = layer["mixer"], 3 * width * layer["mlp"]["ff"]
            if layer["type"] == "lightning":
                own += width * m["heads"] * (2 * m["dim"] + 3 * m["vdim"])
                state += walks * m["heads"] * m["dim"] * m["vdim"]
                recurrent += walks * 2 * m["heads"] * m["dim"] * m["vdim"]
            elif layer["type"] == "attention":
                own += width * (2 * m["heads"] * m["dim"] + 2 * m["kv_heads"] * m["dim"] + (m["kv_heads"] + 2 * m["heads"]) * m["vdim"])
                paged += [(m["kv_heads"] * (2 * m["dim"] + m["vdim"]), 2 * m["heads"] * (m["dim"] + m["vdim"]), None)] * walks
            elif layer["type"] == "latent_attention":
                entry = m["kv_rank"] + m["rot_dim"]
                own += width * (m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) + entry) + m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"])
                paged += [(entry, m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), m["mask"]["size"])] * walks
            elif layer["type"] == "mamba2":
                inner = m["heads"] * m["vdim"]
                own += width * (3 * inner + 2 * m["groups"] * m["state"] + m["heads"])
                state += walks * inner * m["state"]
                recurrent += walks * 2 * inner * m["state"]
            else:
                left, right = m["left"], m["right"]
                kv, delta = right.get("kv_heads", right["heads"]), "conv" in right
                own += width * (2 * left["heads"] + (2 if delta else 1) * left["kv_heads"]) * left["dim"]
                own += width * (2 * kv * right["dim"] + 3 * right["heads"] * right["vdim"] + 2 * right["heads"])
                paged += [(2 * left["kv_heads"] * left["dim"], 2 * left["heads"] * left["dim"], left["mask"]["size"])] * walks
                state += walks * right["heads"] * right["dim"] * right["vdim"]
                recurrent += walks * (3 if delta else 2) * right["heads"] * right["dim"] * right["vdim"]
            if "token_side" in config:
                own += 2 * width * config["token_side"]["dim"]
            stored += own
            runs += walks * own
    total_bytes = total_flops = 0
    for step in schedule(case):
        wanted = sum(wants(case, prompts, part) for part in step)
        total_bytes += size * stored + wanted * 4 * vocab + (size * vocab * width if wanted else 0) + 8 * state * len(step)
        total_flops += 2 * wanted * vocab * width
        for _, first, count in step:
            total_flops += 2 * count * (runs + recurrent)
            for numbers, per_token, reach in paged:
                reach = reach or 1 << 30
                total_bytes += size * numbers * min(first + count, reach + count)
                seen = sum(min(p + 1, reach) for p in range(first, first + count)) if count < 64 or reach < 1 << 30 else \
                    count * first + count * (count + 1) // 2
                total_flops += 2 * per_token * seen
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # Measured: the logits are 0.010 (Llama), 0.006 (Kazodra) and 0.010 (Tibivik) off the 64-bit model in bfloat16 and 1.5e-6 in
    # 32-bit; two builds that round at other places differ by up to 1.4 times that.  A token turns where the two largest
    # logits are nearer than the rounding.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 0.025 if case["model"].startswith("kazodra") else 0.03, "max": 0.3, "differ": 0.01}


# ----------------------------------------------------------------------------- the same in 64 bits, without the package


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def layer_norm(x, weight, bias, eps):
    x = x - x.mean(dim=-1, keepdim=True)
    return rms(x, eps) * weight + bias


def silu(x):
    return x * torch.sigmoid(x)


def angles(positions, frequencies):
    a = positions.double()[:, None] * torch.tensor(frequencies, dtype=torch.float64, device="cuda")[None, :]
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def rotate_halves(x, turn):
    """``x`` ``[T, heads, d]``: number ``i`` turns with number ``i + n``, ``n`` the number of frequencies."""
    cos, sin = turn
    n = cos.shape[-1]
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., 2 * n:]], dim=-1)


def rotate_pairs(x, turn):
    cos, sin = turn
    n = cos.shape[-1]
    u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
    return torch.cat([torch.stack([u * cos - v * sin, v * cos + u * sin], dim=-1).flatten(-2), x[..., 2 * n:]], dim=-1)


def stretched(frequencies, factor, low, high, original):
    """Llama 3.1's way: long wavelengths are divided, those between two limits blended."""
    out = []
    for f in frequencies:
        wavelength = 2 * math.pi / f
        s = min(1.0, max(0.0, (original / wavelength - low) / (high - low)))
        out.append((1 - s) * f / factor + s * f)
    return out


def attend(q, k, v, scale, sees, sink=None):
    """``[T, H, d]`` queries over ``[T, G, d]`` keys and ``[T, G, dv]`` values; ``sees(i, j)`` says which keys a row sees.  Blocks
    of rows, so that the scores fit."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    block = max(1, (1 << 28) // (H * T))
    for at in range(0, T, block):
        rows = q[at:at + block].reshape(-1, G, H // G, q.shape[2])
        last = at + rows.shape[0]
        scores = torch.einsum("ighd,jgd->ghij", rows, k[:last]) * scale
        i, j = torch.arange(at, last, device=q.device)[:, None], torch.arange(last, device=q.device)[None, :]
        scores = scores.masked_fill(~((j <= i) & sees(i, j)), float("-inf"))
        if sink is not None:
            column = sink.reshape(G, H // G, 1, 1).expand(-1, -1, scores.shape[2], 1)
            weights = torch.softmax(torch.cat([scores, column], dim=-1), dim=-1)[..., :-1]
        else:
            weights = torch.softmax(scores, dim=-1)
        out[at:last] = torch.einsum("ghij,jge->ighe", weights, v[:last]).reshape(-1, H, v.shape[2])
    return out


def padded(x, spans):
    """``[rows, ...]`` of several requests as ``[longest, requests, ...]``, zeros behind the shorter ones."""
    return torch.nn.utils.rnn.pad_sequence([x[a:b] for a, b in spans])


def packed(x, spans):
    return torch.cat([x[:b - a, r] for r, (a, b) in enumerate(spans)])


class Exact:
    """One model over the rows of all requests, side by side; ``spans`` are the requests' rows."""

    def __init__(self, case, seed):
        self.case, self.config = case, config_of(case)
        self.tensors = weights_of(case)[3]
        tokens = [t[:n + case["new"] - 1] for t, n in zip(inputs_of(case, seed), lengths_of(case))]
        edges = np.cumsum([0] + [len(t) for t in tokens]).tolist()
        self.spans = list(zip(edges[:-1], edges[1:]))
        self.ids = torch.tensor([t for row in tokens for t in row], device="cuda")
        self.positions = torch.cat([torch.arange(b - a, device="cuda") for a, b in self.spans])

    def weight(self, name):
        return self.tensors[name].double()

    def product(self, x, name):
        return x @ self.weight(name).T

    def per_request(self, function, *rows):
        return torch.cat([function(*(x[a:b] for x in rows)) for a, b in self.spans])

    def rows_wanted(self):
        prompts = lengths_of(self.case)
        return [self.spans[r][0] + first + count - 1 for step in schedule(self.case) for r, first, count in step
                if wants(self.case, prompts, (r, first, count))]

    def run_order(self):
        loop, count = self.config["loop"], len(self.config["layers"])
        order = [(i, None) for i in range(loop["start"])]
        for walk in range(loop["times"]):
            order += [(i, walk if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
        return order + [(i, None) for i in range(loop["stop"], count)]

    # -- Llama
    def llama(self):
        c = self.config
        H, G, d, eps, T = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"], len(self.ids)
        s = c["rope_scaling"]
        frequencies = stretched([c["rope_theta"] ** (-2.0 * i / d) for i in range(d // 2)], s["factor"], s["low_freq_factor"],
                                s["high_freq_factor"], s["original_max_position_embeddings"])
        turn = angles(self.positions, frequencies)
        x = self.tensors["model.embed_tokens.weight"][self.ids].double()
        for layer in range(c["num_hidden_layers"]):
            p = "model.layers.%d." % layer
            h = rms(x, eps) * self.weight(p + "input_layernorm.weight")
            q, k, v = (self.product(h, p + "self_attn.%s_proj.weight" % n).view(T, -1, d) for n in "qkv")
            q, k = rotate_halves(q, turn), rotate_halves(k, turn)
            a = self.per_request(lambda q, k, v: attend(q, k, v, d ** -0.5, lambda i, j: j <= i), q, k, v)
            x = x + self.product(a.reshape(T, H * d), p + "self_attn.o_proj.weight")
            h = rms(x, eps) * self.weight(p + "post_attention_layernorm.weight")
            h = silu(self.product(h, p + "mlp.gate_proj.weight")) * self.product(h, p + "mlp.up_proj.weight")
            x = x + self.product(h, p + "mlp.down_proj.weight")
        x = rms(x[self.rows_wanted()], eps) * self.weight("model.norm.weight")
        return self.product(x, "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight")

    def gated(self, h, p):
        return self.product(silu(self.product(h, p + "gate")) * self.product(h, p + "up"), p + "down")

    # -- Kazodra
    def kazodra(self):
        c, eps = self.config, self.config["norm"]["eps"]
        x = self.tensors["embed"][self.ids].double()
        side = c["token_side"]["dim"]
        for index, walk in self.run_order():
            p, layer = "l%d." % index, c["layers"][index]
            if walk is not None:
                x = x + self.weight("loop.step")[walk]

            def norm(y, name):
                return layer_norm(y, self.weight(p + name), self.weight(p + name + ".b"), eps)

            mixer = {"lightning": self.lightning, "attention": self.two_maps, "latent_attention": self.latent}[layer["type"]]
            x = x + norm(mixer(norm(x, "norm1"), layer["mixer"], p + "mix."), "norm1b")
            x = x + norm(self.gated(norm(x, "norm2"), p + "mlp."), "norm2b")
            e = self.tensors["side.embed"][self.ids][:, index * side:(index + 1) * side].double()
            g = torch.nn.functional.gelu(self.product(x, p + "side.gate"), approximate="tanh") * e
            x = x + rms(self.product(g, p + "side.proj"), eps) * self.weight(p + "side.norm")
        x = layer_norm(x[self.rows_wanted()], self.weight("final.norm"), self.weight("final.norm.b"), eps)
        return self.product(x, "embed")

    def lightning(self, h, m, p):
        T, H = h.shape[0], m["heads"]
        q, k, v = (silu(self.product(h, p + n)).view(T, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None, None]
        o = self.recurrence(q, k, v, lambda t: decay)
        o = rms(o.reshape(T, -1), self.config["norm"]["eps"]) * self.weight(p + "norm")
        return self.product(o * torch.sigmoid(self.product(h, p + "g")), p + "o")

    def recurrence(self, q, k, v, keep):
        """``S <- keep_t S + k_t v_t^T``, ``o_t = S^T q_t`` for every head of every request; ``keep(t)`` broadcasts over
        ``[requests, heads, dim, columns]``."""
        q, k, v = (padded(x, self.spans) for x in (q, k, v))
        S = torch.zeros((*k.shape[1:], v.shape[-1]), dtype=q.dtype, device=q.device)
        out = torch.empty_like(v)
        for t in range(q.shape[0]):
            S = torch.addcmul(S * keep(t), k[t].unsqueeze(-1), v[t].unsqueeze(-2))
            out[t] = torch.matmul(q[t].unsqueeze(-2), S).squeeze(-2)
        return packed(out, self.spans)

    def two_maps(self, h, m, p):
        T, H, G, d, s = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["rot"]["scaling"]
        frequencies = stretched([m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"]) for i in range(m["rot"]["dims"] // 2)],
                                s["factor"], s["low"], s["high"], s["original"])
        turn = angles(self.positions, frequencies)
        q = rotate_pairs(self.product(h, p + "q").view(T, 2 * H, d), turn).view(T, H, 2, d)
        k = rotate_pairs(self.product(h, p + "k").view(T, 2 * G, d), turn).view(T, G, 2, d)
        v = self.product(h, p + "v").view(T, G, -1)
        first, second = (self.per_request(lambda q, k, v: attend(q, k, v, m["scale"], lambda i, j: j <= i), q[:, :, n], k[:, :, n], v)
                         for n in (0, 1))
        share = torch.exp((self.weight(p + "lq1") * self.weight(p + "lk1")).sum()) \
            - torch.exp((self.weight(p + "lq2") * self.weight(p + "lk2")).sum()) + m["diff"]
        o = rms(first - share * second, self.config["norm"]["eps"]) * (1.0 - m["diff"])
        return self.product(o.reshape(T, -1) * torch.sigmoid(self.product(h, p + "g")), p + "o")

    def latent(self, h, m, p):
        T, H, d = h.shape[0], m["heads"], m["dim"]
        turn = angles(self.positions, [m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"]) for i in range(m["rot"]["dims"] // 2)])
        q = self.product(h, p + "q").view(T, H, -1)
        down = self.product(h, p + "dkv")
        vector = rms(down[:, :m["kv_rank"]], self.config["norm"]["eps"]) * self.weight(p + "dkv.norm")
        shared = rotate_pairs(down[:, None, m["kv_rank"]:], turn).expand(T, H, -1)
        k = torch.cat([self.product(vector, p + "uk").view(T, H, d), shared], dim=-1)
        q = torch.cat([q[..., :d], rotate_pairs(q[..., d:], turn)], dim=-1)
        v = self.product(vector, p + "uv").view(T, H, -1)
        o = self.per_request(lambda q, k, v: attend(q, k, v, m["scale"], lambda i, j: i - j < m["mask"]["size"]), q, k, v)
        return self.product(o.reshape(T, -1), p + "o")

    # -- Tibivik
    def tibivik(self):
        c, eps, b = self.config, self.config["norm"]["eps"], self.config["embedding"]["bigram"]
        before = torch.cat([self.ids[:1], self.ids[:-1]])
        pairs = torch.where(self.positions == 0, b["buckets"], (before * b["mul_prev"] + self.ids * b["mul_cur"]) % b["buckets"])
        x = (self.tensors["embed"][self.ids].double() + self.tensors["bigram"][pairs].double()).expand(c["streams"], -1, -1)
        for index, _ in self.run_order():
            p, layer = "l%d." % index, c["layers"][index]
            for number, sublayer in ((1, lambda h: self.tibivik_mixer(h, layer, p + "mix.")), (2, lambda h: self.gated(h, p + "mlp."))):
                hc = p + "hc%d." % number
                u = torch.einsum("s,stw->tw", self.weight(hc + "in"), x)
                y = sublayer(rms(u, eps) * self.weight(p + "norm%d" % number))
                x = torch.einsum("sr,stw->rtw", self.weight(hc + "mix"), x) + self.weight(hc + "out")[:, None, None] * y
        x = rms(x.sum(dim=0)[self.rows_wanted()], eps) * self.weight("final.norm")
        return self.product(x, "embed")

    def tibivik_mixer(self, h, layer, p):
        m = layer["mixer"]
        if layer["type"] == "mamba2":
            return self.state_space(h, m, p)
        left, right = (self.shared_keys, self.memory) if layer["type"] == "parallel" else (self.chunks, self.delta)
        return m["left_scale"] * left(h, m["left"], p + "left.") + m["right_scale"] * right(h, m["right"], p + "right.")

    def shared_keys(self, h, m, p):
        T, G, eps = h.shape[0], m["kv_heads"], self.config["norm"]["eps"]
        turn = angles(self.positions, [m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"]) for i in range(m["rot"]["dims"] // 2)])
        raw = self.product(h, p + "k")
        q = rotate_halves((rms(self.product(h, p + "q"), eps) * self.weight(p + "q.norm")).view(T, -1, m["dim"]), turn)
        k = rotate_halves((rms(raw, eps) * self.weight(p + "k.norm")).view(T, G, -1), turn)
        sink = self.weight(p + "sink")
        o = self.per_request(lambda q, k, v: attend(q, k, v, m["scale"], lambda i, j: i - j < m["mask"]["size"], sink), q, k, raw.view(T, G, -1))
        return self.product(o.reshape(T, -1), p + "o")

    def chunks(self, h, m, p):
        T, size = h.shape[0], m["mask"]["size"]
        q, k, v = ((self.product(h, p + n) + self.weight(p + n + ".b")).view(T, -1, m["dim"]) for n in "qkv")
        sink = self.weight(p + "sink")
        o = self.per_request(lambda q, k, v: attend(q, k, v, m["scale"], lambda i, j: i // size == j // size, sink), q, k, v)
        return self.product((o * torch.sigmoid(self.product(h, p + "g")).unsqueeze(-1)).reshape(T, -1), p + "o")

    def convolved(self, x, taps, bias=0.0):
        def one(rows):
            wide = torch.nn.functional.pad(rows, (0, 0, taps.shape[1] - 1, 0))
            return sum(wide[j:j + rows.shape[0]] * taps[:, j] for j in range(taps.shape[1]))

        return silu(self.per_request(one, x) + bias)

    def state_space(self, h, m, p):
        T, H, N, G = h.shape[0], m["heads"], m["state"], m["groups"]
        inner = H * m["vdim"]
        rows = self.product(h, p + "in")
        mixed = self.convolved(rows[:, inner:2 * inner + 2 * G * N], self.weight(p + "conv"), self.weight(p + "conv.b"))
        x = mixed[:, :inner].view(T, H, -1)
        B, C = (part.reshape(T, G, N).repeat_interleave(H // G, dim=1) for part in mixed[:, inner:].split(G * N, dim=1))
        step = torch.nn.functional.softplus(rows[:, 2 * inner + 2 * G * N:] + self.weight(p + "dt_bias"), threshold=1e3)
        keep = padded(torch.exp(-torch.exp(self.weight(p + "A_log")) * step), self.spans)[..., None, None]
        y = self.recurrence(C, B * step.unsqueeze(-1), x, lambda t: keep[t]) + self.weight(p + "D")[:, None] * x
        gated = (y.reshape(T, inner) * silu(rows[:, :inner])).view(T, m["norm_groups"], -1)
        return self.product(rms(gated, self.config["norm"]["eps"]).reshape(T, inner) * self.weight(p + "norm"), p + "o")

    def memory(self, h, m, p):
        T, H, cap = h.shape[0], m["heads"], m["gate_cap"]
        q, k, v = (self.product(h, p + n).view(T, H, -1) for n in "qkv")
        i, f = (cap * torch.tanh((self.product(h, p + n) + self.weight(p + n + ".b")) / cap) for n in "if")
        i, f = padded(i, self.spans), torch.nn.functional.logsigmoid(padded(f, self.spans))
        top, keep, write, peaks = torch.zeros_like(i[0]), [], [], []
        for t in range(i.shape[0]):
            new = torch.maximum(f[t] + top, i[t])
            keep.append(torch.exp(f[t] + top - new))
            write.append(torch.exp(i[t] - new))
            top = new
            peaks.append(top)
        k = k * packed(torch.stack(write), self.spans).unsqueeze(-1)
        ones = torch.ones_like(v[..., :1])
        o = self.recurrence(q * m["dim"] ** -0.5, k, torch.cat([v, ones], dim=-1), lambda t: keep[t][..., None, None])
        weight = torch.maximum(o[..., -1:].abs(), torch.exp(-packed(torch.stack(peaks), self.spans)).unsqueeze(-1)) + 1e-6
        o = rms(o[..., :-1] / weight, self.config["norm"]["eps"]).reshape(T, -1) * self.weight(p + "norm")
        return self.product(o * torch.sigmoid(self.product(h, p + "g")), p + "o")

    def delta(self, h, m, p):
        T, H, G = h.shape[0], m["heads"], m["kv_heads"]
        q, k, v = (self.convolved(self.product(h, p + n), self.weight(p + n + ".conv")) for n in "qkv")

        def unit(x):
            x = x.view(T, G, -1)
            return (x / torch.sqrt((x * x).sum(dim=-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)

        q, k, v = (padded(x, self.spans) for x in (unit(q) * m["dim"] ** -0.5, unit(k), v.view(T, H, -1)))
        beta = padded(torch.sigmoid(self.product(h, p + "b")), self.spans)
        step = torch.nn.functional.softplus(self.product(h, p + "a") + self.weight(p + "dt_bias"), threshold=1e3)
        keep = padded(torch.exp(-torch.exp(self.weight(p + "A_log")) * step), self.spans)
        S = torch.zeros((*k.shape[1:], v.shape[-1]), dtype=q.dtype, device=q.device)
        out = torch.empty_like(v)
        for t in range(q.shape[0]):
            S = S * keep[t][..., None, None]
            u = beta[t].unsqueeze(-1) * (v[t] - torch.matmul(k[t].unsqueeze(-2), S).squeeze(-2))
            S = torch.addcmul(S, k[t].unsqueeze(-1), u.unsqueeze(-2))
            out[t] = torch.matmul(q[t].unsqueeze(-2), S).squeeze(-2)
        o = (rms(packed(out, self.spans), self.config["norm"]["eps"]) * self.weight(p + "norm")).reshape(T, -1)
        return self.product(o * silu(self.product(h, p + "g")), p + "o")


def exact(case, seed):
    model = Exact(case, seed)
    with torch.no_grad():
        logits = getattr(model, case["model"].split("-")[0])()
    return {"logits": logits, "tokens": None}
