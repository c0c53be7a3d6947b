"""What a user of the engine has it do, as cases that can be timed and compared.

A case is one step of the dense Qwen3 decoder through :class:`StepRunner`, the call that ``Engine``, the replay program
and ``bench.py`` make for every batch: a flat batch of prompt portions and single (decoded) tokens goes through all
layers against the paged cache, and the float32 logits of every request's last token come back.

``size``      layer sizes: ``8b`` and ``0.6b`` as in ``bench.py``, ``tiny`` as the tests' smallest untied model
``dtype``     ``bfloat16`` or the true ``float32`` path
``decodes``   requests that bring one token each, behind ``context`` cached tokens
``prompts``   requests that bring a portion of ``portion`` tokens each, behind ``prefix`` cached tokens
``ragged``    requests differ in length: contexts in eight levels, portions and prefixes in four
``page``      cache positions per page

Outputs: ``logits`` [requests, vocab] and the cache pages (single tokens: the rows) that the step wrote, as views of
the cache.  A pass leaves the state as it found it but for those rows: it starts by setting the requests' progress
back, so every pass does the same work.
"""
import hashlib
import math

import torch

SIZES = {
    "8b": dict(vocab_size=151936, hidden_size=4096, intermediate_size=12288, num_hidden_layers=36,
               num_attention_heads=32, num_key_value_heads=8, head_dim=128, max_position_embeddings=40960,
               rms_norm_eps=1e-6, rope_theta=1000000.0, tie_word_embeddings=False),
    "0.6b": dict(vocab_size=151936, hidden_size=1024, intermediate_size=3072, num_hidden_layers=28,
                 num_attention_heads=16, num_key_value_heads=8, head_dim=128, max_position_embeddings=40960,
                 rms_norm_eps=1e-6, rope_theta=1000000.0, tie_word_embeddings=True),
    "tiny": dict(vocab_size=1000, hidden_size=96, intermediate_size=200, num_hidden_layers=3,
                 num_attention_heads=6, num_key_value_heads=2, head_dim=32, max_position_embeddings=512,
                 rms_norm_eps=1e-5, rope_theta=1000000.0, tie_word_embeddings=False),
}
LEVELS = 8


def _std(name, sizes):
    """Standard deviation of a random matrix, such that the residual stream is an embedding plus many small branches, as in
    a trained model: what leads back into the stream is scaled down by the square root of their number.  (With
    equal matrices everywhere the stream is the last branches' alone and doubles a rounding error every few layers.)"""
    if name.startswith("model.embed_tokens"):
        return sizes["hidden_size"] / 1024
    return 0.02 / math.sqrt(2 * sizes["num_hidden_layers"]) if "o_proj" in name or "down_proj" in name else 0.02


def _case(name, size, dtype, *, prompts=0, portion=0, prefix=0, decodes=0, context=0, ragged=False, page=16):
    case = dict(size=size, dtype=dtype, prompts=prompts, portion=portion, prefix=prefix, decodes=decodes,
                context=context, ragged=ragged, page=page)
    return dict(name=name, **case) if name else case


def listed():
    return [
        # the smallest model of the tests, five requests: nothing but launches and the host's work on a step
        _case("tiny_f32_decode_5", "tiny", "float32", decodes=5, context=100, page=8),
        # one user in front of a small model, a long chat: the latency of a token
        _case("0.6b_decode_1", "0.6b", "bfloat16", decodes=1, context=4096),
        # a small model serving 64 requests of every length
        _case("0.6b_decode_64", "0.6b", "bfloat16", decodes=64, context=2000, ragged=True),
        # the same while new requests arrive: prompt portions of all lengths beside the decoded tokens
        _case("0.6b_mixed", "0.6b", "bfloat16", prompts=4, portion=1021, decodes=60, context=2000, ragged=True),
        # the true 32-bit path, for those who check numerics or compare with another engine: decode and a prompt
        _case("0.6b_f32_decode_8", "0.6b", "float32", decodes=8, context=2000, ragged=True),
        _case("0.6b_f32_prompt_512", "0.6b", "float32", prompts=1, portion=512),
        # the benchmark's decode points: one user, a small batch at a long context, a large one at a short context
        _case("8b_decode_1", "8b", "bfloat16", decodes=1, context=8192),
        _case("8b_decode_8", "8b", "bfloat16", decodes=8, context=8192),
        _case("8b_decode_64", "8b", "bfloat16", decodes=64, context=1024),
        # the benchmark's prompt; a short question (time to first token); and chunked prefill: the last portion of a
        # long prompt beside the decoded tokens of requests that are already running
        _case("8b_prompt_2048", "8b", "bfloat16", prompts=1, portion=2048),
        _case("8b_prompt_37", "8b", "bfloat16", prompts=1, portion=37),
        _case("8b_chunk_beside_decode", "8b", "bfloat16", prompts=1, portion=509, prefix=1536, decodes=12, context=3000,
              ragged=True),
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    size = rng.choices(("8b", "0.6b", "tiny"), (8, 9, 3))[0]
    dtype = "bfloat16" if size == "8b" else rng.choice(("bfloat16", "float32"))
    kind = rng.choices(("decode", "prompt", "mixed"), (10, 5, 5))[0]
    longest = {"8b": 8192, "0.6b": 4096, "tiny": 300}[size]
    cached = {"8b": 8 * 8192, "0.6b": 64 * 2000, "tiny": 64 * 300}[size]        # cached tokens over all requests
    tokens = {"8b": 2048, "0.6b": 4096 if dtype == "bfloat16" else 512, "tiny": 200}[size]
    case = dict(prompts=0, portion=0, prefix=0, decodes=0, context=0)
    if kind != "prompt":
        case["decodes"] = _log_uniform(rng, 1, 64)
        case["context"] = _log_uniform(rng, 16, min(longest, cached // case["decodes"]))
        if kind == "mixed" and dtype == "float32":
            case["context"] = min(case["context"], 2000)
    if kind != "decode":
        case["prompts"] = 1 if kind == "prompt" or rng.random() < 0.5 else rng.randint(2, 4)
        most = (tokens if kind == "prompt" else tokens // 2) // case["prompts"]
        case["portion"] = _log_uniform(rng, 2, most)
        if rng.random() < 0.5:
            case["prefix"] = _log_uniform(rng, 1, longest // 4)
    return _case(None, size, dtype, ragged=rng.random() < 0.6, page=rng.choice((8, 16, 16, 32)), **case)


def _segments(case):
    """(cached tokens, new tokens) of every request: the single tokens first."""
    def level(value, i, count):
        return value - (i % count) * (value // (count + 1)) if case["ragged"] else value
    found = [(level(case["context"], i, LEVELS), 1) for i in range(case["decodes"])]
    return found + [(level(case["prefix"], i, 4), level(case["portion"], i, 4)) for i in range(case["prompts"])]


def _shape(case):
    """(layers, requests, pages a request, 2, kv heads, page size, head size): the cache, request after request."""
    sizes, segments = SIZES[case["size"]], _segments(case)
    pages = max(-(-(cached + new) // case["page"]) for cached, new in segments)
    return (sizes["num_hidden_layers"], len(segments), pages, 2, sizes["num_key_value_heads"], case["page"],
            sizes["head_dim"])


def _tokens(case, seed):
    generator = torch.Generator().manual_seed(seed)
    return [torch.randint(0, SIZES[case["size"]]["vocab_size"], (new,), generator=generator).tolist()
            for _, new in _segments(case)]


def _fill(storage, seed):
    """What earlier steps left in the cache."""
    storage.normal_(0.0, 0.5, generator=torch.Generator(storage.device).manual_seed(seed))


def _written(case, cache):
    """The rows of the cache that a step writes: of the single tokens the row alone, level by level, of a prompt
    portion its pages.  ``cache``: [layers, requests, pages, 2, kv heads, page size, head size]; the results are views."""
    page, segments, decodes = case["page"], _segments(case), case["decodes"]
    found = []
    for j in range(min(decodes, LEVELS if case["ragged"] else 1)):
        at = segments[j][0]
        step = LEVELS if case["ragged"] else 1
        found.append(cache[:, j:decodes:step, at // page, :, :, at % page])
    for i in range(decodes, len(segments)):
        cached, new = segments[i]
        found.append(cache[:, i, cached // page:(cached + new - 1) // page + 1])
    return found


def prepare(case, seed):
    import qwen_inference_lab_b200.models  # noqa: F401  (registers the architectures)
    from qwen_inference_lab_b200.cache import CacheManager
    from qwen_inference_lab_b200.config import registry
    from qwen_inference_lab_b200.engine import StepEntry, StepRunner
    from qwen_inference_lab_b200.weights import init_random

    dtype = getattr(torch, case["dtype"])
    data = dict(SIZES[case["size"]], architectures=["Qwen3ForCausalLM"], model_type="qwen3", attention_bias=False,
                eos_token_id=None)
    entry = registry.lookup(data)
    model = entry.build(entry.config_class.from_dict(data))
    for name, param in model.all_named_params().items():
        if param.init == "normal" and not name.startswith("lm_head"):     # a tied head is the embedding
            param.std = _std(name, data)
    init_random(model, seed, device="cuda", dtype=dtype)
    segments, shape = _segments(case), _shape(case)
    requests, pages = shape[1], shape[2]
    cache = CacheManager(model.cache_specs(), num_pages=requests * pages, page_size=case["page"],
                         max_requests=requests, max_context=pages * case["page"], dtype=dtype, device=model.device)
    _fill(cache.kv_groups[0].storage, seed)
    for request in range(requests):          # every request holds its pages from the start, one after another
        cache.admit(request)
        cache.ensure(request, pages * case["page"])
        cache.advance(request, segments[request][0])
    runner = StepRunner(model, cache, max_step_tokens=max(64, sum(new for _, new in segments)))
    entries = [StepEntry(request, tokens, [len(tokens) - 1]) for request, tokens in enumerate(_tokens(case, seed))]
    return dict(runner=runner, cache=cache, entries=entries, cached=[c for c, _ in segments],
                written=_written(case, cache.kv_groups[0].storage.view(shape)))


def run(state):
    progress = state["cache"].progress
    for request, cached in enumerate(state["cached"]):
        progress[request] = cached
    return {"logits": state["runner"].run(state["entries"]), "cache": state["written"]}


def work(case):
    sizes, segments = SIZES[case["size"]], _segments(case)
    h, d, layers = sizes["hidden_size"], sizes["head_dim"], sizes["num_hidden_layers"]
    q_heads, kv_heads = sizes["num_attention_heads"], sizes["num_key_value_heads"]
    layer = layers * ((2 * q_heads + 2 * kv_heads) * d * h + 3 * sizes["intermediate_size"] * h)
    head, norms = sizes["vocab_size"] * h, layers * (2 * h + 2 * d) + h
    tokens = sum(new for _, new in segments)
    pairs = sum(new * cached + new * (new + 1) // 2 for cached, new in segments)
    cached_tokens = sum(cached for cached, _ in segments)
    itemsize = 2 if case["dtype"] == "bfloat16" else 4
    values = layer + head + norms + tokens * h + (cached_tokens + tokens) * layers * 2 * kv_heads * d
    return {"bytes": itemsize * values + 4 * len(segments) * sizes["vocab_size"],
            "flops": 2.0 * tokens * layer + 2.0 * len(segments) * head + 4.0 * layers * q_heads * d * pairs}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 5e-6}      # two orders of summation differ by about 1e-6 after all layers
    return {"rel": 0.03, "max": 0.3}        # other kernels for the same step: 0.002 to 0.01, single values 0.06


# ------------------------------------------------------------------ the same in 64 bits
def _drawn(seed, name, shape, std, mean, dtype, device):
    """The random weights of (seed, tensor name): the sum of twelve 16-bit uniforms from splitmix64, centred and scaled
    in float32 and rounded to the model's dtype."""
    start = int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:8], "little") & 0x7FFFFFFFFFFFFFFF
    signed = lambda v: v - (1 << 64) if v >= 1 << 63 else v
    golden, mix1, mix2 = (signed(v) for v in (0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB))
    count = math.prod(shape)
    out = torch.empty(count, dtype=torch.float64, device=device)
    shifted = lambda z, n: (z >> n) & ((1 << (64 - n)) - 1)
    for first in range(0, count, 1 << 22):
        index = torch.arange(first, min(count, first + (1 << 22)), dtype=torch.int64, device=device)
        total = torch.zeros_like(index)
        for turn in range(3):
            z = (index * 3 + (turn + 1)) * golden + start
            z = (z ^ shifted(z, 30)) * mix1
            z = (z ^ shifted(z, 27)) * mix2
            z = z ^ shifted(z, 31)
            for n in (0, 16, 32, 48):
                total += (z >> n) & 0xFFFF
        values = (total - 393210).float() * (1.0 / 65536.0)
        values = values * torch.tensor(std, dtype=torch.float32) + torch.tensor(mean, dtype=torch.float32)
        out[first:first + len(index)] = values.to(dtype).double()
    return out.view(shape)


def exact(case, seed):
    sizes, segments, shape = SIZES[case["size"]], _segments(case), _shape(case)
    dtype, device = getattr(torch, case["dtype"]), torch.device("cuda")
    h, d, inner, eps = sizes["hidden_size"], sizes["head_dim"], sizes["intermediate_size"], sizes["rms_norm_eps"]
    q_heads, kv_heads, page = sizes["num_attention_heads"], sizes["num_key_value_heads"], case["page"]
    group = q_heads // kv_heads

    def matrix(name, rows, cols):
        return _drawn(seed, name + ".weight", (rows, cols), _std(name, sizes), 0.0, dtype, device)

    def gain(name, width):
        return _drawn(seed, name + ".weight", (width,), 0.05, 1.0, dtype, device)

    def normed(x, weight):
        return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt() * weight

    # the rotation's table is part of the model: angles in float32, cosines and sines rounded to its dtype
    longest = max(cached + new for cached, new in segments)
    inverse = 1.0 / (sizes["rope_theta"] ** (torch.arange(0, d, 2, dtype=torch.float32) / d))
    angles = torch.arange(longest).float()[:, None] * inverse[None, :]
    cosines, sines = (t.to(dtype).double().to(device) for t in (angles.cos(), angles.sin()))
    positions = torch.cat([torch.arange(cached, cached + new) for cached, new in segments]).to(device)
    cosine, sine = cosines[positions][:, None], sines[positions][:, None]

    def rotated(x):
        left, right = x[..., :d // 2], x[..., d // 2:]
        return torch.cat((left * cosine - right * sine, left * sine + right * cosine), -1)

    # rows of earlier steps as they are, and of this step in 64 bits
    storage = torch.empty((shape[0], shape[1] * shape[2], *shape[3:]), dtype=dtype, device=device)
    _fill(storage, seed)
    pages = storage.view(shape)
    kept = [[None] * len(w) for w in ([0] * shape[0] for _ in segments)]
    embedding = matrix("model.embed_tokens", sizes["vocab_size"], h)
    tokens = torch.tensor([t for row in _tokens(case, seed) for t in row], device=device)
    x = embedding[tokens]
    for layer in range(sizes["num_hidden_layers"]):
        prefix = f"model.layers.{layer}."
        n = normed(x, gain(prefix + "input_layernorm", h))
        q, k, v = (n @ matrix(prefix + f"self_attn.{name}_proj", heads * d, h).t()
                   for name, heads in (("q", q_heads), ("k", kv_heads), ("v", kv_heads)))
        q = rotated(normed(q.view(-1, q_heads, d), gain(prefix + "self_attn.q_norm", d)))
        k = rotated(normed(k.view(-1, kv_heads, d), gain(prefix + "self_attn.k_norm", d)))
        v = v.view(-1, kv_heads, d)
        attended, first = [], 0
        for i, (cached, new) in enumerate(segments):
            rows = slice(first, first + new)
            first += new
            kept[i][layer] = (k[rows], v[rows])
            held = pages[layer, i, :-(-cached // page)].permute(1, 2, 0, 3, 4).reshape(2, kv_heads, -1, d)[:, :, :cached]
            keys = torch.cat((held[0].double(), k[rows].transpose(0, 1)), 1)          # [kv heads, keys, d]
            values = torch.cat((held[1].double(), v[rows].transpose(0, 1)), 1)
            mask = torch.arange(cached + new, device=device)[None, :] > torch.arange(cached, cached + new, device=device)[:, None]
            out = torch.empty((kv_heads, group, new, d), dtype=torch.float64, device=device)
            queries = q[rows].view(new, kv_heads, group, d).permute(1, 2, 0, 3)
            for j in range(group):
                scores = (queries[:, j] @ keys.transpose(1, 2)) * d ** -0.5
                out[:, j] = scores.masked_fill(mask, -math.inf).softmax(-1) @ values
            attended.append(out.permute(2, 0, 1, 3).reshape(new, q_heads * d))
        x = x + torch.cat(attended) @ matrix(prefix + "self_attn.o_proj", h, q_heads * d).t()
        n = normed(x, gain(prefix + "post_attention_layernorm", h))
        hidden = torch.nn.functional.silu(n @ matrix(prefix + "mlp.gate_proj", inner, h).t())
        hidden = hidden * (n @ matrix(prefix + "mlp.up_proj", inner, h).t())
        x = x + hidden @ matrix(prefix + "mlp.down_proj", h, inner).t()
    last = torch.tensor([new for _, new in segments]).cumsum(0).to(device) - 1
    n = normed(x[last], gain("model.norm", h))
    head = embedding if sizes["tie_word_embeddings"] else matrix("lm_head", sizes["vocab_size"], h)
    logits = n @ head.t()
    written, decodes = [], case["decodes"]
    for j, view in enumerate(_written(case, pages)):
        result = view.double()
        if j < min(decodes, LEVELS if case["ragged"] else 1):
            step = LEVELS if case["ragged"] else 1
            for at, i in enumerate(range(j, decodes, step)):
                for layer in range(shape[0]):
                    result[layer, at, 0], result[layer, at, 1] = (rows[0] for rows in kept[i][layer])
        else:
            i = decodes + j - min(decodes, LEVELS if case["ragged"] else 1)
            cached, new = segments[i]
            slots = torch.arange(cached, cached + new, device=device) - cached // page * page
            for layer in range(shape[0]):
                for plane in (0, 1):
                    result[layer, slots // page, plane, :, slots % page] = kept[i][layer][plane]
        written.append(result)
    return {"logits": logits, "cache": written}
