"""Performance cases of the tree speculative decoding framework, through its public entry points.

What a program that uses the package does, from the smallest call to a whole request:

``matmul``    the 4-bit operator on its own: weights as quantised (``matmul``) or re-laid-out (``matmul_tiled``)
``rope``      ``rope_positions`` on one layer's queries
``forward``   ``Model.__call__``: a prompt, a chunk of one, or the next token, on an empty or a filled cache
``verify``    ``tree_decoding``: one target pass over a token tree, on a filled cache
``generate``  ``SpecDecoder.generate``: a whole request, prompt ingestion and speculative steps
``batch``     ``BatchSpecDecoder.generate``: several requests that share every pass

Model shapes are the presets of the benchmark configurations.  Weights are random: linear layers as
``Model.random_init`` draws them, norm weights so small that the residual stream keeps the token it started from, and for
whole requests the output projection tied to the embedding through a successor table, so that the next token of a context
has a clear lead over the rest, as it mostly has in a trained model; draft and target share most of that table.  Greedy
output then is a property of the weights and not of how the last bit of a sum was rounded.  (Sampled generation is not
among the cases: a draw that falls on a boundary of the distribution may go either way.)
"""
import dataclasses
import math

import numpy as np
import torch

import b200_eagle as be

GROUP = 64
DEVICE = "cuda"
# target and draft of a request, by the benchmark's shapes
PAIRS = {
    "7b+0.5b": ("qwen2-7b", "qwen2-0.5b"),
    "8b+1b": ("llama3-8b", "llama3.2-1b"),
    "0.5b+0.5b": ("qwen2-0.5b", "qwen2-0.5b"),
}
MODELS = ("qwen2-0.5b", "llama3.2-1b", "qwen2-7b", "llama3-8b")
AGREEMENT = 0.75             # share of tokens after which draft and target expect the same one


# --------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one row through a small projection: the single-token call of a draft-sized layer, all latency
        dict(name="matmul 1 row", kind="matmul", layout="mlx", rows=1, n=896, k=896, bias=True),
        # the operator benchmark's matrix at the rows of a small tree
        dict(name="matmul 8 rows", kind="matmul", layout="mlx", rows=8, n=8192, k=2048, bias=False),
        # the widest layer of the 7B shape at a full tree, weights in the streaming layout
        dict(name="matmul 31 rows tiled", kind="matmul", layout="tiled", rows=31, n=18944, k=3584, bias=False),
        # a prompt chunk through the operator, a row count that fills no tile
        dict(name="matmul 203 rows", kind="matmul", layout="mlx", rows=203, n=4096, k=14336, bias=False),
        # the queries of a tree at one layer
        dict(name="rope 31 tokens", kind="rope", batch=1, heads=32, tokens=31, dim=128),
        # plain decoding with the small model: one token on a cache of a few hundred
        dict(name="next token 0.5b", kind="forward", model="qwen2-0.5b", tokens=1, cached=411, last=True),
        # a short prompt of a request, all its logits wanted (scoring)
        dict(name="prompt of 61 0.5b", kind="forward", model="qwen2-0.5b", tokens=61, cached=0, last=False),
        # a long prompt into the large model: time to the first token
        dict(name="prompt of 1024 8b", kind="forward", model="llama3-8b", tokens=1024, cached=0, last=True),
        # verification of a 15-node tree, the middle of a request
        dict(name="verify 16 7b", kind="verify", model="qwen2-7b", nodes=16, cached=300),
        # verification of the largest tree late in a long conversation
        dict(name="verify 32 8b long", kind="verify", model="llama3-8b", nodes=32, cached=3500),
        # a whole request of the benchmark's headline configuration
        dict(name="request 7b", kind="generate", pair="7b+0.5b", prompt=256, tokens=64, depth=3, verify=15),
        # two requests that share a GPU
        dict(name="two requests 8b", kind="batch", pair="8b+1b", requests=2, prompt=517, tokens=48, depth=3, verify=15),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "rope", "forward", "forward", "forward", "verify", "verify",
                       "generate", "generate", "batch"])
    if kind == "matmul":
        layout = rng.choice(["mlx", "tiled"])
        return dict(kind=kind, layout=layout, rows=_log(rng, 1, 256 if layout == "mlx" else 32), n=8 * _log(rng, 16, 2400),
                    k=128 * _log(rng, 2, 148), bias=rng.random() < 0.5)
    if kind == "rope":
        return dict(kind=kind, batch=rng.randint(1, 4), heads=rng.randint(2, 64), tokens=_log(rng, 1, 512),
                    dim=rng.choice([64, 128]))
    if kind == "forward":
        tokens = rng.choice([1, _log(rng, 2, 32), _log(rng, 33, 1024), _log(rng, 33, 1024)])
        return dict(kind=kind, model=rng.choice(MODELS), tokens=tokens, cached=rng.choice([0, _log(rng, 16, 3000)]),
                    last=tokens > 256 or rng.random() < 0.5)
    if kind == "verify":
        return dict(kind=kind, model=rng.choice(MODELS), nodes=rng.randint(2, 32), cached=_log(rng, 16, 4000))
    pair = rng.choice(sorted(PAIRS))
    if kind == "generate":
        depth = rng.randint(1, 6)
        return dict(kind=kind, pair=pair, prompt=_log(rng, 8, 700), tokens=_log(rng, 8, 48), depth=depth,
                    verify=rng.randint(4, 31))
    requests = rng.randint(2, 4)
    return dict(kind=kind, pair=pair, requests=requests, prompt=_log(rng, 8, 300), tokens=_log(rng, 8, 32),
                depth=rng.randint(1, 5), verify=rng.randint(4, 32 // requests - 1))


# --------------------------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _successors(vocab, seed, other=None):
    """For every token the one that follows it: a random permutation, or ``other`` with the entries of a quarter of
    the tokens dealt out anew among them."""
    g = _generator(seed)
    if other is None:
        return torch.randperm(vocab, generator=g, device=DEVICE)
    again = (torch.rand(vocab, generator=g, device=DEVICE) >= AGREEMENT).nonzero().reshape(-1)
    table = other.clone()
    table[again] = other[again.roll(1)]
    return table


def _model(preset, seed, successors=None):
    """A model of a preset's shape, ready for use.  With ``successors`` its output row of a token's successor is the
    token's embedding."""
    args = be.shape_preset(preset)
    if successors is not None:
        args = dataclasses.replace(args, tie_word_embeddings=False)
    model = be.Model.random_init(args, int(seed), DEVICE)
    gain = 30.0 / args.hidden_size
    for layer in model.layers:
        layer["input_norm"].mul_(gain)
        layer["post_norm"].mul_(gain)
        if layer["qkv"].bias is not None:
            layer["qkv"].bias.mul_(gain)
    if successors is not None:
        head, embed, known = model.lm_head, model.embed, successors.numel()
        head.weight[successors] = embed.weight[:known]
        head.scales[successors] = embed.scales[:known]
        head.biases[successors] = embed.biases[:known]
        model.norm.mul_(2.0)                              # a trained model's confidence in the likely token
    return model.relayout()


def _tokens(count, vocab, seed):
    return torch.randint(0, vocab, (count,), generator=torch.Generator().manual_seed(int(seed)), dtype=torch.int32)


def _filled_cache(model, cached, room, seed):
    """A cache with the keys and values of ``cached`` earlier tokens and space for ``room`` more."""
    cache = model.make_cache(64 * ((cached + room + 63) // 64))
    if cached:
        rows = cache.data[:, :, :, :cached]
        rows.copy_(0.15 * torch.randn(rows.shape, generator=_generator(seed), device=DEVICE))
    cache.offset = cached
    return cache


def _tree(nodes, rng):
    """A token tree: parents before children, the likelier nodes with more of them.  Depths and the ancestor mask."""
    depth, mask = [0], np.eye(nodes, dtype=bool)
    mask[:, 0] = True
    for i in range(1, nodes):
        parent = int(rng.integers(0, i) * rng.random())
        while depth[parent] >= 6:
            parent = int(rng.integers(0, parent))
        depth.append(depth[parent] + 1)
        mask[i] |= mask[parent]
    return np.array(depth, dtype=np.int32), mask


_widest = []


def _load_widest_first():
    """A program that holds several models in turn: prompt chunks are replayed from captured graphs, which keep the
    address of the operator's scratch, and the scratch grows with the widest layer met.  So the widest comes first (a
    one-layer model of that width, kept), and no later model makes it move."""
    if not _widest:
        width = max(be.shape_preset(m).intermediate_size for m in MODELS)
        args = be.ModelArgs(model_type="llama", hidden_size=128, num_hidden_layers=1, intermediate_size=width,
                            num_attention_heads=2, num_key_value_heads=1, rms_norm_eps=1e-5, vocab_size=1024)
        model = be.Model.random_init(args, 0, DEVICE).relayout()
        cache = model.make_cache(256)
        model(_tokens(128, args.vocab_size, 0)[None].to(DEVICE), cache, logits_last_only=True)
        _widest.append((model, cache))


def prepare(case, seed):
    if case["kind"] not in ("matmul", "rope"):
        _load_widest_first()
    return dict(run=_RUN[case["kind"]], **_PREPARE[case["kind"]](case, seed))


def _prepare_matmul(c, seed):
    g = _generator(seed)
    w = be.quantize.quantize(torch.randn(c["n"], c["k"], generator=g, device=DEVICE) * 0.02)
    x = torch.randn(c["rows"], c["k"], generator=g, device=DEVICE).half()
    bias = (torch.randn(c["n"], generator=g, device=DEVICE) * 0.02).half() if c["bias"] else None
    if c["layout"] == "tiled":
        return dict(x=x, w=be.qmm_kernel.relayout(*w), n=c["n"], bias=bias)
    return dict(x=x, w=w, n=None, bias=bias)


def _prepare_rope(c, seed):
    g = _generator(seed)
    x = torch.randn(c["batch"], c["heads"], c["tokens"], c["dim"], generator=g, device=DEVICE).half()
    positions = torch.randint(0, 8192, (c["batch"], c["tokens"]), generator=g, device=DEVICE, dtype=torch.int32)
    frequencies = 5e5 ** (-torch.arange(0, c["dim"], 2, dtype=torch.float32, device=DEVICE) / c["dim"])
    return dict(x=x, positions=positions, frequencies=frequencies)


def _prepare_forward(c, seed):
    model = _model(c["model"], seed)
    cache = _filled_cache(model, c["cached"], c["tokens"] + 64, seed + 1)
    tokens = _tokens(c["tokens"], model.args.vocab_size, seed + 2).to(DEVICE)
    return dict(model=model, cache=cache, tokens=tokens, cached=c["cached"], last=c["last"])


def _prepare_verify(c, seed):
    model = _model(c["model"], seed)
    cache = _filled_cache(model, c["cached"], 128, seed + 1)
    depth, mask = _tree(c["nodes"], np.random.default_rng(seed))
    return dict(model=model, cache=cache, cached=c["cached"],
                tokens=_tokens(c["nodes"], model.args.vocab_size, seed + 2)[None].to(DEVICE),
                depth=torch.from_numpy(depth).to(DEVICE), mask=torch.from_numpy(mask).to(DEVICE))


def _pair(c, seed):
    target, draft = PAIRS[c["pair"]]
    vocab = min(be.shape_preset(target).vocab_size, be.shape_preset(draft).vocab_size)
    table = _successors(vocab, seed)
    return _model(target, seed, table), _model(draft, seed + 1, _successors(vocab, seed + 1, table)), vocab


def _prepare_generate(c, seed):
    target, draft, vocab = _pair(c, seed)
    rows = c["prompt"] + c["tokens"] + 8 * (c["depth"] + 2) + c["verify"] + 128
    decoder = be.SpecDecoder(target, draft, c["depth"], c["verify"], 64 * ((rows + 63) // 64))
    decoder.warmup()
    return dict(decoder=decoder, prompt=_tokens(c["prompt"], vocab, seed + 2).pin_memory(), tokens=c["tokens"])


def _prepare_batch(c, seed):
    target, draft, vocab = _pair(c, seed)
    rows = c["prompt"] + (c["tokens"] + 8) * (c["depth"] + 2) + c["verify"] + 128
    decoder = be.BatchSpecDecoder(target, draft, c["depth"], c["verify"], 64 * ((rows + 63) // 64), c["requests"])
    decoder.warmup()
    # prompts of different requests differ in length
    prompts = [_tokens(max(1, c["prompt"] - 5 * r), vocab, seed + 2 + r).pin_memory() for r in range(c["requests"])]
    return dict(decoder=decoder, prompts=prompts, tokens=c["tokens"])


_PREPARE = dict(matmul=_prepare_matmul, rope=_prepare_rope, forward=_prepare_forward, verify=_prepare_verify,
                generate=_prepare_generate, batch=_prepare_batch)


# --------------------------------------------------------------------------------------------------- one pass
def run(state):
    return state["run"](state)


def _run_matmul(s):
    if s["n"] is not None:
        return be.qmm_kernel.matmul_tiled(s["x"], s["w"], s["n"], bias=s["bias"])
    return be.matmul(s["x"], *s["w"], GROUP, bias=s["bias"])[0]


def _run_rope(s):
    return be.rope_positions(s["x"], s["positions"], s["frequencies"], 1.0)


def _run_forward(s):
    cache = s["cache"]
    cache.offset = s["cached"]                             # rewound, as the decode loop rewinds it
    logits = s["model"](s["tokens"][None], cache, logits_last_only=s["last"])
    return [logits, *cache.state]


def _run_verify(s):
    cache = s["cache"]
    cache.offset = s["cached"]
    logits = be.eagle.tree_decoding(s["tokens"], s["mask"], s["depth"], s["model"], cache)
    return [logits, *cache.state]


def _run_generate(s):
    result = s["decoder"].generate(s["prompt"], max_tokens=s["tokens"], N=s["tokens"], clip=True)
    return np.array(result["tokens"], dtype=np.int64)


def _run_batch(s):
    results = s["decoder"].generate(s["prompts"], max_tokens=s["tokens"], N=s["tokens"], clip=True)
    return [np.array(r["tokens"], dtype=np.int64) for r in results]


_RUN = dict(matmul=_run_matmul, rope=_run_rope, forward=_run_forward, verify=_run_verify, generate=_run_generate,
            batch=_run_batch)


# --------------------------------------------------------------------------------------------------- what a pass needs
def _matmul_bytes(n, k):
    return n * k // 2 + 4 * n * k // GROUP                 # packed codes, a scale and a bias per group


def _pass_work(preset, tokens, cached, logits_rows):
    """One pass of ``tokens`` tokens over ``cached`` earlier ones: the weights once, the keys and values the tokens look
    at once, their own written, logits written."""
    a = be.shape_preset(preset)
    h, i, hd = a.hidden_size, a.intermediate_size, a.head_dim
    nq, nkv = a.num_attention_heads * hd, a.num_key_value_heads * hd
    layer = _matmul_bytes(nq + 2 * nkv, h) + _matmul_bytes(h, nq) + 3 * _matmul_bytes(i, h)
    weights = a.num_hidden_layers * layer + _matmul_bytes(a.vocab_size, h)
    kv = a.num_hidden_layers * 2 * nkv * 2 * (cached + tokens)
    linear = a.num_hidden_layers * (h * (nq + 2 * nkv) + nq * h + 3 * h * i)
    attention = a.num_hidden_layers * 2 * nq * tokens * (cached + tokens / 2)
    return dict(bytes=weights + kv + 2 * logits_rows * a.vocab_size,
                flops=2 * (linear * tokens + a.vocab_size * h * logits_rows + attention))


def work(case):
    c, kind = case, case["kind"]
    if kind == "matmul":
        return dict(bytes=_matmul_bytes(c["n"], c["k"]) + 2 * c["rows"] * (c["k"] + c["n"]) + 2 * c["n"] * c["bias"],
                    flops=2 * c["rows"] * c["n"] * c["k"])
    if kind == "rope":
        values = c["batch"] * c["heads"] * c["tokens"] * c["dim"]
        return dict(bytes=4 * values + 4 * c["batch"] * c["tokens"] + 2 * c["dim"], flops=3 * values)
    if kind in ("forward", "verify"):
        tokens = c["tokens"] if kind == "forward" else c["nodes"]
        return _pass_work(c["model"], tokens, c["cached"], 1 if c.get("last") else tokens)
    # a request: the prompt through both models, then the fewest steps that can give the tokens, each of depth + 1
    # passes of the draft and one of the target; requests of a batch share the weights of every step
    requests = c.get("requests", 1)
    target, draft = PAIRS[c["pair"]]
    steps = math.ceil(c["tokens"] / (c["depth"] + 2))
    length = c["prompt"] + c["tokens"] // 2
    parts = [(requests, _pass_work(target, c["prompt"], 0, 1)), (requests, _pass_work(draft, c["prompt"], 0, 0)),
             (steps, _pass_work(target, requests * (c["verify"] + 1), length, requests * (c["verify"] + 1))),
             (steps * (c["depth"] + 1), _pass_work(draft, requests * 8, length, requests * 8))]
    return {k: sum(n * w[k] for n, w in parts) for k in ("bytes", "flops")}


def tolerance(case):
    kind = case["kind"]
    if kind in ("generate", "batch"):
        return "exact"                                      # greedy tokens of contexts with a clear favourite
    if kind in ("matmul", "rope"):
        return {"rel": 1e-3, "max": 4e-3}                   # fp16 results of fp32 sums
    return {"rel": 1e-2, "max": 0.1}                        # fp16 activations through all layers
