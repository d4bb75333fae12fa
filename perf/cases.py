"""What the engine is timed on: steps of the step function over the sizes, batches, contexts and types that
serving meets, and the sampler's draws behind them.

A case is one of two kinds.

``step``: ONE call of ``ModelRunner.step``, which is how tokens reach a model in generation, in trace
replay and in the benchmark: ``decodes`` requests with one token each, whose contexts are spread between
``shortest`` and ``context`` keys, beside ``prompts`` requests with a portion of ``portion`` tokens behind
``behind`` keys.  Weights are random, of the named size of ``velox_b200.config.presets`` with all its
layers; what the caches hold is random too (for the design with a recurrent state it is what the engine
itself makes of the tokens before).  The step hands back logits for every decoded token and for the last
token of every portion; the last layer's pages (and state) come with them, since the step writes them.
``ahead``: the step is queued as ``LLM.generate`` queues it (portions launched kernel by kernel); without it
as ``Engine.step`` and trace replay run it (portions replayed from a captured graph once their shape has
come back).  Steps of single tokens are replayed from the graphs captured at warm-up either way.

``sample``: ONE call of ``Sampler.sample`` on a step's logits.
"""
import gc
import math
import zlib

import numpy as np
import torch

from velox_b200.cache.manager import CacheManager
from velox_b200.config.presets import model_size
from velox_b200.config.registry import architecture_of
from velox_b200.engine.model import CausalLM
from velox_b200.engine.runner import ModelRunner, StepChunk
from velox_b200.sampling.params import SamplingParams
from velox_b200.sampling.sampler import Sampler
from velox_b200.weights.loader import WeightStore

DEVICE = "cuda:0"
STD = 0.02          # of matrices and biases, as in the engine's own random-weights mode
F64 = torch.float64
MOST_CACHE_BYTES = 10 * 10**9
MOST_RECURRENT_TOKENS = 8192


# ------------------------------------------------------------------------------------------ cases
def _step(name, size, decodes=0, context=0, shortest=0, prompts=0, portion=0, behind=0, dtype="bfloat16", page=64,
          ahead=False):
    return {"name": name, "kind": "step", "size": size, "dtype": dtype, "decodes": decodes, "context": context,
            "shortest": shortest or context, "prompts": prompts, "portion": portion, "behind": behind, "page": page,
            "ahead": ahead}


def listed():
    return [
        # The smallest call: four short requests of a tiny model, where launches and the host are everything.
        _step("tiny-decode-4", "tiny-b", decodes=4, context=90, shortest=14, page=8),
        # One user and the smallest published size: every kernel is short, the chain between them is the time.
        _step("0.5b-decode-1", "0.5b", decodes=1, context=701),
        # The benchmark's configuration: batch 8 at 4,096 keys with 16-key pages.
        _step("1.5b-decode-8", "1.5b", decodes=8, context=4096, page=16),
        # A full batch of ragged requests.
        _step("1.5b-decode-64", "1.5b", decodes=64, context=4096, shortest=333),
        # The benchmark's prompt: 2,048 tokens in one step.
        _step("1.5b-prompt-2048", "1.5b", prompts=1, portion=2048),
        # The serving workload of the 7B sizes while decoding: 31 ragged requests (not a power of two) ...
        _step("7b-decode-31", "7b", decodes=31, context=2304, shortest=130),
        # ... and while a prompt comes in, a 512-token portion beside the decoded tokens, queued ahead.
        _step("7b-mixed-512", "7b", decodes=24, context=2304, shortest=130, prompts=1, portion=512, behind=1024, ahead=True),
        # A long prompt of the 14B sizes, its last portion behind all the others.
        _step("14b-portion-2048", "14b", prompts=1, portion=2048, behind=6100, ahead=True),
        # The 32-bit path as trace replay runs it: odd portions beside decoded tokens.
        _step("1.5b-float32-mixed", "1.5b", decodes=3, context=411, shortest=200, prompts=2, portion=75, behind=53,
              dtype="float32", page=16),
        # Attention over a cached latent, gated and normed results, depth mix: eight ragged requests.
        _step("peratar-1.5b-decode-8", "peratar-1.5b", decodes=8, context=4000, shortest=900),
        # Convolutions, a delta rule and windows: a prompt's second portion beside decoded tokens.
        _step("mamivik-0.5b-mixed", "mamivik-0.5b", decodes=5, context=900, shortest=210, prompts=1, portion=500,
              behind=512, ahead=True),
        # The draws behind a full batch: temperature with top-k and top-p.
        {"name": "sample-64", "kind": "sample", "rows": 64, "vocab": 151936, "temperature": 0.7, "top_k": 50, "top_p": 0.9},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    if rng.random() < 0.1:
        return {"kind": "sample", "rows": _log_int(rng, 1, 64), "vocab": rng.choice((151936, 152064)),
                "temperature": round(rng.uniform(0.3, 1.2), 2), "top_k": rng.choice((0, 20, 50, 200)),
                "top_p": rng.choice((1.0, 0.95, 0.9, 0.8))}
    size = rng.choice(("tiny-b", "0.5b", "0.5b", "1.5b", "1.5b", "1.5b", "3b", "3b", "7b", "7b", "14b", "peratar-0.5b",
                       "peratar-1.5b", "mamivik-0.5b", "mamivik-1.5b"))
    dtype = "float32" if size in ("tiny-b", "0.5b", "1.5b") and rng.random() < 0.2 else "bfloat16"
    page = rng.choice((16, 64, 64))
    form = rng.choice(("decode", "decode", "prompt", "mixed"))
    decodes = prompts = portion = behind = context = shortest = 0
    longest = {"tiny-b": 200}.get(size, 1536 if size.startswith("mamivik") else 8192)
    if form != "prompt":
        decodes = _log_int(rng, 1, 4 if dtype == "float32" else 64)
        context = _log_int(rng, 32, longest)
        shortest = rng.randint(max(1, context // 8), context)
    if form != "decode":
        prompts = 1 if rng.random() < 0.7 else 2
        most = {"tiny-b": 48}.get(size, 128 if dtype == "float32" else 2048 // prompts)
        portion = _log_int(rng, 16, most)
        if size == "14b":
            behind = 0 if rng.random() < 0.5 else _log_int(rng, 16, 6000)
        else:
            behind = 0 if rng.random() < 0.5 else _log_int(rng, 16, max(16, longest - 2048) if longest > 4096 else longest // 2)
        if form == "mixed":
            decodes = min(decodes, 31)
    case = _step(None, size, decodes, context, shortest, prompts, portion, behind, dtype, page,
                 ahead=form != "decode" and rng.random() < 0.6)
    del case["name"]
    # Three such states fit the card, and making one stays quick.
    while case["decodes"] > 1 and (
            sum(_contexts(case)) * _cache_bytes_per_key(_config(case)) > MOST_CACHE_BYTES
            or (size.startswith("mamivik") and sum(_contexts(case)) + prompts * behind > MOST_RECURRENT_TOKENS)):
        case["decodes"] //= 2
    return case


def _contexts(case):
    """Keys of every decoded request after the step, spread between the shortest and the longest."""
    n, low, high = case["decodes"], case["shortest"], case["context"]
    if n == 1:
        return [high]
    return [low + int(round((high - low) * math.modf((i + 1) * 0.6180339887498949)[0])) for i in range(n - 1)] + [high]


def _sequences(case):
    """(keys before the step, tokens of the step) of every request."""
    decodes = [(c - 1, 1) for c in _contexts(case)] if case["decodes"] else []
    return decodes + [(case["behind"], case["portion"])] * case["prompts"]


def _config(case):
    return model_size(case["size"])


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


# ------------------------------------------------------------------------------------------ weights
def _tensors(cfg):
    """Checkpoint name -> (shape, how it is drawn): the tensors of a model folder of this configuration.

    A layer changes the stream by a part of what it holds, as in a trained model: the embedding's rows are of
    unit scale, and where nothing norms a layer's result its last matrices are as many times smaller as
    their sum over the layers asks for.  (With one scale for everything the first layers are the whole
    stream, and every later layer multiplies their rounding.)"""
    out = {}
    into_stream = f"over:{math.sqrt(2 * (cfg['num_hidden_layers'] if 'layers' not in cfg else len(cfg['layers'])))}"
    if "layers" not in cfg:
        E, V, I = cfg["hidden_size"], cfg["vocab_size"], cfg["intermediate_size"]
        H, G, D = _heads(cfg)
        out["model.embed_tokens.weight"] = ((V, E), "unit")
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for name, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
                out[p + f"self_attn.{name}_proj.weight"] = ((rows, E), "normal")
                out[p + f"self_attn.{name}_proj.bias"] = ((rows,), "normal")
            out[p + "self_attn.o_proj.weight"] = ((E, H * D), into_stream)
            out[p + "mlp.gate_proj.weight"] = ((I, E), "normal")
            out[p + "mlp.up_proj.weight"] = ((I, E), "normal")
            out[p + "mlp.down_proj.weight"] = ((E, I), into_stream)
            out[p + "input_layernorm.weight"] = ((E,), "one")
            out[p + "post_attention_layernorm.weight"] = ((E,), "one")
        out["model.norm.weight"] = ((E,), "one")
        if not cfg["tie_word_embeddings"]:
            out["lm_head.weight"] = ((V, E), "normal")
        return out
    E, V = cfg["width"], cfg["vocab"]
    out["embed"], out["head"] = ((V, E), "unit"), ((V, E), "normal")
    mamivik = cfg["architecture"] == "Mamivik"
    out["final.norm"] = (() if mamivik else (E,), "one")
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        if mamivik:
            out[p + "norm1"] = out[p + "norm2"] = ((), "one")
            out[p + "canon1"] = ((E, cfg["canon"]["taps"]), "wide")
            out[p + "mlp.gate"] = out[p + "mlp.up"] = ((ff, E), "normal")
            out[p + "mlp.down"] = ((E, ff), into_stream)
        else:
            out[p + "norm1"] = out[p + "norm2"] = ((E,), "one")
            out[p + "rg1"] = out[p + "rg2"] = ((E, E), "normal")
            out[p + "rg1.b"] = out[p + "rg2.b"] = ((E,), "normal")
            out[p + "mlp.up"], out[p + "mlp.up.b"] = ((ff, E), "normal"), ((ff,), "normal")
            out[p + "mlp.down"], out[p + "mlp.down.b"] = ((E, ff), "normal"), ((E,), "normal")
            out[p + "mlp.act"] = ((2,), "normal")
            out[p + "dwa"] = ((i + 2,), "average")
        p += "mix."
        if layer["type"] == "latent_attention":
            H, q_head = m["heads"], m["dim"] + m["rot_dim"]
            if mamivik:
                out[p + "dq"], out[p + "dq.norm"] = ((m["q_rank"], E), "normal"), ((m["q_rank"],), "one")
                out[p + "uq"] = ((H * q_head, m["q_rank"]), "normal")
                out[p + "sink"] = ((H,), "wide")
                out[p + "g"] = ((H * m["vdim"], E), "normal")
            else:
                out[p + "q"] = ((H * q_head, E), "normal")
                out[p + "g"] = ((H, E), "normal")
            if m.get("kv_from") is None:
                out[p + "dkv"] = ((m["kv_rank"] + m["rot_dim"], E), "normal")
                out[p + "dkv.norm"] = ((m["kv_rank"],), "one")
            out[p + "uk"], out[p + "uv"] = ((H * m["dim"], m["kv_rank"]), "normal"), ((H * m["vdim"], m["kv_rank"]), "normal")
            out[p + "o"] = ((E, H * m["vdim"]), into_stream if mamivik else "normal")
        else:
            a, d = m["left"], m["right"]
            for name, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"])):
                out[p + f"left.{name}"], out[p + f"left.{name}.b"] = ((rows, E), "normal"), ((rows,), "normal")
            out[p + "left.o"] = ((E, a["heads"] * a["vdim"]), into_stream)
            inner = d["heads"] * d["dim"]
            rank = max(8, inner // 8 // 8 * 8)
            for name in ("r", "k", "v", "g", "a"):
                out[p + f"right.{name}"] = ((inner, E), "normal")
            out[p + "right.w1"], out[p + "right.w2"] = ((rank, E), "normal"), ((inner, rank), "wide")
            out[p + "right.w0"] = out[p + "right.a.b"] = ((inner,), "wide")
            out[p + "right.norm"], out[p + "right.o"] = ((inner,), "one"), ((E, inner), into_stream)
    return out


def _generator(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) << 32) ^ zlib.crc32(name.encode()))


def _tensor(name, shape, how, seed, dtype):
    values = torch.empty(shape, dtype=dtype, device=DEVICE)
    std = 1.0 if how == "unit" else 10 * STD if how == "wide" else STD / float(how[5:]) if how.startswith("over:") else STD
    values.normal_(0.0, std, generator=_generator(seed, name))
    if how == "one":
        values += 1.0
    elif how == "average":
        values += 1.0 / shape[0]
    return values


class _Weights:
    """A model folder's tensors, made on the GPU from the seed when they are asked for."""

    model_dir = "random weights"

    def __init__(self, cfg, seed, dtype):
        self.tensors, self.seed, self.dtype = _tensors(cfg), seed, dtype

    def names(self):
        return sorted(self.tensors)

    def __contains__(self, name):
        return name in self.tensors

    def shape(self, name):
        return self.tensors[name][0]

    def get(self, name):
        shape, how = self.tensors[name]
        return _tensor(name, shape, how, self.seed, self.dtype)

    def __getitem__(self, name):
        return self.get(name).to(F64)


def _token_ids(case, vocab, seed):
    """All tokens of every request, those before the step first."""
    rng = np.random.default_rng([int(seed), 17])
    return [rng.integers(0, vocab, before + n).tolist() for before, n in _sequences(case)]


def _cached(case, cfg, layer, seed):
    """What a layer's cache holds for all requests before the step, one after the other: (keys, values) of
    the scale that random weights give, or (latent and rotated key part,)."""
    keys = sum(before for before, _ in _sequences(case))
    dtype = _dtype(case)

    def rows(name, heads, dim, std):
        values = torch.empty((keys, heads, dim), dtype=dtype, device=DEVICE)
        return values.normal_(0.0, std, generator=_generator(seed, f"cache.{layer}.{name}"))

    if "layers" not in cfg:
        _, G, D = _heads(cfg)
        std = STD * math.sqrt(cfg["hidden_size"])
        return rows("k", G, D, std), rows("v", G, D, std)
    m = cfg["layers"][layer]["mixer"]
    return (torch.cat([rows("c", 1, m["kv_rank"], 1.0), rows("r", 1, m["rot_dim"], STD * math.sqrt(cfg["width"]))], dim=-1),)


def _recurrent(cfg):
    return cfg.get("architecture") == "Mamivik"


def _heads(cfg):
    heads = cfg["num_attention_heads"]
    return heads, cfg["num_key_value_heads"], cfg.get("head_dim") or cfg["hidden_size"] // heads


# ------------------------------------------------------------------------------------------ a pass
class _Store(WeightStore):
    """Remembers the weights it has made, so that a state can let go of them."""

    def __init__(self, *args):
        super().__init__(*args)
        self.made = []

    def load(self, weight):
        tensor = super().load(weight)
        self.made.append(tensor)
        return tensor


class _Step:
    def __init__(self, runner, chunks, capture, store):
        self.runner, self.chunks, self.capture, self.store = runner, chunks, capture, store

    def __del__(self):
        # Views of a weight that are kept on the weight itself keep it for good.
        for weight in self.store.made:
            vars(weight).clear()


class _Sample:
    def __init__(self, sampler, logits, params, names, draws):
        self.sampler, self.logits, self.params, self.names, self.draws = sampler, logits, params, names, draws


def prepare(case, seed):
    gc.collect()  # models of earlier states that are in reference cycles
    if case["kind"] == "sample":
        rows, vocab = case["rows"], case["vocab"]
        logits = torch.empty((rows, vocab), dtype=torch.float32, device=DEVICE)
        logits.normal_(0.0, 2.0, generator=_generator(seed, "logits"))
        sampler = Sampler(torch.device(DEVICE), vocab, rows, 4096, seed=int(seed))
        params = [SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], seed=int(seed) + r)
                  for r in range(rows)]
        return _Sample(sampler, logits, params, [f"r{r}" for r in range(rows)], [3 * r % 97 for r in range(rows)])
    cfg, dtype, device = _config(case), _dtype(case), torch.device(DEVICE)
    sequences = _sequences(case)
    longest = max(before + n for before, n in sequences)
    page = case["page"]
    arch = architecture_of(cfg)
    spec = arch.build_spec(arch.parse_config(cfg))
    store = _Store(_Weights(cfg, seed, dtype), spec, dtype, device)
    model = CausalLM(spec, store, dtype, device, max_position=longest + 1)
    pages = sum(-(-(before + n) // page) for before, n in sequences) + 1
    cache = CacheManager(model.cache_groups, num_pages=pages, page_size=page, max_model_len=longest + 1,
                         max_num_seqs=len(sequences))
    portions = [n for _, n in sequences if n > 1]
    behind = [before for before, _ in sequences if _recurrent(cfg)]
    runner = ModelRunner(model, cache, max_num_seqs=len(sequences),
                         max_num_batched_tokens=max([len(sequences), case["decodes"] + sum(portions)] + [min(2048, b) for b in behind]))
    tokens = _token_ids(case, model.vocab_size, seed)
    if not portions:
        runner.capture_decode_graphs()  # as the engine's warm-up does
    seqs = []
    for index, (before, n) in enumerate(sequences):
        seq = cache.new_sequence(f"request {index}")
        assert cache.acquire_slot(seq)
        if _recurrent(cfg):
            while seq.num_computed < before:
                n_before = min(2048, before - seq.num_computed)
                assert cache.append_slots(seq, n_before)
                runner.step([StepChunk(seq, tokens[index][seq.num_computed : seq.num_computed + n_before])], capture=False)
                cache.advance(seq, n_before)
            assert cache.append_slots(seq, n)
        else:
            assert cache.append_slots(seq, before + n)
            cache.advance(seq, before)
        seqs.append(seq)
    if not _recurrent(cfg) and any(before for before, _ in sequences):
        slots = torch.cat([_slots(seq, before, page) for seq, (before, _) in zip(seqs, sequences)]).to(device)
        for layer, pages in enumerate(runner.layer_caches):
            if pages.read_only:
                continue
            for pool, rows in zip((pages.k, pages.v), _cached(case, cfg, layer, seed)):
                pool.view(-1, pool.shape[2], pool.shape[3])[slots, :, : rows.shape[2]] = rows
    chunks = [StepChunk(seq, ids[before:], (n - 1,)) for seq, ids, (before, n) in zip(seqs, tokens, sequences)]
    return _Step(runner, chunks, not case["ahead"], store)


def _slots(seq, count, page):
    positions = np.arange(count)
    return torch.from_numpy(np.asarray(seq.tables[0], dtype=np.int64)[positions // page] * page + positions % page)


def run(state):
    if isinstance(state, _Sample):
        return {"tokens": state.sampler.sample(state.logits, state.params, state.names, state.draws)}
    logits = state.runner.step(state.chunks, capture=state.capture)
    last = state.runner.layer_caches[-1]
    # (The last state row belongs to padding.)
    return {"logits": logits, "keys": last.k, "values": None if last.v is last.k else last.v,
            "state": None if last.state is None else last.state[:-1]}


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _cache_bytes_per_key(cfg, element=2):
    """Bytes of one key and value in all layers that cache their own."""
    if "layers" not in cfg:
        _, G, D = _heads(cfg)
        return cfg["num_hidden_layers"] * 2 * G * D * element
    total = 0
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            total += 0 if m.get("kv_from") is not None else (m["kv_rank"] + m["rot_dim"]) * element
        else:
            total += 2 * m["left"]["kv_heads"] * m["left"]["dim"] * element
    return total


def _attention_shapes(cfg):
    """(query heads, key and value dims of a head together, window or None) of every layer."""
    if "layers" not in cfg:
        H, _, D = _heads(cfg)
        return [(H, 2 * D, None)] * cfg["num_hidden_layers"]
    out = []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "latent_attention":
            out.append((m["heads"], m["dim"] + m["rot_dim"] + m["vdim"], m.get("mask", {}).get("size")))
        else:
            out.append((m["left"]["heads"], m["left"]["dim"] + m["left"]["vdim"], m["left"]["mask"]["size"]))
    return out


def work(case):
    if case["kind"] == "sample":
        values = case["rows"] * case["vocab"]
        return {"bytes": 4 * values + 4 * case["rows"], "flops": 4 * values}
    cfg = _config(case)
    element = 4 if case["dtype"] == "float32" else 2
    sequences = _sequences(case)
    tokens, wanted = sum(n for _, n in sequences), len(sequences)
    vocab, width = (cfg["vocab_size"], cfg["hidden_size"]) if "layers" not in cfg else (cfg["vocab"], cfg["width"])
    # Every matrix once and every product with it; the embedding's rows of the step's tokens; the head on the wanted rows.
    matrices = sum(math.prod(shape) for name, (shape, _) in _tensors(cfg).items()
                   if len(shape) == 2 and shape != (vocab, width))
    vectors = sum(math.prod(shape) for shape, _ in _tensors(cfg).values() if len(shape) < 2)
    bytes_ = (matrices + vocab * width + tokens * width) * element + 4 * vectors + 4 * wanted * vocab
    flops = 2 * matrices * tokens + 2 * vocab * width * wanted
    per_key = _cache_bytes_per_key(cfg, element)
    shapes = _attention_shapes(cfg)
    for before, n in sequences:
        bytes_ += n * per_key
        seen = {}
        for heads, dims, window in shapes:
            if window not in seen:
                first = before + 1
                if window is None or before + n <= window:
                    pairs = n * (first + before + n) // 2
                else:
                    pairs = sum(min(window, first + i) for i in range(n))
                seen[window] = pairs, before if window is None else min(before, window + n - 1)
            flops += 2 * heads * dims * seen[window][0]
        # (The designs here have one window or none in all their layers.)
        bytes_ += per_key * max(read for _, read in seen.values())
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 5e-5}
    return {"rel": 0.02, "max": 0.2}


# ------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    if case["kind"] == "sample":
        return None
    cfg = _config(case)
    w = _Weights(cfg, seed, _dtype(case))
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    tokens = _token_ids(case, vocab, seed)
    sequences = _sequences(case)
    if "layers" not in cfg:
        logits = _exact_qwen2(case, cfg, w, tokens, sequences, seed)
    elif _recurrent(cfg):
        logits = torch.stack([_exact_mamivik(cfg, w, ids) for ids in tokens])
    else:
        logits = _exact_peratar(case, cfg, w, tokens, sequences, seed)
    return {"logits": logits, "keys": None, "values": None, "state": None}


def _rms(x, weight, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _spans(sequences):
    """(rows of the step, rows of the cached keys, keys before) of every request."""
    row = key = 0
    for before, n in sequences:
        yield slice(row, row + n), slice(key, key + before), before
        row, key = row + n, key + before


def _attend(q, k, v, first, scale, window=None, sink=None):
    """q [n, H, d] at positions first ..; k [s, G, d], v [s, G, e] from position 0 on."""
    n, H, _ = q.shape
    G = k.shape[1]
    q = q.view(n, G, H // G, -1)
    scores = torch.einsum("tghd,sgd->ghts", q, k).mul_(scale)
    behind = torch.arange(first, first + n, device=q.device)[:, None] - torch.arange(k.shape[0], device=q.device)[None]
    hidden = behind < 0 if window is None else (behind < 0) | (behind >= window)
    scores.masked_fill_(hidden, -math.inf)
    if sink is not None:
        scores = torch.cat([scores, sink.view(G, H // G, 1, 1).expand(-1, -1, n, 1)], dim=-1)
    probs = torch.softmax(scores, dim=-1)[..., : k.shape[0]]
    return torch.einsum("ghts,sge->tghe", probs, v).reshape(n, H, -1)


def _last_rows(x, sequences):
    rows = np.cumsum([n for _, n in sequences]) - 1
    return x[torch.from_numpy(rows).to(x.device)]


def _positions(sequences):
    return torch.cat([torch.arange(before, before + n) for before, n in sequences])


def _exact_qwen2(case, cfg, w, tokens, sequences, seed):
    H, G, D = _heads(cfg)
    eps = cfg["rms_norm_eps"]
    ids = [t for span, (before, _) in zip(tokens, sequences) for t in span[before:]]
    # The design forms the angles in 32 bits.
    exponent = torch.arange(0, D, 2, dtype=torch.float32) / D
    angles = torch.outer(_positions(sequences).to(torch.float32), 1.0 / (cfg["rope_theta"] ** exponent)).to(F64)
    cos, sin = angles.cos().to(DEVICE)[:, None], angles.sin().to(DEVICE)[:, None]

    def rotate(x):
        low, high = x.chunk(2, dim=-1)
        return torch.cat([low * cos - high * sin, low * sin + high * cos], dim=-1)

    x = w.get("model.embed_tokens.weight")[torch.tensor(ids, device=DEVICE)].to(F64)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"], eps)
        q, k, v = (h @ w[p + f"self_attn.{n}_proj.weight"].T + w[p + f"self_attn.{n}_proj.bias"] for n in "qkv")
        q, k, v = rotate(q.view(-1, H, D)), rotate(k.view(-1, G, D)), v.view(-1, G, D)
        old_k, old_v = _cached(case, cfg, i, seed)
        out = torch.cat([_attend(q[new], torch.cat([old_k[old].to(F64), k[new]]), torch.cat([old_v[old].to(F64), v[new]]), before, D ** -0.5)
                         for new, old, before in _spans(sequences)])
        x = x + out.reshape(-1, H * D) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, w[p + "post_attention_layernorm.weight"], eps)
        h = torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)
        x = x + h @ w[p + "mlp.down_proj.weight"].T
    x = _rms(_last_rows(x, sequences), w["model.norm.weight"], eps)
    return x @ w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"].T


def _layer_norm(x, weight, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _exact_peratar(case, cfg, w, tokens, sequences, seed):
    eps = cfg["norm"]["eps"]
    ids = [t for span, (before, _) in zip(tokens, sequences) for t in span[before:]]
    positions = _positions(sequences).to(F64)

    def rotate(x, rot):  # pairs of neighbours
        dims = rot["dims"]
        angles = torch.outer(positions, rot["base"] ** (-torch.arange(0, dims, 2, dtype=F64) / dims)).to(DEVICE)[:, None]
        c, s = angles.cos(), angles.sin()
        u, v = x[..., :dims:2], x[..., 1:dims:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2), x[..., dims:]], dim=-1)

    x = w.get("embed")[torch.tensor(ids, device=DEVICE)].to(F64)
    results, cached = [x], {}
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        H, d, rank = m["heads"], m["dim"], m["kv_rank"]
        source = m.get("kv_from")
        if source is None:
            down = x @ w[p + "mix.dkv"].T
            new = torch.cat([_rms(down[:, :rank], w[p + "mix.dkv.norm"], eps), rotate(down[:, None, rank:], m["rot"])[:, 0]], dim=-1)
            old, = _cached(case, cfg, i, seed)
            cached[i] = [torch.cat([old[before_rows, 0].to(F64), new[rows]]) for rows, before_rows, _ in _spans(sequences)]
            source = i
        q = (x @ w[p + "mix.q"].T).view(-1, H, d + m["rot_dim"])
        q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"])], dim=-1)
        out = []
        for c, (rows, _, before) in zip(cached[source], _spans(sequences)):
            keys = (c[:, :rank] @ w[p + "mix.uk"].T).view(-1, H, d)
            keys = torch.cat([keys, c[:, None, rank:].expand(-1, H, -1)], dim=-1)
            out.append(_attend(q[rows], keys, (c[:, :rank] @ w[p + "mix.uv"].T).view(-1, H, m["vdim"]), before, m["scale"]))
        out = torch.cat(out) * torch.sigmoid(x @ w[p + "mix.g"].T)[..., None]
        out = (out.flatten(1) @ w[p + "mix.o"].T) * torch.sigmoid(x @ w[p + "rg1"].T + w[p + "rg1.b"])
        x = x + _layer_norm(out, w[p + "norm1"], eps)
        z = x @ w[p + "mlp.up"].T + w[p + "mlp.up.b"]
        a, b = torch.nn.functional.softplus(w[p + "mlp.act"])
        z = torch.where(z > 0, a * z * z + z / 2, (0.5 + b) * (torch.expm1(z.clamp(max=0)) - z) + z / 2)
        out = (z @ w[p + "mlp.down"].T + w[p + "mlp.down.b"]) * torch.sigmoid(x @ w[p + "rg2"].T + w[p + "rg2.b"])
        results.append(x + _layer_norm(out, w[p + "norm2"], eps))
        x = torch.einsum("j,jte->te", w[p + "dwa"], torch.stack(results))
    logits = _layer_norm(_last_rows(x, sequences), w["final.norm"], eps) @ w["head"].T
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])


def _exact_mamivik(cfg, w, ids):
    """The logits behind one whole sequence."""
    eps, T, taps = cfg["norm"]["eps"], len(ids), cfg["canon"]["taps"]
    positions = torch.arange(T, dtype=F64)

    def rotate(x, rot):  # dim i of the first ``dims`` with dim i + dims / 2, slow pairs stretched
        dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
        i = torch.arange(dims // 2, dtype=F64)
        f, magnitude = base ** (-2.0 * i / dims), 1.0
        if s:
            turn = [dims * math.log(s["original"] / (2.0 * math.pi * s[t])) / (2.0 * math.log(base)) for t in ("fast", "slow")]
            low, high = max(math.floor(turn[0]), 0), min(math.ceil(turn[1]), dims - 1)
            ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
            f, magnitude = f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0
        angles = torch.outer(positions, f).to(DEVICE)[:, None]
        c, s = angles.cos() * magnitude, angles.sin() * magnitude
        u, v = x[..., : dims // 2], x[..., dims // 2 : dims]
        return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)

    x = w.get("embed")[torch.tensor(ids, device=DEVICE)].to(F64)
    for index, layer in enumerate(cfg["layers"]):
        L, m = f"l{index}.", layer["mixer"]
        h = _rms(x, w[L + "norm1"], eps)
        padded, conv = torch.cat([h.new_zeros(taps - 1, h.shape[1]), h]), w[L + "canon1"]
        h = h + sum(padded[j : j + T] * conv[:, j] for j in range(taps))
        if layer["type"] == "latent_attention":
            p = L + "mix."
            H, d, rank = m["heads"], m["dim"], m["kv_rank"]
            q = (_rms(h @ w[p + "dq"].T, w[p + "dq.norm"], eps) @ w[p + "uq"].T).view(T, H, -1)
            q = torch.cat([q[..., :d], rotate(q[..., d:], m["rot"])], dim=-1)
            down = h @ w[p + "dkv"].T
            c = _rms(down[:, :rank], w[p + "dkv.norm"], eps)
            keys = torch.cat([(c @ w[p + "uk"].T).view(T, H, d), rotate(down[:, None, rank:], m["rot"]).expand(-1, H, -1)], dim=-1)
            out = _attend(q, keys, (c @ w[p + "uv"].T).view(T, H, -1), 0, m["scale"], m["mask"]["size"], w[p + "sink"])
            x = x + (out.flatten(1) * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T
        else:
            p, a = L + "mix.left.", m["left"]
            q = (h @ w[p + "q"].T + w[p + "q.b"]).view(T, a["heads"], -1)
            k = (h @ w[p + "k"].T + w[p + "k.b"]).view(T, a["kv_heads"], -1)
            out = _attend(rotate(q, a["rot"]), rotate(k, a["rot"]), k, 0, a["scale"], a["mask"]["size"])
            left = out.flatten(1) @ w[p + "o"].T
            p, d = L + "mix.right.", m["right"]
            H, D = d["heads"], d["dim"]
            r, k, v = (h @ w[p + n].T for n in ("r", "k", "v"))
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"]))
            remove = torch.sigmoid(h @ w[p + "a"].T + w[p + "a.b"])
            r, k, v, decay, remove = (t.view(T, H, D) for t in (r, k, v, decay, remove))
            unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            # S <- decay S - (remove unit) (unit^T S) + k v^T,  out = S^T r, with the heads side by side.
            out, S = torch.empty_like(v), v.new_zeros(H, D, D)
            remove = (remove * unit)[..., None]
            unit, decay, r, add = unit[:, :, None], decay[..., None], r[:, :, None], k[..., None] * v[:, :, None]
            for t in range(T):
                S = torch.baddbmm(decay[t] * S + add[t], remove[t], unit[t] @ S, alpha=-1)
                out[t] = (r[t] @ S)[:, 0]
            out = _rms(out, 1.0, eps).reshape(T, H * D) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)
            x = x + m["left_scale"] * left + m["right_scale"] * (out @ w[p + "o"].T)
        h = _rms(x, w[L + "norm2"], eps)
        h = torch.nn.functional.gelu(h @ w[L + "mlp.gate"].T, approximate="tanh") * (h @ w[L + "mlp.up"].T)
        x = x + h @ w[L + "mlp.down"].T
    return (_rms(x[-1], w["final.norm"], eps)) @ w["head"].T
