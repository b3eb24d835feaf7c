"""Performance cases: steps of the three model families as a serving loop or a trace replay runs them.

A case is one step of one model: `decode` sequences that each add one token to a context of `context_low`..`context_high`
tokens, and `prompts` portions of `prompt_low`..`prompt_high` tokens behind `prefix_low`..`prefix_high` cached ones.
Sizes inside a step are spread evenly over those ranges.  Pure decode steps replay from a CUDA graph, as in the serving
engine; LFM2 ones include the upload of the step's metadata and the download of the sampled ids (`serve_step`), those of
the layer-stack models and prompts leave their logits.  Weights, caches and recurrent state are random.

Outputs are the logits, the recurrent state and convolution inputs of all sequences, and the key/value caches.  Sampled ids
are left out: they follow from the logits, and with random weights the two largest of 65536 logits are too often closer
than bf16 resolves.
"""
from __future__ import annotations

import ctypes
import importlib
import math
import zlib

import numpy as np
import torch

_PACKAGE = "lfm25-inference_b200"
_abi = importlib.import_module(_PACKAGE + "._abi")
fegidra = importlib.import_module(_PACKAGE + ".fegidra")
lfm_model = importlib.import_module(_PACKAGE + ".model")
ops = importlib.import_module(_PACKAGE + ".ops")
ribivik = importlib.import_module(_PACKAGE + ".ribivik")
stack = importlib.import_module(_PACKAGE + ".stack")
workloads = importlib.import_module(_PACKAGE + ".workloads")

PAGE = 16
TAPS = 4
DECAY_RANK = 64
FP8_MAXIMUM_TOKENS = 256          # larger steps of the LFM2 model run their FP8 sites in BF16


def _case(name, family, *, size="2048", dtype="bfloat16", fp8=False, decode=0, context=(0, 0), prompts=0, prompt=(0, 0),
          prefix=(0, 0)) -> dict:
    case = {"family": family, "size": size, "dtype": dtype, "fp8": fp8, "decode": decode, "context_low": context[0],
            "context_high": context[1], "prompts": prompts, "prompt_low": prompt[0], "prompt_high": prompt[1],
            "prefix_low": prefix[0], "prefix_high": prefix[1]}
    return case if name is None else {"name": name, **case}


def listed() -> list[dict]:
    return [
        # one interactive user of the FP8 deployment: weight streaming and launches
        _case("lfm2 decode 1 fp8", "lfm2", fp8=True, decode=1, context=(1024, 1024)),
        # a lightly loaded BF16 server, an odd number of sequences
        _case("lfm2 decode 23 bf16", "lfm2", decode=23, context=(61, 2309)),
        # the headline serving step: a full batch of mixed contexts under the FP8 policy
        _case("lfm2 decode 128 fp8", "lfm2", fp8=True, decode=128, context=(128, 4096)),
        # a continuous-batching step in which one prompt's remainder joins the running decodes
        _case("lfm2 mixed 31 and 201 fp8", "lfm2", fp8=True, decode=31, context=(97, 3001), prompts=1, prompt=(201, 201)),
        # a full prefill step: eight chunks of 512 tokens at every depth of long prompts
        _case("lfm2 prompts 8x512", "lfm2", fp8=True, prompts=8, prompt=(512, 512), prefix=(0, 3584)),
        # the layer-stack designs: a busy decode batch each
        _case("fegidra decode 32", "fegidra", decode=32, context=(128, 4096)),
        _case("ribivik decode 32", "ribivik", decode=32, context=(128, 4096)),
        # a batch of fresh prompts of unequal lengths
        _case("fegidra prompts 7x300-700", "fegidra", prompts=7, prompt=(300, 700)),
        # one long prompt in one step: the recurrences run over thousands of tokens
        _case("fegidra prompt 4096", "fegidra", prompts=1, prompt=(4096, 4096)),
        _case("ribivik prompt 4096", "ribivik", prompts=1, prompt=(4096, 4096)),
        # a smaller model with wider heads, second portions of prompts
        _case("ribivik-1024 prompts 8x512", "ribivik", size="1024", prompts=8, prompt=(512, 512), prefix=(512, 512)),
        # the 32-bit replay of a given text, as the trace program does it
        _case("fegidra-1024 replay 250 f32", "fegidra", size="1024", dtype="float32", prompts=1, prompt=(250, 250)),
    ]


def _log_uniform(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "prompts", "prompts", "mixed", "replay"))
    family = rng.choice(("lfm2", "fegidra", "ribivik"))
    size = "2048" if family == "lfm2" else rng.choice(("2048", "2048", "1024"))
    fp8 = family == "lfm2" and rng.random() < 0.6
    if kind == "decode":
        low = _log_uniform(rng, 17, 2048)
        return _case(None, family, size=size, fp8=fp8, decode=_log_uniform(rng, 1, 128 if family == "lfm2" else 64),
                     context=(low, _log_uniform(rng, low, 4096)))
    if kind == "mixed":
        low = _log_uniform(rng, 17, 1024)
        tokens = _log_uniform(rng, 5, 900)
        return _case(None, family, size=size, fp8=fp8, decode=_log_uniform(rng, 1, 48),
                     context=(low, _log_uniform(rng, low, 3000)), prompts=rng.randint(1, 2), prompt=(tokens, tokens))
    if kind == "replay":
        family = family if family != "lfm2" else "fegidra"
        tokens = _log_uniform(rng, 16, 250)
        return _case(None, family, size="1024", dtype="float32", prompts=1, prompt=(tokens, tokens))
    prompts = rng.randint(1, 8)
    most = 4000 // prompts
    high = _log_uniform(rng, 40, most)
    prefix = rng.choice((0, 0, rng.randint(1, 1500))) if prompts * high <= 2500 else 0
    return _case(None, family, size=size, fp8=fp8, prompts=prompts, prompt=(max(1, int(high * rng.uniform(0.4, 1.0))), high),
                 prefix=(prefix, prefix))


# ------------------------------------------------------------------------------------------------ sizes of a case

ATTENTION_LAYERS = (2, 5, 8, 10, 12, 14)


def _config(case) -> dict:
    """config.json of the layer-stack models: the sizes of the LFM2 model, and a narrower one with wider heads."""
    wide = case["size"] == "2048"
    width, ff, vocab, count = (2048, 12288, 65536, 16) if wide else (1024, 6144, 32768, 8)
    chosen = ATTENTION_LAYERS if wide else (2, 5)
    if case["family"] == "fegidra":
        dim = 64 if wide else 128
        heads, kv_heads, chunk = (32, 8, 8192) if wide else (8, 2, 512)
        attention = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "mask": {"size": chunk},
                     "rot": {"base": 10000.0, "dims": dim}, "scale": dim ** -0.5}
        recurrent, names = {"heads": 32 if wide else 16, "dim": 64}, ("attention", "general_delta")
        shared = {"canon": {"taps": TAPS}}
    else:
        heads, rot_dim, q_rank, kv_rank = (32, 64, 768, 512) if wide else (16, 32, 384, 256)
        attention = {"heads": heads, "dim": 64, "rot_dim": rot_dim, "vdim": 64, "q_rank": q_rank, "kv_rank": kv_rank,
                     "rot": {"base": 10000.0, "dims": rot_dim}, "scale": (64 + rot_dim) ** -0.5}
        ssm_heads, state, groups = (64, 128, 8) if wide else (32, 64, 1)
        recurrent = {"heads": ssm_heads, "vdim": 64, "state": state, "groups": groups, "norm_groups": groups, "conv": TAPS}
        names, shared = ("latent_attention", "mamba2"), {"logit_softcap": 30.0}
    return {"vocab": vocab, "width": width, "norm": {"eps": 1e-5}, **shared,
            "layers": [{"type": names[0] if index in chosen else names[1],
                        "mixer": attention if index in chosen else recurrent, "mlp": {"kind": "dense", "ff": ff}}
                       for index in range(count)]}


def _spread(low: int, high: int, count: int) -> np.ndarray:
    return np.round(np.linspace(low, high, count)).astype(np.int64)


def _segments(case) -> tuple[np.ndarray, np.ndarray]:
    """(cached tokens, new tokens) of every sequence of the step, decodes first."""
    prefixes = np.concatenate([_spread(case["context_low"], case["context_high"], case["decode"]),
                               _spread(case["prefix_low"], case["prefix_high"], case["prompts"])])
    chunks = np.concatenate([np.ones(case["decode"], np.int64),
                             _spread(case["prompt_low"], case["prompt_high"], case["prompts"])])
    return prefixes, chunks


def _seen(prefix: int, chunk: int, limit: int) -> tuple[float, float]:
    """(query-key pairs, cached keys needed) of one sequence whose tokens see their own `limit`-token piece (0: all)."""
    positions = prefix + np.arange(chunk, dtype=np.float64)
    pairs = (positions % limit if limit else positions) + 1
    first = (prefix // limit * limit) if limit else 0
    return float(pairs.sum()), float(prefix - first)


def work(case) -> dict:
    prefixes, chunks = _segments(case)
    tokens, sequences = int(chunks.sum()), len(chunks)
    element = 4 if case["dtype"] == "float32" else 2
    if case["family"] == "lfm2":
        layers = [("attention" if index in ATTENTION_LAYERS else "conv") for index in range(16)]
        fp8 = case["fp8"] and tokens <= FP8_MAXIMUM_TOKENS
        matrices, small, vocab, width, limit = 0.0, 0.0, 65536, 2048, 0
        weight_bytes = 0.0
        for index, kind in enumerate(layers):
            mixer = 2048 * 2048 * 2 + 2 * 512 * 2048 if kind == "attention" else 6144 * 2048 + 2048 * 2048
            up, down = 2 * 8192 * 2048, 8192 * 2048
            matrices += mixer + up + down
            weight_bytes += 2 * mixer + up * (1 if fp8 and index in lfm_model.FP8_GATE_UP_LAYERS else 2) + \
                down * (1 if fp8 and index in lfm_model.FP8_DOWN_LAYERS else 2)
        head_bytes = vocab * width * (1 if fp8 else 2)
        attentions, cached, per_pair, state = 6, 2 * 512 * 2, 4 * 2048, 10 * 2048 * 2 * 2 * 2
    else:
        node = _config(case)
        vocab, width = node["vocab"], node["width"]
        matrices, state, small, limit = 0.0, 0.0, 0.0, 0
        attentions = cached = per_pair = 0
        for layer in node["layers"]:
            mixer, ff = layer["mixer"], layer["mlp"]["ff"]
            matrices += 2 * ff * width
            if layer["type"] == "attention":
                heads, groups, dim = mixer["heads"], mixer["kv_heads"], mixer["dim"]
                matrices += (2 * heads + 2 * groups) * dim * width
                attentions, cached, per_pair = attentions + 1, 2 * groups * dim * element, 4 * heads * dim
                limit = mixer["mask"]["size"]
            elif layer["type"] == "latent_attention":
                heads, dim, rot, vdim = mixer["heads"], mixer["dim"], mixer["rot_dim"], mixer["vdim"]
                matrices += (mixer["q_rank"] + mixer["kv_rank"] + rot + 2 * heads * vdim) * width + \
                    mixer["q_rank"] * heads * (dim + rot) + mixer["kv_rank"] * heads * (dim + vdim)
                attentions, cached = attentions + 1, (mixer["kv_rank"] + rot) * element
                per_pair = 2 * heads * (dim + rot + vdim)
            elif layer["type"] == "general_delta":
                inner = mixer["heads"] * mixer["dim"]
                matrices += 6 * inner * width + DECAY_RANK * (width + inner)
                small += 8 * inner * mixer["dim"]
                state += 2 * 4 * inner * mixer["dim"]
            else:
                inner = mixer["heads"] * mixer["vdim"]
                matrices += (3 * inner + 2 * mixer["groups"] * mixer["state"] + mixer["heads"]) * width
                small += 5 * inner * mixer["state"]
                state += 2 * 4 * inner * mixer["state"]
        weight_bytes, head_bytes = 2 * matrices, 2 * vocab * width
    pairs = keys = 0.0
    for prefix, chunk in zip(prefixes, chunks):
        one = _seen(int(prefix), int(chunk), limit)
        pairs, keys = pairs + one[0], keys + one[1]
    logit_bytes = sequences * vocab * (2 if case["family"] == "lfm2" else 4)
    return {"bytes": weight_bytes + head_bytes + attentions * cached * (keys + tokens) + sequences * state +
            tokens * width * 2 + logit_bytes,
            "flops": 2.0 * matrices * tokens + 2.0 * vocab * width * sequences + attentions * per_pair * pairs +
            small * tokens}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    # bf16 activations through sixteen layers of random matrices: two routes of the same step (other order of the sums in
    # its GEMMs, attention or recurrence) differ by 0.5 to 2 % here; in FP8 sites a rounding of an activation can become a
    # step of its E4M3 code
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------------------ inputs

def _normal(name: str, seed: int, shape, device="cuda") -> torch.Tensor:
    generator = torch.Generator(device=device).manual_seed(zlib.crc32(name.encode()) * 1000003 + seed)
    return torch.randn(tuple(shape), generator=generator, device=device)


def _source(case, seed: int):
    """`source(name, shape)` for the checkpoint tensors of a layer-stack model, bf16."""
    from_one = ("norm1", "norm1b", "norm2", "norm2b") if case["family"] == "ribivik" else ()   # stored as distance from one

    def source(name, shape):
        last, values = name.split(".")[-1], _normal(name, seed, shape)
        if last == "act":
            values = torch.tensor([0.5, 0.3, 0.2, 0.0], device="cuda")
        elif last in from_one or (from_one and name == "final.norm"):
            values = 0.1 * values
        elif last in ("norm", "norm1", "norm2"):
            values = 1.0 + 0.1 * values
        elif last == "dt_bias":
            values = values - 3.0
        else:
            values = values * (shape[1] ** -0.5 if len(shape) == 2 else 0.1)
        return values.to(torch.bfloat16)
    return source


class _Handles:
    """Executor and library handle of a state, closed when neither it nor a view of their memory is left."""

    def __init__(self, executor, blaslt):
        self.executor, self.blaslt = executor, blaslt

    def __del__(self):
        torch.cuda.synchronize()
        self.executor.close()
        self.blaslt.close()


class _DeviceArray:
    """Memory of the library, for torch.as_tensor; `owner` lives as long as the tensor."""

    def __init__(self, owner, pointer: int, shape, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": tuple(shape), "typestr": typestr, "version": 3}


class _State:
    pass


def _layout(case, seed: int):
    prefixes, chunks = _segments(case)
    pages = int(((prefixes + chunks + PAGE - 1) // PAGE).sum())
    return workloads.mixed_step_batch(seed % (1 << 31), prefixes, chunks, pages)


def _token_ids(case, seed: int, count: int) -> np.ndarray:
    vocab = 65536 if case["family"] == "lfm2" else _config(case)["vocab"]
    return np.random.default_rng(seed + 77).integers(0, vocab, size=count).astype(np.uint32)


def _cache_value(name: str, seed: int, tensor: torch.Tensor) -> None:
    tensor.copy_(_normal(name, seed, tensor.shape).to(tensor.dtype))


def _as_trained(model) -> None:
    """Scales the random LFM2 weights (by powers of two) so that the residual stream is carried through the layers, each
    adding a small part, as in a trained model.  Otherwise every layer's rounding is amplified by the ones behind it and
    two correct steps differ by as much as the logits of an FP8 model."""
    def scale(site, factor):
        site.weight.mul_(factor)
        site.weight_amax *= factor
    scale(model.lm_head, 32.0)                    # shares the embedding's memory
    for layer in model.layers:
        for name in ("conv_output", "output", "down"):
            if name in layer.linears:
                scale(layer.linears[name], 1.0 / 32.0)
    model._build_struct()


def _fresh(case) -> bool:
    """All sequences start in this step: their recurrent state is zero."""
    prefixes, _ = _segments(case)
    return bool((prefixes == 0).all())


def prepare(case, seed):
    """Model, caches of the tokens seen so far, step metadata and executor."""
    seed = int(seed)
    state = _State()
    state.case, state.layout = case, _layout(case, seed)
    state.ids = _token_ids(case, seed, state.layout.num_tokens)
    slots, pages = state.layout.num_segments, state.layout.num_pages
    device = torch.device("cuda")
    state.stream = torch.cuda.Stream()
    if case["family"] == "lfm2":
        model = lfm_model.RandomModel(seed, device, pages, slots, fp8_policy=case["fp8"])
        _as_trained(model)
        state.caches = [layer.tensors[name] for layer in model.layers if layer.is_attention
                        for name in ("key_cache", "value_cache")]
        state.recurrent = [layer.tensors["conv_state"] for layer in model.layers if not layer.is_attention]
        state.histories = []
    else:
        config = _config(case)
        source = _source(case, seed)
        if case["family"] == "fegidra":
            model = fegidra.build(fegidra.FegidraConfig.from_json(config), source, lambda name: (DECAY_RANK,), device, pages,
                                  slots, case["dtype"])
        else:
            model = ribivik.build(ribivik.RibivikConfig.from_json(config), source, device, pages, slots, case["dtype"])
        state.caches = [cache for pair in model.caches for cache in pair]
        state.recurrent, state.histories = _record_views(model, config)
    state.model = model
    if state.layout.prefixes.any():
        for index, cache in enumerate(state.caches):
            _cache_value(f"cache {index}", seed, cache)
    if not _fresh(case):
        for index, tensor in enumerate(state.recurrent):
            _cache_value(f"state {index}", seed, tensor)
        for index, tensor in enumerate(state.histories):
            _cache_value(f"history {index}", seed, tensor)
    torch.cuda.synchronize()
    with torch.cuda.stream(state.stream):
        _prepare_step(state)
    state.stream.synchronize()
    return state


def _record_views(model, config):
    """Per layer the recurrent matrices and the convolution's inputs of all slots, as views of the records."""
    records = model.records.view(model.num_request_slots, model.record_bytes)
    slots, recurrent, histories = model.num_request_slots, [], []

    def view(offset, shape, dtype):
        size = math.prod(shape) * torch.empty(0, dtype=dtype).element_size()
        return records[:, offset:offset + size].view(dtype).view(slots, *shape)

    for index, layer in enumerate(config["layers"]):
        struct, mixer = model.struct.layers[index], layer["mixer"]
        channels = config["width"]
        if layer["type"] == "general_delta":
            recurrent.append(view(struct.state_offset, (mixer["heads"], mixer["dim"], mixer["dim"]), torch.float32))
        elif layer["type"] == "mamba2":
            recurrent.append(view(struct.state_offset, (mixer["heads"], mixer["state"], mixer["vdim"]), torch.float32))
            channels = mixer["heads"] * mixer["vdim"] + 2 * mixer["groups"] * mixer["state"]
        if layer["type"] != "latent_attention":
            histories.append(view(struct.conv_offset, (TAPS - 1, channels), model.dtype))
    return recurrent, histories


def _prepare_step(state) -> None:
    case, layout, model = state.case, state.layout, state.model
    device = torch.device("cuda")
    tokens, rows = layout.num_tokens, layout.num_segments
    blaslt = ops.BlasLt()
    blaslt.bind_current_stream()
    lfm2 = case["family"] == "lfm2"
    if lfm2:
        state.executor = lfm_model.DecodeExecutor(blaslt, tokens, rows if case["prompts"] else None)
    else:
        state.executor = stack.StackExecutor(blaslt, model, tokens, rows)
    state.handles = _Handles(state.executor, blaslt)
    if case["prompts"]:
        state.batch = lfm_model.RaggedBatch(device, layout, state.ids)
    else:
        tables = layout.block_tables
        state.batch = lfm_model.DecodeBatch(device, tables, layout.segment_slots, layout.prefixes.astype(np.uint32),
                                            state.ids, int(layout.prefixes.max()) + 1)
        state.metadata = torch.from_numpy(np.concatenate(
            [state.ids, layout.prefixes.astype(np.uint32), layout.segment_slots]).view(np.int32).copy()).pin_memory()
    state.sampled = torch.zeros(rows, dtype=torch.int32).pin_memory()
    if lfm2:
        pointer = _abi.library().lfm25_decode_executor_logits(state.executor._handle)
        state.logits = torch.as_tensor(_DeviceArray(state.handles, pointer, (rows, model.vocab), "<i2"),
                                       device="cuda").view(torch.bfloat16)
    else:
        state.logits = torch.zeros((rows, model.vocab), dtype=torch.float32).pin_memory()


def run(state):
    """One step, and what it leaves behind."""
    case = state.case
    with torch.cuda.stream(state.stream):
        if case["family"] == "lfm2":
            if case["prompts"]:
                state.executor.forward_ragged(state.model, state.batch, use_fp8=case["fp8"])
                state.executor.download_sampled(state.sampled)
            else:
                state.executor.serve_step(state.model, state.batch, state.metadata, state.sampled, use_fp8=case["fp8"])
        else:
            if case["prompts"]:
                state.executor.forward_ragged(state.batch)
            else:
                state.executor.step_graph(state.batch, advance=False)
            # logits for a sampler on the host, into its pinned buffer
            _abi.check(_abi.library().lfm25_stack_executor_read_logits(
                state.executor._handle, ctypes.cast(state.logits.data_ptr(), ctypes.POINTER(ctypes.c_float)),
                state.logits.shape[0]))
    return {"logits": state.logits, "recurrent": state.recurrent, "histories": state.histories, "caches": state.caches}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def exact(case, seed):
    """`run`'s logits and recurrent state in float64, from the equations of the designs."""
    with torch.no_grad():
        state = prepare(case, seed)
        torch.cuda.synchronize()
        step = _ExactStep(state)
        logits = (step.lfm2 if case["family"] == "lfm2" else step.stack)(int(seed))
        return {"logits": logits, "recurrent": step.recurrent, "histories": step.histories,
                "caches": [None] * len(state.caches)}


def _f64(tensor) -> torch.Tensor:
    return tensor.to("cuda", torch.float64)


def _rms(x, eps: float):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, positions, frequencies):
    """x [T, H, D] with entry i paired with i + half, on the first 2 * half entries."""
    half = len(frequencies)
    angle = positions.double()[:, None] * frequencies[None, :]
    cosine, sine = angle.cos()[:, None], angle.sin()[:, None]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * cosine - v * sine, v * cosine + u * sine, x[..., 2 * half:]], -1)


def _attend(query, keys, values, positions, scale: float, limit: int):
    """query [T, H, D], keys [N, G, D], values [N, G, E]; position p sees the keys up to p of its `limit`-token piece."""
    group = query.shape[1] // keys.shape[1]
    out = torch.empty(*query.shape[:2], values.shape[2], dtype=torch.float64, device="cuda")
    at = torch.arange(len(keys), device="cuda")
    for first in range(0, len(query), 512):
        rows = slice(first, first + 512)
        p = positions[rows, None]
        hidden = at[None, :] > p
        if limit:
            hidden |= at[None, :] // limit != p // limit
        for head in range(query.shape[1]):
            scores = (query[rows, head] @ keys[:, head // group].T) * scale
            out[rows, head] = torch.softmax(scores.masked_fill(hidden, -math.inf), -1) @ values[:, head // group]
    return out


class _ExactStep:
    def __init__(self, state):
        layout = state.layout
        self.state, self.layout = state, layout
        self.offsets = layout.segment_offsets.astype(np.int64)
        self.slots = torch.from_numpy(layout.segment_slots.astype(np.int64)).cuda()
        self.positions = torch.from_numpy(layout.positions.astype(np.int64)).cuda()
        self.tokens = torch.from_numpy(state.ids.astype(np.int64)).cuda()
        self.last = torch.from_numpy(layout.output_rows.astype(np.int64)).cuda()
        self.recurrent, self.histories = [], []
        self.start_recurrent = [_f64(tensor) for tensor in state.recurrent]
        self.start_histories = [_f64(tensor) for tensor in state.histories]

    def cached(self, cache, segment: int):
        """The rows [prefix, ...] that `segment`'s sequence has in a cache [pages, (heads,) 16, entries], f64."""
        prefix, slot = int(self.layout.prefixes[segment]), int(self.layout.segment_slots[segment])
        pages = torch.from_numpy(self.layout.block_tables[slot, :-(-prefix // PAGE)].astype(np.int64)).cuda()
        rows = _f64(cache[pages])
        rows = rows.transpose(1, 2) if rows.dim() == 4 else rows
        return rows.reshape(-1, *rows.shape[2:])[:prefix]

    def segments(self):
        return [(index, slice(int(self.offsets[index]), int(self.offsets[index + 1]))) for index in range(len(self.slots))]

    def convolve(self, x, taps, start):
        """Causal convolution per channel, taps [channels, J], behind the inputs `start` [slots, J - 1, channels]."""
        out, left = torch.empty_like(x), start.clone()
        count = taps.shape[1]
        for index, rows in self.segments():
            padded = torch.cat([start[self.slots[index]], x[rows]])
            length = rows.stop - rows.start
            out[rows] = sum(taps[:, j] * padded[j:j + length] for j in range(count))
            left[self.slots[index]] = padded[len(padded) - (count - 1):]
        return out, left

    def recur(self, step, inputs, start):
        """step(state [n, ..], inputs of n tokens) -> (state, output) over all sequences side by side."""
        matrices, out = start[self.slots].clone(), None
        lengths = np.diff(self.offsets)
        offsets = torch.from_numpy(self.offsets[:-1]).cuda()
        for t in range(int(lengths.max())):
            if t == 0 or (lengths == t).any():
                live = torch.from_numpy(np.nonzero(lengths > t)[0]).cuda()
            rows = offsets[live] + t
            matrices[live], produced = step(matrices[live], [value[rows] for value in inputs])
            if out is None:
                out = torch.empty(len(self.positions), *produced.shape[1:], dtype=torch.float64, device="cuda")
            out[rows] = produced
        final = start.clone()
        final[self.slots] = matrices
        return out, final

    # ---------------------------------------------------------------------------------------- LFM2

    def lfm2(self, seed: int):
        model, case = self.state.model, self.state.case
        fp8 = case["fp8"] and len(self.positions) <= FP8_MAXIMUM_TOKENS
        eps = lfm_model.NORM_EPS

        def linear(x, site):
            if not (fp8 and site.codes is not None):
                return x @ _f64(site.weight).T
            scaled = (x * (448.0 / site.activation_amax)).clamp(-448.0, 448.0)
            codes = _f64(scaled.float().to(torch.float8_e4m3fn).float())
            weight = _f64(site.codes.view(torch.float8_e4m3fn).float())
            return codes @ weight.T * (site.activation_amax / 448.0 * site.weight_amax / 448.0)

        x = _f64(model.embedding[self.tokens])
        caches = iter(self.state.caches)
        starts = iter(self.start_recurrent)
        frequencies = _f64(model.inv_freq)
        for layer in model.layers:
            sites, tensors = layer.linears, layer.tensors
            h = _rms(x, eps) * _f64(tensors["operator_norm"])
            if layer.is_attention:
                heads = [linear(h, sites[name]).reshape(len(h), -1, 64) for name in ("query", "key", "value")]
                query, key = (_rotate(_rms(part, eps) * _f64(tensors[name]), self.positions, frequencies)
                              for part, name in zip(heads, ("query_norm", "key_norm")))
                mixed = self.attention(query, key, heads[2], next(caches), next(caches), 0.125, 0)
            else:
                b, c, value = linear(h, sites["conv_input"]).split(2048, 1)
                convolved, left = self.convolve(b * value, _f64(tensors["conv_kernel"]), next(starts).transpose(1, 2))
                self.recurrent.append(left.transpose(1, 2).contiguous())
                mixed = c * convolved
            x = x + linear(mixed, sites["output" if layer.is_attention else "conv_output"])
            gate, up = linear(_rms(x, eps) * _f64(tensors["ffn_norm"]), sites["gate_up"]).split(8192, 1)
            x = x + linear(torch.nn.functional.silu(gate) * up, sites["down"])
        return linear(_rms(x[self.last], eps) * _f64(model.final_norm), model.lm_head)

    def attention(self, query, key, value, key_cache, value_cache, scale, limit):
        out = torch.empty(len(query), query.shape[1], value.shape[2], dtype=torch.float64, device="cuda")
        for index, rows in self.segments():
            keys = torch.cat([self.cached(key_cache, index), key[rows]])
            values = torch.cat([self.cached(value_cache, index), value[rows]])
            out[rows] = _attend(query[rows], keys, values, self.positions[rows], scale, limit)
        return out.reshape(len(query), -1)

    # ---------------------------------------------------------------------------------------- layer stacks

    def stack(self, seed: int):
        case, config = self.state.case, _config(self.state.case)
        source = _source(case, seed)

        def get(name, *shape):
            return _f64(source(name, shape))

        parallel = case["family"] == "fegidra"
        width, vocab = config["width"], config["vocab"]
        x = get("embed", vocab, width)[self.tokens]
        self.caches = iter(zip(self.state.caches[::2], self.state.caches[1::2]))
        self.starts, self.start_inputs = iter(self.start_recurrent), iter(self.start_histories)
        eps = config["norm"]["eps"]
        for index, layer in enumerate(config["layers"]):
            x = (self.parallel_layer if parallel else self.sandwich_layer)(x, f"l{index}.", layer, get, width, eps)
        final = _rms(x[self.last], eps) * (get("final.norm", width) + (0.0 if parallel else 1.0))
        logits = final @ get("head", vocab, width).T
        cap = config.get("logit_softcap")
        return cap * torch.tanh(logits / cap) if cap else logits

    def parallel_layer(self, x, prefix, layer, get, width, eps):
        ff, mixer = layer["mlp"]["ff"], layer["mixer"]
        h = _rms(x, eps) * get(prefix + "norm1", width)
        convolved, left = self.convolve(h, get(prefix + "canon1", width, TAPS), next(self.start_inputs))
        self.histories.append(left)
        h = h + convolved

        def project(name, rows):
            return h @ get(prefix + "mix." + name, rows, width).T

        heads, dim = mixer["heads"], mixer["dim"]
        size = heads * dim
        if layer["type"] == "attention":
            groups, frequencies = mixer["kv_heads"], self.frequencies(mixer)
            parts = []
            for name, rows in (("q", size), ("k", groups * dim), ("v", groups * dim)):
                part = project(name, rows) + get(prefix + f"mix.{name}.b", rows)
                if name != "v":
                    part = _rms(part, eps) * get(prefix + f"mix.{name}.norm", rows)
                part = part.reshape(len(h), -1, dim)
                parts.append(part if name == "v" else _rotate(part, self.positions, frequencies))
            mixed = self.attention(*parts, *next(self.caches), mixer["scale"], mixer["mask"]["size"])
        else:
            r, k, v = (project(name, size).reshape(-1, heads, dim) for name in "rkv")
            removal = torch.sigmoid(project("a", size) + get(prefix + "mix.a.b", size)).reshape(-1, heads, dim)
            low = torch.tanh(project("w1", DECAY_RANK))
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(
                low @ get(prefix + "mix.w2", size, DECAY_RANK).T + get(prefix + "mix.w0", size))).reshape(-1, heads, dim)
            unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)

            def step(matrix, inputs):      # matrix [n, heads, value, key]
                r, k, v, decay, strength, unit = inputs
                recalled = (matrix @ unit[..., None])
                matrix = matrix * decay[..., None, :] - recalled * strength[..., None, :] + v[..., None] * k[..., None, :]
                return matrix, (matrix @ r[..., None])[..., 0]

            produced, left = self.recur(step, [r, k, v, decay, removal * unit, unit], next(self.starts))
            self.recurrent.append(left)
            mixed = _rms(produced, eps).reshape(len(h), size) * get(prefix + "mix.norm", size) * \
                torch.sigmoid(project("g", size))
        update = mixed @ get(prefix + "mix.o", width, size).T
        up = (_rms(x, eps) * get(prefix + "norm2", width)) @ get(prefix + "mlp.up", ff, width).T
        a, b, c, e = get(prefix + "mlp.act", 4)
        activated = a * _rms(up, eps) + b * _rms(up ** 2, eps) + c * _rms(up ** 3, eps) + e
        return x + update + activated @ get(prefix + "mlp.down", width, ff).T

    @staticmethod
    def frequencies(mixer):
        dims = mixer["rot"]["dims"]
        return mixer["rot"]["base"] ** (-2.0 * torch.arange(dims // 2, device="cuda", dtype=torch.float64) / dims)

    def sandwich_layer(self, x, prefix, layer, get, width, eps):
        ff, mixer = layer["mlp"]["ff"], layer["mixer"]
        h = _rms(x, eps) * (1.0 + get(prefix + "norm1", width))

        def weight(name, *shape):
            return get(prefix + "mix." + name, *shape)

        mixed = (self.latent if layer["type"] == "latent_attention" else self.state_space)(h, mixer, weight, width, eps)
        x = x + _rms(mixed, eps) * (1.0 + get(prefix + "norm1b", width))
        n = _rms(x, eps) * (1.0 + get(prefix + "norm2", width))
        hidden = torch.relu(n @ get(prefix + "mlp.up", ff, width).T) ** 2
        return x + _rms(hidden @ get(prefix + "mlp.down", width, ff).T, eps) * (1.0 + get(prefix + "norm2b", width))

    def latent(self, h, mixer, weight, width, eps):
        heads, dim, rot, vdim = mixer["heads"], mixer["dim"], mixer["rot_dim"], mixer["vdim"]
        rank, q_rank = mixer["kv_rank"], mixer["q_rank"]
        frequencies = self.frequencies(mixer)
        compressed = _rms(h @ weight("dq", q_rank, width).T, eps) * weight("dq.norm", q_rank)
        query = (compressed @ weight("uq", heads * (dim + rot), q_rank).T).reshape(len(h), heads, dim + rot)
        query = torch.cat([query[..., :dim], _rotate(query[..., dim:], self.positions, frequencies)], -1)
        both = h @ weight("dkv", rank + rot, width).T
        latent = _rms(both[:, :rank], eps) * weight("dkv.norm", rank)
        turned = _rotate(both[:, None, rank:], self.positions, frequencies)[:, 0]
        up_key, up_value = weight("uk", heads * dim, rank), weight("uv", heads * vdim, rank)
        key_cache, latent_cache = next(self.caches)
        out = torch.empty(len(h), heads, vdim, dtype=torch.float64, device="cuda")
        for index, rows in self.segments():
            latents = torch.cat([self.cached(latent_cache, index), latent[rows]])
            shared = torch.cat([self.cached(key_cache, index), turned[rows]])[:, None].expand(-1, heads, -1)
            keys = torch.cat([(latents @ up_key.T).reshape(-1, heads, dim), shared], -1)
            values = (latents @ up_value.T).reshape(-1, heads, vdim)
            out[rows] = _attend(query[rows], keys, values, self.positions[rows], mixer["scale"], 0)
        gated = out.reshape(len(h), -1) * torch.sigmoid(h @ weight("g", heads * vdim, width).T)
        return gated @ weight("o", width, heads * vdim).T

    def state_space(self, h, mixer, weight, width, eps):
        heads, vdim, size, groups = mixer["heads"], mixer["vdim"], mixer["state"], mixer["groups"]
        inner = heads * vdim
        channels = inner + 2 * groups * size
        z, raw, steps = (h @ weight("in", inner + channels + heads, width).T).split([inner, channels, heads], 1)
        convolved, left = self.convolve(raw, weight("conv", channels, TAPS), next(self.start_inputs))
        self.histories.append(left)
        value, b, c = torch.nn.functional.silu(convolved + weight("conv.b", channels)).split(
            [inner, groups * size, groups * size], 1)
        value = value.reshape(-1, heads, vdim)
        b, c = (part.reshape(-1, groups, size).repeat_interleave(heads // groups, 1) for part in (b, c))
        steps = torch.nn.functional.softplus(steps + weight("dt_bias", heads), threshold=700.0)
        decay = torch.exp(-torch.exp(weight("A_log", heads)) * steps)

        def step(matrix, inputs):          # matrix [n, heads, state, value]
            value, b, c, decay, size = inputs
            matrix = matrix * decay[..., None, None] + (b * size[..., None])[..., None] * value[..., None, :]
            return matrix, (matrix * c[..., None]).sum(-2)

        produced, left = self.recur(step, [value, b, c, decay, steps], next(self.starts))
        self.recurrent.append(left)
        y = (produced + weight("D", heads)[None, :, None] * value).reshape(len(h), inner) * torch.nn.functional.silu(z)
        normed = _rms(y.reshape(len(h), mixer["norm_groups"], -1), eps).reshape(len(h), inner) * weight("norm", inner)
        return normed @ weight("o", width, inner).T
