"""Workloads that measure the engine through its public entry points (pluto_b200.layers).

A case is a dict of plain values whose "kind" names one of the uses below; `prepare` makes what a
program holds before the call, `run` is one pass of the call, `work` the bytes and operations the
pass cannot do without, `tolerance` how far another correct implementation may be off.

    token_attention   generation: one decoder attention layer over a key/value cache, token by token
    token_delta       generation: one gated delta-net layer, token by token
    decode            serving: one new token for every sequence of a batch against long caches
    prefill           serving: the attention core over a whole prompt
    delta_prefill     serving: the delta-net recurrence over a whole prompt
    attention         training: causal multi-head attention over packed Q, K, V, forward and backward
    qwen_sequence     fine-tuning: the grouped-query attention layer, forward and backward
    delta_sequence    fine-tuning: the delta-net layer, forward and backward
    imported          generation: an up and a down projection with frozen checkpoint weights
    dense             training: the dense projection (fp32 master weights), forward and backward
    block_linear      fine-tuning: the projection with resident bf16 weights, forward and backward
"""
import torch

from pluto_b200.layers import (AttentionLayer, BlockLinearLayer, BlockParameter, DataType, DeltaNetLayer,
                               DeltaNetParameters, DenseLayer, FullAttentionParameters, FullyConnectedLayer,
                               KeyValueCache, MatrixStorage, QwenAttentionLayer, SequenceDeltaNetLayer,
                               gdn_prefill, gqa_decode, gqa_prefill)

# Head shapes in use: (query heads, key/value heads, head width).  40/8/128 is the prefill and
# decode configuration the engine is benchmarked on (5/1/128: one GPU's share of it when the heads
# are split eight ways), 24/4/256 the default of FullAttentionParameters, 12/12/64 GPT-2 small.
GQA_SHAPES = ((40, 8, 128), (24, 4, 256), (12, 12, 64), (5, 1, 128))
# Delta-net (key heads, value heads), widths 128: the default of DeltaNetParameters and the
# benchmarked configuration.
DELTA_HEADS = ((16, 48), (16, 16))
ROTARY = {256: 64, 128: 128, 64: 64}
PAGE = 64


def listed():
    return [
        # the first 24 tokens of a reply, one layer: latency and launches are all there is
        dict(name="token attention 24/4/256", kind="token_attention", tokens=24, q_heads=24, kv_heads=4, dim=256),
        dict(name="token delta-net 16/48", kind="token_delta", tokens=24, key_heads=16, value_heads=48),
        # a few users with medium contexts in a paged cache, output gate on
        dict(name="decode b4 24/4/256 gate", kind="decode", batch=4, longest=3000, q_heads=24, kv_heads=4, dim=256,
             paged=True, gate=True),
        # a full serving batch with long contexts: the whole memory system
        dict(name="decode b64 40/8/128", kind="decode", batch=64, longest=32768, q_heads=40, kv_heads=8, dim=128,
             paged=False, gate=False),
        # a long prompt
        dict(name="prefill 8192 40/8/128", kind="prefill", batch=1, tokens=8192, q_heads=40, kv_heads=8, dim=128,
             gate=False),
        dict(name="delta prefill 2x16384", kind="delta_prefill", batch=2, tokens=16384, key_heads=16, value_heads=16),
        # GPT-2 small training step, and the small fp32 model the CPU layer also runs
        dict(name="attention bf16 8x1024 12x64", kind="attention", batch=8, tokens=1024, heads=12, dim=64, bf16=True),
        dict(name="attention fp32 16x256 6x64", kind="attention", batch=16, tokens=256, heads=6, dim=64, bf16=False),
        # fine-tuning samples of ragged length through the two layer kinds of a hybrid decoder
        dict(name="qwen sequence 1000", kind="qwen_sequence", tokens=1000, q_heads=24, kv_heads=4, dim=256),
        dict(name="delta sequence 1000", kind="delta_sequence", tokens=1000, key_heads=16, value_heads=48),
        # one token through two FP8 checkpoint matrices
        dict(name="imported fp8 5120-10240", kind="imported", tokens=1, width=5120, hidden=10240, fp8=True),
        # the QKV projection of a GPT-2 small training step
        dict(name="dense 8192x768x2304", kind="dense", rows=8192, width=768, out=2304, bf16=True),
    ]


def _log(rng, low, high):
    """An integer whose logarithm is uniform, so odd and ragged sizes come as often as round ones."""
    return max(low, min(high, round(low * (high / low) ** rng.random())))


def draw(rng):
    kind = rng.choice(("token_attention", "token_delta", "decode", "decode", "prefill", "prefill", "delta_prefill",
                       "attention", "attention", "qwen_sequence", "delta_sequence", "imported", "dense",
                       "block_linear"))
    hq, hkv, dim = rng.choice(GQA_SHAPES)
    hk, hv = rng.choice(DELTA_HEADS)
    if kind == "token_attention":
        return dict(kind=kind, tokens=_log(rng, 8, 56), q_heads=hq, kv_heads=hkv, dim=dim)
    if kind == "token_delta":
        return dict(kind=kind, tokens=_log(rng, 8, 56), key_heads=hk, value_heads=hv)
    if kind == "decode":
        batch = _log(rng, 1, 64)
        longest = _log(rng, 64, min(32768, 64 * 8192 // batch))
        return dict(kind=kind, batch=batch, longest=longest, q_heads=hq, kv_heads=hkv, dim=dim,
                    paged=rng.random() < 0.5, gate=rng.random() < 0.5)
    if kind == "prefill":
        batch = rng.choice((1, 1, 2, 3))
        return dict(kind=kind, batch=batch, tokens=_log(rng, 64, 4096), q_heads=hq, kv_heads=hkv, dim=dim,
                    gate=rng.random() < 0.5)
    if kind == "delta_prefill":
        return dict(kind=kind, batch=rng.choice((1, 2)), tokens=_log(rng, 64, 8192), key_heads=hk, value_heads=hv)
    if kind == "attention":
        bf16 = rng.random() < 0.5
        heads, width = rng.choice(((12, 64), (6, 64), (6, 128)))
        tokens = _log(rng, 64, 2048 if bf16 else 512)
        return dict(kind=kind, batch=_log(rng, 1, max(1, 8192 // tokens)), tokens=tokens, heads=heads, dim=width,
                    bf16=bf16)
    if kind == "qwen_sequence":
        return dict(kind=kind, tokens=_log(rng, 64, 2048), q_heads=hq, kv_heads=hkv, dim=dim)
    if kind == "delta_sequence":
        return dict(kind=kind, tokens=_log(rng, 64, 2048), key_heads=hk, value_heads=hv)
    if kind == "imported":
        return dict(kind=kind, tokens=rng.choice((1, 1, 2, 4, 8)), width=128 * rng.randint(6, 40),
                    hidden=128 * rng.randint(16, 80), fp8=rng.random() < 0.5)
    return dict(kind=kind, rows=_log(rng, 64, 8192), width=8 * rng.randint(48, 320), out=8 * rng.randint(48, 640),
                bf16=kind == "block_linear" or rng.random() < 0.5)


def _lengths(case):
    """Cached lengths of a decode batch, spread evenly over [longest / 8, longest]."""
    b, longest = case["batch"], case["longest"]
    low = max(1, longest // 8)
    return [longest - (longest - low) * i // max(1, b - 1) for i in range(b)]


def _causal_pairs(tokens):
    return tokens * (tokens + 1) // 2


# ------------------------------------------------------------------------------------------------
# prepare
# ------------------------------------------------------------------------------------------------
class _Source:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.empty(shape, device="cuda", dtype=dtype).normal_(0.0, std, generator=self.gen)

    def f32(self, *shape, std=1.0):
        return self.normal(*shape, std=std, dtype=torch.float32)

    def unit(self, *shape):
        return torch.nn.functional.normalize(self.f32(*shape), dim=-1).bfloat16()

    def permutation(self, n):
        return torch.randperm(n, device="cuda", generator=self.gen)


def _attention_parameters(case):
    return FullAttentionParameters(query_heads=case["q_heads"], key_value_heads=case["kv_heads"],
                                   head_dim=case["dim"], rotary_dim=ROTARY[case["dim"]], capacity=4096)


def _delta_parameters(case):
    return DeltaNetParameters(key_heads=case["key_heads"], value_heads=case["value_heads"])


def _delta_weights(p, src):
    channels = 2 * p.key_heads * p.key_head_dim + p.value_heads * p.value_head_dim
    return channels, [src.f32(channels, p.conv_kernel_dim, std=0.5), src.f32(p.value_heads, std=0.5) - 1.0,
                      src.f32(p.value_heads, std=0.5), 1.0 + src.f32(p.value_head_dim, std=0.1)]


def _prepare_token_attention(case, src):
    p = _attention_parameters(case)
    cache = KeyValueCache.Create(p.capacity, p.key_value_heads, p.head_dim)
    layer = QwenAttentionLayer.Create(p, src.f32(p.head_dim, std=0.1), src.f32(p.head_dim, std=0.1), 1, cache)
    kv = (1, p.key_value_heads * p.head_dim)
    tokens = [[src.normal(1, 2 * p.query_heads * p.head_dim), src.normal(*kv), src.normal(*kv)]
              for _ in range(case["tokens"])]
    return dict(layer=layer, cache=cache, tokens=tokens)


def _prepare_token_delta(case, src):
    p = _delta_parameters(case)
    channels, weights = _delta_weights(p, src)
    tokens = [[src.normal(1, channels), src.normal(1, p.value_heads * p.value_head_dim),
               src.normal(1, p.value_heads), src.normal(1, p.value_heads)] for _ in range(case["tokens"])]
    return dict(layer=DeltaNetLayer.Create(p, *weights), tokens=tokens)


def _prepare_decode(case, src):
    batch, longest, hq, hkv, dim = (case[k] for k in ("batch", "longest", "q_heads", "kv_heads", "dim"))
    blocks = (longest + PAGE - 1) // PAGE
    capacity = blocks * PAGE
    pool = (batch * blocks, PAGE, hkv, dim) if case["paged"] else (batch, capacity, hkv, dim)
    table = src.permutation(batch * blocks).to(torch.int32).view(batch, blocks) if case["paged"] else None
    lens = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")[src.permutation(batch)]
    return dict(q=src.normal(batch, hq, dim, std=0.5), k=src.normal(*pool, std=0.5), v=src.normal(*pool, std=0.5),
                lens=lens, longest=longest, table=table, gate=src.normal(batch, hq, dim) if case["gate"] else None)


def _prepare_prefill(case, src):
    batch, tokens, hq, hkv, dim = (case[k] for k in ("batch", "tokens", "q_heads", "kv_heads", "dim"))
    return dict(q=src.normal(batch, tokens, hq, dim, std=0.5), k=src.normal(batch, tokens, hkv, dim, std=0.5),
                v=src.normal(batch, tokens, hkv, dim, std=0.5),
                gate=src.normal(batch, tokens, hq, dim) if case["gate"] else None)


def _prepare_delta_prefill(case, src):
    batch, tokens, hk, hv = (case[k] for k in ("batch", "tokens", "key_heads", "value_heads"))
    return dict(q=src.unit(batch, tokens, hk, 128), k=src.unit(batch, tokens, hk, 128),
                v=src.normal(batch, tokens, hv, 128), g=torch.sigmoid(src.f32(batch, tokens, hv) * 2 + 2),
                beta=torch.sigmoid(src.f32(batch, tokens, hv)),
                state=torch.zeros(batch, hv, 128, 128, device="cuda"))


def _prepare_attention(case, src):
    rows, width = case["batch"] * case["tokens"], case["heads"] * case["dim"]
    kind = DataType.BF16 if case["bf16"] else DataType.FP16   # the FP16 policy stores fp32 activations
    return dict(layer=AttentionLayer.Create(case["tokens"], case["heads"], width, kind),
                inputs=[src.normal(rows, 3 * width, dtype=torch.bfloat16 if case["bf16"] else torch.float32)],
                gradients=[src.f32(rows, width)], parameters=[])


def _prepare_qwen_sequence(case, src):
    p, t = _attention_parameters(case), case["tokens"]
    norms = [BlockParameter.Create(src.f32(p.head_dim, std=0.1)) for _ in range(2)]
    for n in norms:
        n.Activate()
    kv = (t, p.key_value_heads * p.head_dim)
    return dict(layer=QwenAttentionLayer.Create(p, *norms, t), parameters=norms,
                inputs=[src.normal(t, 2 * p.query_heads * p.head_dim), src.normal(*kv), src.normal(*kv)],
                gradients=[src.f32(t, p.query_heads * p.head_dim)])


def _prepare_delta_sequence(case, src):
    p, t = _delta_parameters(case), case["tokens"]
    channels, weights = _delta_weights(p, src)
    parameters = [BlockParameter.Create(w) for w in weights]
    for w in parameters:
        w.Activate()
    width = p.value_heads * p.value_head_dim
    return dict(layer=SequenceDeltaNetLayer.Create(p, *parameters, t), parameters=parameters,
                inputs=[src.normal(t, channels), src.normal(t, width), src.normal(t, p.value_heads),
                        src.normal(t, p.value_heads)],
                gradients=[src.f32(t, width)])


def _prepare_imported(case, src):
    layers = []
    for cols, rows in ((case["width"], case["hidden"]), (case["hidden"], case["width"])):
        if case["fp8"]:
            weight = src.normal(rows, cols).to(torch.float8_e4m3fn).view(torch.uint8)
            scales = (1.0 + 0.1 * torch.rand(rows // 128, cols // 128, device="cuda", generator=src.gen)) * cols ** -0.5
            layers.append(FullyConnectedLayer.Create(weight, MatrixStorage.kFp8E4M3, cols, rows, scales))
        else:
            weight = src.normal(rows, cols, std=cols ** -0.5)
            layers.append(FullyConnectedLayer.Create(weight, MatrixStorage.kBFloat16, cols, rows))
    return dict(layers=layers, x=src.normal(case["tokens"], case["width"]))


def _prepare_dense(case, src):
    layer = DenseLayer.Create(case["width"], case["out"], DataType.BF16 if case["bf16"] else DataType.FP16)
    layer.weights()[0].normal_(0.0, 0.02, generator=src.gen)
    layer.weights()[1].normal_(0.0, 0.02, generator=src.gen)
    return dict(layer=layer, parameters=[], gradients=[src.f32(case["rows"], case["out"])],
                inputs=[src.normal(case["rows"], case["width"],
                                   dtype=torch.bfloat16 if case["bf16"] else torch.float32)])


def _prepare_block_linear(case, src):
    weight = BlockParameter.Create(src.normal(case["out"], case["width"], std=0.02))
    weight.Activate()
    return dict(layer=BlockLinearLayer.Create(weight, case["width"], case["out"], case["rows"]), parameters=[weight],
                inputs=[src.normal(case["rows"], case["width"])], gradients=[src.f32(case["rows"], case["out"])])


_PREPARE = dict(token_attention=_prepare_token_attention, token_delta=_prepare_token_delta, decode=_prepare_decode,
                prefill=_prepare_prefill, delta_prefill=_prepare_delta_prefill, attention=_prepare_attention,
                qwen_sequence=_prepare_qwen_sequence, delta_sequence=_prepare_delta_sequence,
                imported=_prepare_imported, dense=_prepare_dense, block_linear=_prepare_block_linear)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, _Source(seed)), kind=case["kind"])


# ------------------------------------------------------------------------------------------------
# run
# ------------------------------------------------------------------------------------------------
def _generate(state):
    """A fresh sequence, token by token."""
    (state["cache"] if "cache" in state else state["layer"]).Reset()
    outputs = [state["layer"].fwd(token).outputs[0] for token in state["tokens"]]
    if "cache" in state:
        return outputs, state["cache"].keys(), state["cache"].values()
    return outputs, state["layer"].cache_.recurrent_state_, state["layer"].cache_.convolution_state_


def _decode(state):
    return gqa_decode(state["q"], state["k"], state["v"], state["lens"], state["longest"],
                      block_table=state["table"], gate=state["gate"])


def _prefill(state):
    return gqa_prefill(state["q"], state["k"], state["v"], gate=state["gate"])["out"]


def _delta_prefill(state):
    state["state"].zero_()
    out = gdn_prefill(state["q"], state["k"], state["v"], state["g"], state["beta"], state["state"])
    return out, state["state"]


def _train(state):
    """One layer's part of a training step: cleared parameter gradients, forward, backward."""
    layer = state["layer"]
    for parameter in state["parameters"]:
        parameter.gradient().zero_()
    result = layer.fwd(state["inputs"])
    return result.outputs, layer.bwd(state["gradients"], result.state), layer.gradients()


def _imported(state):
    up, down = state["layers"]
    hidden = up.fwd([state["x"]]).outputs
    return hidden, down.fwd(hidden).outputs


_RUN = dict(token_attention=_generate, token_delta=_generate, decode=_decode, prefill=_prefill,
            delta_prefill=_delta_prefill, attention=_train, qwen_sequence=_train, delta_sequence=_train,
            imported=_imported, dense=_train, block_linear=_train)


def run(state):
    return _RUN[state["kind"]](state)


# ------------------------------------------------------------------------------------------------
# work and tolerance
# ------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "token_attention":
        n, hq, hkv, d = (case[k] for k in ("tokens", "q_heads", "kv_heads", "dim"))
        # every call: query, gate, K and V in, the output out, K and V appended; the cache so far
        return {"bytes": n * (2 * d * (3 * hq + 4 * hkv)) + 4 * d * hkv * _causal_pairs(n),
                "flops": 4 * d * hq * _causal_pairs(n)}
    if kind == "token_delta":
        n, hk, hv = (case[k] for k in ("tokens", "key_heads", "value_heads"))
        channels = 128 * (2 * hk + hv)
        # every call: the fp32 state and the convolution window in and out, weights, token, output
        return {"bytes": n * (8 * hv * 128 * 128 + 48 * channels + 2 * channels + 512 * hv),
                "flops": n * (6 * hv * 128 * 128 + 8 * channels)}
    if kind == "decode":
        total, hq, hkv, d = sum(_lengths(case)), case["q_heads"], case["kv_heads"], case["dim"]
        return {"bytes": 4 * d * hkv * total + 2 * d * hq * case["batch"] * (3 if case["gate"] else 2),
                "flops": 4 * d * hq * total}
    if kind == "prefill":
        b, t, hq, hkv, d = (case[k] for k in ("batch", "tokens", "q_heads", "kv_heads", "dim"))
        return {"bytes": 2 * b * t * d * (hq * (3 if case["gate"] else 2) + 2 * hkv),
                "flops": 4 * d * _causal_pairs(t) * b * hq}
    if kind == "delta_prefill":
        b, t, hk, hv = (case[k] for k in ("batch", "tokens", "key_heads", "value_heads"))
        return {"bytes": b * t * (256 * (2 * hk + 2 * hv) + 8 * hv) + 8 * b * hv * 128 * 128,
                "flops": 6 * b * t * hv * 128 * 128}
    if kind == "attention":
        b, t, h, d = (case[k] for k in ("batch", "tokens", "heads", "dim"))
        element = 2 if case["bf16"] else 4
        # packed input and output in the activation type; upstream and packed gradient fp32
        return {"bytes": b * t * h * d * (4 * element + 16), "flops": 14 * d * _causal_pairs(t) * b * h}
    if kind == "qwen_sequence":
        t, hq, hkv, d = (case[k] for k in ("tokens", "q_heads", "kv_heads", "dim"))
        return {"bytes": t * d * (hq * (2 * 3 + 4 + 8) + hkv * (4 + 8)), "flops": 14 * d * _causal_pairs(t) * hq}
    if kind == "delta_sequence":
        t, hk, hv = (case[k] for k in ("tokens", "key_heads", "value_heads"))
        channels, width = 128 * (2 * hk + hv), 128 * hv
        return {"bytes": t * (channels * (2 + 4) + width * (2 + 2 + 4 + 4) + hv * 12),
                "flops": t * (18 * hv * 128 * 128 + 24 * channels)}
    if kind == "imported":
        n, w, h = case["tokens"], case["width"], case["hidden"]
        matrix = w * h if case["fp8"] else 2 * w * h
        return {"bytes": 2 * matrix + 2 * n * (2 * w + 2 * h), "flops": 4 * n * w * h}
    rows, w, o = case["rows"], case["width"], case["out"]
    weight = 2 + 4 if kind == "block_linear" else 8   # the matrix in, its fp32 gradient out
    element = 2 if case["bf16"] else 4
    return {"bytes": w * o * weight + rows * (w * (element + 4) + o * (element + 4)), "flops": 6 * rows * w * o}


def tolerance(case):
    # fp32 activations and arithmetic: sums of a few hundred fp32 products
    if case["kind"] == "attention" and not case["bf16"]:
        return {"rel": 1e-5}
    # the dense layer's FP16 policy: fp32 activations, products of fp16 operands
    if case["kind"] == "dense" and not case["bf16"]:
        return {"rel": 2e-3}
    # bf16 activations, operands or results
    return {"rel": 1e-2}
