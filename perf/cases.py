"""The work a user of this library has it do, as cases that can be timed and compared.

Five kinds, each one pass through the public entry points:

* ``attend``   one decode step of attention over a layer's packed cache, through the attention
               backend's forward function; with ``tail`` > 0 the layer keeps its newest tokens dense
               (``quantize_decode=False``)
* ``eager``    one generated token of one layer as an eager model step makes it: the cache's
               ``update`` with the new key / value, then the backend's forward function
* ``replay``   the same append + attend for ``layers`` layers with the cache length on the device,
               recorded once in a CUDA graph and replayed, as the recorded decode loop does
* ``pack``     packing the dense prompt cache of ``layers`` layers, norm guard on
* ``dequant``  reading a packed layer's keys and values back dense (``verify=True``, attention
               backends other than this library's)

Keys and values are iid N(0,1) coordinates with lognormal(0, 0.5) per-token norms; a cache that is only read
holds the codes of such vectors.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

from tq_local_b200.runtime.attention import turboquant_attention_forward
from tq_local_b200.runtime.packed_qmse_cache import PackedMSELayer, build_packed_mse_cache

D = 128
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
# the largest listed cases: tokens x KV heads x batch of one packed layer, and of one prompt pass
MOST_UNITS = 4 * 8 * 131072
MOST_PACK_UNITS = 8 * 8 * 32768
HEADS = ((32, 8), (28, 4), (8, 2), (16, 2))  # query heads, KV heads: 4, 7, 4 and 8 queries per KV head


def _case(kind, batch, ctx, q_heads=32, kv_heads=8, bits=4, qjl=True, dtype="bf16", tail=0, layers=1, padded=False):
    return dict(kind=kind, batch=batch, ctx=ctx, q_heads=q_heads, kv_heads=kv_heads, bits=bits, qjl=qjl, dtype=dtype,
                tail=tail, layers=layers, padded=padded)


def listed():
    return [
        # a chat turn's first tokens, eager: launches and host work are everything
        dict(_case("eager", 1, 77), name="eager_b1_ctx77"),
        # one user, a few thousand tokens, eight layers of a recorded decode step
        dict(_case("replay", 1, 4099, layers=8), name="replay_b1_ctx4099_x8"),
        # a small left-padded batch under 7 queries per KV head, keys without the sketch
        dict(_case("replay", 4, 8191, 28, 4, qjl=False, layers=4, padded=True), name="replay_b4_ctx8191_padded_g7"),
        # one user with a long document, fp16
        dict(_case("attend", 1, 32768, 28, 4, dtype="f16"), name="attend_b1_ctx32768_g7_f16"),
        # the benchmark's layer: batch 8 at 32k
        dict(_case("attend", 8, 32768), name="attend_b8_ctx32768"),
        # the longest contexts, 3-bit
        dict(_case("attend", 4, 131072, bits=3), name="attend_b4_ctx131072_3bit"),
        # generated tokens kept dense after a packed prompt
        dict(_case("attend", 1, 12001, tail=300), name="attend_b1_ctx12001_tail300"),
        # fp32 caches, where 1e-5 is asked for
        dict(_case("attend", 1, 4096, qjl=False, dtype="f32"), name="attend_b1_ctx4096_f32"),
        # a short prompt: two layers
        dict(_case("pack", 1, 1000, layers=2), name="pack_b1_ctx1000_x2"),
        # a ragged middle-sized prompt batch, 3-bit fp16 without the sketch
        dict(_case("pack", 3, 5003, 28, 4, bits=3, qjl=False, dtype="f16"), name="pack_b3_ctx5003_3bit_f16"),
        # one layer of a batch of long prompts
        dict(_case("pack", 8, 32768), name="pack_b8_ctx32768"),
        # the reconstruction of one long prompt's layer
        dict(_case("dequant", 1, 32768), name="dequant_b1_ctx32768"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("attend", "attend", "attend", "eager", "replay", "pack", "pack", "dequant"))
    q_heads, kv_heads = rng.choice(HEADS)
    batch = _log_int(rng, 1, 16)
    bits, qjl = rng.choice((2, 3, 4, 4, 4)), rng.random() < 0.7
    dtype = rng.choice(("bf16", "bf16", "bf16", "f16"))
    padded = batch > 1 and rng.random() < 0.3
    tail, layers = 0, 1
    if kind == "attend" and rng.random() < 0.2:  # fp32 caches: short ones (they serve as a reference)
        ctx = _log_int(rng, 16, max(16, 32768 // batch))
        return _case(kind, batch, ctx, q_heads, kv_heads, bits, qjl, "f32", padded=padded)
    if kind == "attend":
        ctx = _log_int(rng, 16, min(131072, MOST_UNITS // (batch * kv_heads)))
        if rng.random() < 0.25:
            tail, padded = _log_int(rng, 1, 1024), False
    elif kind == "eager":
        ctx = _log_int(rng, 16, min(32768, MOST_UNITS // (batch * kv_heads)))
    elif kind == "replay":
        layers = rng.choice((2, 4, 8))
        ctx = _log_int(rng, 16, min(32768, MOST_UNITS // (batch * kv_heads * layers)))
    elif kind == "pack":
        layers = rng.choice((1, 1, 2, 4))
        ctx, padded = _log_int(rng, 16, min(32768, MOST_PACK_UNITS // (batch * kv_heads * layers))), False
        dtype = rng.choice(("bf16", "bf16", "bf16", "f16", "f32"))
    else:
        ctx, padded = _log_int(rng, 16, min(32768, MOST_PACK_UNITS // (4 * batch * kv_heads))), False
    return _case(kind, batch, ctx, q_heads, kv_heads, bits, qjl, dtype, tail, layers, padded)


def _vectors(gen, batch, heads, tokens, dtype):
    out = torch.empty(batch, heads, tokens, D, dtype=dtype, device="cuda")
    for lo in range(0, tokens, 8192):  # in token chunks: the fp32 temporaries stay small
        hi = min(tokens, lo + 8192)
        x = torch.randn(batch, heads, hi - lo, D, generator=gen, device="cuda")
        x *= torch.exp(0.5 * torch.randn(batch, heads, hi - lo, 1, generator=gen, device="cuda"))
        out[:, :, lo:hi] = x
    return out


def _codes(gen, shape, boundaries, bits):
    """The code bytes of unit vectors with Gaussian coordinates: 8 codes of ``bits`` bits make ``bits`` bytes, LSB first."""
    z = torch.randn(*shape, D // 8, 8, generator=gen, device="cuda") * D ** -0.5
    idx = torch.bucketize(z, boundaries, out_int32=True)
    words = (idx << (bits * torch.arange(8, dtype=torch.int32, device="cuda"))).sum(dim=-1, dtype=torch.int32)
    return words.view(torch.uint8).view(*shape, D // 8, 4)[..., :bits].reshape(*shape, 16 * bits)


def _layer(case, gen):
    """A packed layer holding the ``ctx`` tokens of a prompt, with room for the tokens generated after them.  What it
    holds is drawn as packed bytes and not encoded here, so that it does not depend on the encoder."""
    dtype, bits = DTYPES[case["dtype"]], case["bits"]
    key_bits = bits - 1 if case["qjl"] else bits
    layer = PackedMSELayer(bits=bits, use_qjl_keys=case["qjl"], quantize_decode=case["tail"] == 0,
                           reserve_tokens=max(64, case["tail"]))
    shape = (case["batch"], case["kv_heads"])
    blank = torch.zeros(*shape, case["ctx"], D, dtype=dtype, device="cuda")
    layer.initialize_from_dense(blank, blank)
    del blank
    streams = _streams(layer)
    key_bounds = layer._key_boundaries if case["qjl"] else layer.boundaries
    for lo in range(0, case["ctx"], 8192):
        hi = min(case["ctx"], lo + 8192)
        rows = (*shape, hi - lo)
        norms = [math.sqrt(D) * torch.exp(0.5 * torch.randn(rows, generator=gen, device="cuda")) for _ in range(2)]
        parts = [_codes(gen, rows, key_bounds, key_bits), norms[0], _codes(gen, rows, layer.boundaries, bits), norms[1]]
        if case["qjl"]:
            left = {1: 0.60, 2: 0.34, 3: 0.19}[key_bits]  # what a key code of that many bits leaves of a unit vector
            parts += [torch.randint(0, 256, (*rows, 16), generator=gen, device="cuda", dtype=torch.uint8),
                      norms[0] * left * (1 + 0.05 * torch.randn(rows, generator=gen, device="cuda"))]
        for stream, part in zip(streams, parts):
            stream[:, :, lo:hi] = part
    layer._lazy_update = True  # what the attention backend sets when it takes a model over
    if case["tail"]:
        layer.update(_vectors(gen, *shape, case["tail"], dtype), _vectors(gen, *shape, case["tail"], dtype))
    mask = None
    if case["padded"]:  # left padding of up to half the prompt, the longest row unpadded
        starts = (torch.rand(case["batch"], generator=gen, device="cuda") * (case["ctx"] // 2)).long()
        starts[0] = 0
        mask = torch.arange(case["ctx"], device="cuda")[None, :] >= starts[:, None]
    layer.bind_attention_mask(mask, lock=True)
    return layer


def _streams(layer):
    """The stored bytes of a layer: key codes, norms, sign sketch, residual norms, value codes, norms."""
    k, v, s = layer.keys_packed, layer.values_packed, layer._keys_qjl
    out = [k.packed_indices, k.norms, v.packed_indices, v.norms]
    return out + ([s.packed_signs, s.residual_norms] if s is not None else [])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    batch, kv_heads, n_layers = case["batch"], case["kv_heads"], case["layers"]
    state = SimpleNamespace(case=case)
    if kind == "pack":
        state.prompt = [(_vectors(gen, batch, kv_heads, case["ctx"], dtype), _vectors(gen, batch, kv_heads, case["ctx"], dtype))
                        for _ in range(n_layers)]
        return state
    state.layers = [_layer(case, gen) for _ in range(n_layers)]
    if kind == "dequant":
        return state
    state.modules = [SimpleNamespace(_tq_cache_layer=layer, num_key_value_groups=case["q_heads"] // kv_heads)
                     for layer in state.layers]
    state.q = [torch.randn(batch, case["q_heads"], 1, D, generator=gen, device="cuda").to(dtype) for _ in range(n_layers)]
    if kind == "attend":
        return state
    state.new = [(_vectors(gen, batch, kv_heads, 1, dtype), _vectors(gen, batch, kv_heads, 1, dtype)) for _ in range(n_layers)]
    if kind == "replay":
        state.pos = torch.tensor([case["ctx"]], dtype=torch.int32, device="cuda")
        for layer in state.layers:
            layer.begin_static_decode(state.pos, 1)
        _steps(state)  # one step before recording, as the decode loop does
        torch.cuda.synchronize()
        state.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state.graph):
            state.out = _steps(state)
        state.graph.replay()
        for layer in state.layers:  # the views below show the appended token
            layer.store.length = case["ctx"] + 1
        state.stored = [_streams(layer) for layer in state.layers]
    return state


def _steps(state):
    out = []
    for module, q, (k, v) in zip(state.modules, state.q, state.new):
        k, v = module._tq_cache_layer.update(k, v)
        out.append(turboquant_attention_forward(module, q, k, v, None)[0])
    return out


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "attend":
        return turboquant_attention_forward(state.modules[0], state.q[0], None, None, None)[0]
    if kind == "eager":
        layer = state.layers[0]
        layer.end_static_decode(case["ctx"])  # back to the prompt's length: every pass generates the same token
        out = _steps(state)
        return out, _streams(layer)
    if kind == "replay":
        state.graph.replay()
        return state.out, state.stored
    if kind == "pack":
        cache = build_packed_mse_cache(state.prompt, bits=case["bits"], use_qjl_keys=case["qjl"], quantize_decode=True,
                                       norm_guard=True, reserve_tokens=64)
        return [_streams(layer) for layer in cache.layers]
    store, dtype = state.layers[0].store, DTYPES[case["dtype"]]
    return store.dequant("keys", dtype=dtype), store.dequant("values", dtype=dtype)


def work(case):
    batch, ctx, layers, bits = case["batch"], case["ctx"], case["layers"], case["bits"]
    size = 4 if case["dtype"] == "f32" else 2
    rows = batch * case["kv_heads"]
    key_bits = bits - 1 if case["qjl"] else bits
    packed = 16 * key_bits + 2 + (18 if case["qjl"] else 0) + 16 * bits + 2  # bytes of a token of a KV head
    dense = 2 * D * size
    rotation = 2 * D * D
    token_flops = rotation * (4 if case["qjl"] else 2)  # encode one key and one value
    if case["kind"] == "pack":
        units = layers * rows * ctx
        return {"bytes": units * (packed + dense), "flops": units * token_flops}
    if case["kind"] == "dequant":
        return {"bytes": rows * ctx * (packed + dense), "flops": rows * ctx * rotation * (3 if case["qjl"] else 2)}
    queries = batch * case["q_heads"]
    new = 0 if case["kind"] == "attend" else 1
    attended = ctx + new
    nbytes = rows * (attended * packed + case["tail"] * dense + new * dense) + 2 * queries * D * size
    flops = queries * (2 * D * (3 if case["qjl"] else 2) * attended + 4 * D * case["tail"]
                       + rotation * (3 if case["qjl"] else 2)) + new * rows * token_flops
    return {"bytes": layers * nbytes, "flops": layers * flops}


def tolerance(case):
    """Four times what was measured against the same path in 64 bits (attention, dequantisation), and against the
    encoder that sums in another order (packing, 131072 vectors of each mode)."""
    dtype = case["dtype"]
    if case["kind"] == "pack":
        # codes at a bin's edge: 5e-6 of the bytes; sign bits, whose residual is taken after a rounding to the cache's
        # type: 1.7e-4; norms one fp16 ulp off: 4.5e-5 over a stream (a few in a short one)
        stream = case["batch"] * case["kv_heads"] * case["ctx"]
        return {"rel": 2e-4 + 1e-3 / math.sqrt(stream), "max": 8e-3, "differ": (7e-4 if case["qjl"] else 2e-5) + 4 / (16 * stream)}
    if case["kind"] == "dequant":  # measured 3.6e-5 / 2e-2 (bf16), 1.2e-5 / 1.9e-3 (f16)
        return {"rel": 1.5e-4, "max": 8e-2} if dtype == "bf16" else {"rel": 5e-5, "max": 8e-3}
    # measured 1.8e-3 / 8e-3 (bf16), 6.5e-4 / 4e-3 (f16), 1.1e-6 / 7e-6 (f32); the appended token of the steps as in packing
    limits = {"bf16": {"rel": 7e-3, "max": 4e-2}, "f16": {"rel": 2.5e-3, "max": 2e-2}, "f32": {"rel": 5e-6, "max": 4e-5}}[dtype]
    return limits if case["kind"] == "attend" else dict(limits, differ=1e-3)
