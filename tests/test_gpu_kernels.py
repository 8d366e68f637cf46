"""GPU: kernels and dispatch branches at the sizes where they can go wrong (edges of tiles, remainders,
the smallest and largest of a range, unaligned and strided operands), against the oracle or a
64-bit restatement of the same sum."""

from __future__ import annotations

import math

import pytest
import torch

from helpers import oracle_params, make_codec, rel_inf, store_to_layer
from oracle import tq_oracle as O

pytestmark = pytest.mark.gpu

BF16, F16, F32 = torch.bfloat16, torch.float16, torch.float32
# relative to the largest reference magnitude: the bounds of the parity tests (1e-5 for fp32 caches, 2e-3 for the
# 16-bit kernels) plus half an ulp of the output's rounding
ATTN_TOL = {F32: 1e-5, BF16: 2e-3 + 2.0 ** -9, F16: 2e-3 + 2.0 ** -12}


def vectors(shape, seed, dtype, device="cuda"):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(shape, generator=g) * torch.exp(0.5 * torch.randn(*shape[:-1], 1, generator=g))
    return x.to(dtype).to(device)


def query(shape, seed, dtype):
    """iid N(0,1), what the 2e-3 bound is stated for: with more than four heads per KV head the rotated query is one f16
    term, so a logit is off by up to 2^-12 of |q||k| / sqrt(128) and the bound only holds while that stays of order 1e-3."""
    return torch.randn((*shape, 128), generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()


def off_by_one(x):
    """The same tensor one element off its 16-byte alignment."""
    buf = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:]
    return buf.view(x.shape).copy_(x)


def attend64(store, p, q, groups, tail_k=None, tail_v=None):
    """Decode attention in fp64 over the store's dequantised tokens (not rounded to the cache dtype), then the tail."""
    layer = store_to_layer(store, p, torch.float32)
    k, v = O.dequant_keys(layer).double(), O.dequant_values(layer).double()
    if tail_k is not None:
        k, v = torch.cat((k, tail_k.cpu().double()), dim=2), torch.cat((v, tail_v.cpu().double()), dim=2)
    k, v = k.repeat_interleave(groups, dim=1), v.repeat_interleave(groups, dim=1)
    w = torch.softmax(q.cpu().double() @ k.transpose(-1, -2) / math.sqrt(128), dim=-1)
    return w @ v


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 2, 15), (3, 5, 7), (2, 3, 129), (1, 4, 4097)])
@pytest.mark.parametrize("form", ["contiguous", "transposed", "unaligned"])
def test_key_norm_mean(dtype, shape, form):
    from tq_local_b200.runtime.packed_store import key_norm_mean, key_norm_means

    x = vectors((*shape, 128), 3, dtype)
    want = float(x.double().norm(dim=-1).mean())
    if form == "transposed":
        x = x.transpose(1, 2).contiguous().transpose(1, 2)
    elif form == "unaligned":
        x = off_by_one(x)
    # fp32 sum of 128 squares and a square root per vector, then fp64: a relative error below 128 x 2^-24
    assert abs(float(key_norm_mean(x)) - want) <= 128 * 2.0 ** -24 * want
    both = key_norm_means([x, x[:, :, :1]])
    assert abs(both[0] - want) <= 128 * 2.0 ** -24 * want and both[1] > 0


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("groups", [1, 4, 5, 8])
@pytest.mark.parametrize("n_tail", [1, 63, 64, 255, 256, 257, 700])
def test_dense_tail(setup_golden, dtype, groups, n_tail):
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    store = PackedStore(codec, 2, 2, capacity=256)
    store.pack(vectors((2, 2, 70, 128), 1, dtype), vectors((2, 2, 70, 128), 2, dtype))
    q = query((2, 2 * groups, 1), 3, dtype)
    tk, tv = vectors((2, 2, n_tail, 128), 4, dtype), vectors((2, 2, n_tail, 128), 5, dtype)
    want = attend64(store, p, q, groups, tk, tv)
    got = store.decode_attn(q, tail_k=tk, tail_v=tv)
    assert rel_inf(got, want) <= ATTN_TOL[dtype]
    # the same values, a row stride that is no multiple of the row and unaligned rows: the same bits
    wide = torch.zeros(2, 2, n_tail, 136, dtype=dtype, device="cuda")
    wide[..., :128] = tk
    assert torch.equal(got, store.decode_attn(q, tail_k=wide[..., :128], tail_v=off_by_one(tv)))
    store.length = 0  # nothing packed: the tail alone
    k, v = tk.cpu().double().repeat_interleave(groups, dim=1), tv.cpu().double().repeat_interleave(groups, dim=1)
    alone = torch.softmax(q.cpu().double() @ k.transpose(-1, -2) / math.sqrt(128), dim=-1) @ v
    assert rel_inf(store.decode_attn(q, tail_k=tk, tail_v=tv), alone) <= ATTN_TOL[dtype]


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("splits", [1, 2, 8, 9, 31, 32, 33, 41, 70])
def test_split_merge(setup_golden, dtype, splits):
    """Every remainder of the merge's batches of 8 and 32 partials (one long row, so that the splits are used)."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(3, True, setup_golden), make_codec(3, True, setup_golden)
    n = 512 * (splits - 1) + 3 if splits > 1 else 77
    store = PackedStore(codec, 1, 1, capacity=n)
    store.pack(vectors((1, 1, n, 128), 1, dtype), vectors((1, 1, n, 128), 2, dtype))
    q = query((1, 5, 1), 3, dtype)
    assert rel_inf(store.decode_attn(q, splits=splits), attend64(store, p, q, 5)) <= ATTN_TOL[dtype]


@pytest.mark.parametrize("bits,qjl", [(2, False), (3, False), (4, False), (2, True), (3, True), (4, True)])
@pytest.mark.parametrize("groups", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("n", [1, 31, 33, 511, 513])
def test_fp32_attention(setup_golden, bits, qjl, groups, n):
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    store = PackedStore(codec, 2, 2, capacity=n)
    store.pack(vectors((2, 2, n, 128), 1, F32), vectors((2, 2, n, 128), 2, F32))
    q = query((2, 2 * groups, 1), 3, F32)
    want = attend64(store, p, q, groups)
    assert rel_inf(store.decode_attn(q), want) <= 1e-5
    assert rel_inf(store.decode_attn(q, splits=3), want) <= 1e-5
