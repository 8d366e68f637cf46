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

