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
@pytest.mark.parametrize("shape", [(1, 1, 8191), (1, 1, 8192), (1, 1, 8193), (2, 5, 819), (2, 5, 820), (4, 8, 5003)])
@pytest.mark.parametrize("form", ["contiguous", "unaligned"])
def test_key_norm_mean_of_few_and_many(dtype, shape, form):
    """Both sides of the size from which a lane makes eight loads, and more vectors than one round of the grid."""
    from tq_local_b200.runtime.packed_store import key_norm_mean

    x = vectors((*shape, 128), 3, dtype)
    want = float(x.double().norm(dim=-1).mean())
    x = off_by_one(x) if form == "unaligned" else x
    assert abs(float(key_norm_mean(x)) - want) <= 128 * 2.0 ** -24 * want


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


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("n_tail,masked", [(1, (0, 1)), (64, (0, 64)), (130, (0, 44)), (130, (44, 130)), (1100, (0, 275)), (1100, (300, 600)),
                                           (1100, (0, 1099))])
def test_dense_tail_with_infinite_logits(setup_golden, dtype, n_tail, masked):
    """Tail tokens whose logit is -inf weigh nothing, also where they fill a chunk or a CTA's whole share; with nothing
    else to attend the result is undefined, as that softmax is."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    store = PackedStore(codec, 1, 2, capacity=80)
    store.pack(vectors((1, 2, 70, 128), 1, dtype), vectors((1, 2, 70, 128), 2, dtype))
    q = query((1, 10, 1), 3, dtype)
    q[..., 7] = q[..., 7].abs() + 0.5
    tk, tv = vectors((1, 2, n_tail, 128), 4, dtype), vectors((1, 2, n_tail, 128), 5, dtype)
    tk[:, :, masked[0]:masked[1], 7] = -float("inf")
    assert rel_inf(store.decode_attn(q, tail_k=tk, tail_v=tv), attend64(store, p, q, 5, tk, tv)) <= ATTN_TOL[dtype]
    store.length = 0
    k, v = tk.cpu().double().repeat_interleave(5, dim=1), tv.cpu().double().repeat_interleave(5, dim=1)
    alone, got = torch.softmax(q.cpu().double() @ k.transpose(-1, -2) / math.sqrt(128), dim=-1) @ v, store.decode_attn(q, tail_k=tk, tail_v=tv)
    if masked[1] - masked[0] == n_tail:
        assert got.isnan().all() and alone.isnan().all()
    else:
        assert rel_inf(got, alone) <= ATTN_TOL[dtype]


def attend_tail64(store, p, q, groups, tk, tv, starts):
    """``attend64`` with the packed tokens before ``starts[b]`` left out."""
    layer = store_to_layer(store, p, torch.float32)
    k, v = O.dequant_keys(layer).double(), O.dequant_values(layer).double()
    k, v = torch.cat((k, tk.cpu().double()), dim=2), torch.cat((v, tv.cpu().double()), dim=2)
    k, v = k.repeat_interleave(groups, dim=1), v.repeat_interleave(groups, dim=1)
    logits = q.cpu().double() @ k.transpose(-1, -2) / math.sqrt(128)
    masked = torch.arange(logits.shape[-1])[None, None, None] < torch.tensor(starts)[:, None, None, None]
    return torch.softmax(logits.masked_fill(masked, -float("inf")), dim=-1) @ v


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("batch,heads,groups,n_tail", [
    (1, 2, 4, 85), (1, 2, 4, 86), (1, 2, 5, 1024), (1, 2, 4, 1025), (1, 2, 5, 1029), (1, 1, 1, 2500),  # one CTA, four, second chunks
    (4, 8, 1, 128), (4, 8, 1, 129), (4, 8, 4, 513),                                                     # one, two, four CTAs
    (8, 8, 1, 384), (8, 8, 4, 385), (8, 8, 1, 600),                                                     # one CTA, two
    (16, 8, 4, 5), (16, 8, 4, 6), (16, 4, 7, 300), (32, 8, 4, 23), (32, 8, 1, 24), (19, 8, 8, 33), (19, 8, 5, 34),  # a row a block
    (64, 8, 1, 95), (64, 8, 1, 96), (128, 8, 1, 256), (128, 8, 1, 257)])
def test_dense_tail_ranges(setup_golden, dtype, batch, heads, groups, n_tail):
    """Every way a tail is shared out, on both sides of each limit (on 148 SMs): clusters of one, two and four CTAs, shares of
    more than one chunk of 256, more rows than SMs in both kernels; the largest logits in the last quarter of the tail,
    so that every merge rescales."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    store = PackedStore(codec, batch, heads, capacity=40)
    store.pack(vectors((batch, heads, 33, 128), 1, dtype), vectors((batch, heads, 33, 128), 2, dtype))
    q = query((batch, heads * groups, 1), 3, dtype)
    tk, tv = vectors((batch, heads, n_tail, 128), 4, dtype), vectors((batch, heads, n_tail, 128), 5, dtype)
    tk[:, :, n_tail - (n_tail + 3) // 4:] *= 4
    want = attend64(store, p, q, groups, tk, tv)
    got = store.decode_attn(q, tail_k=tk, tail_v=tv)
    assert rel_inf(got, want) <= ATTN_TOL[dtype]
    assert torch.equal(got, store.decode_attn(q, tail_k=off_by_one(tk), tail_v=off_by_one(tv)))
    assert codec.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("copies,n_tail", [(1, 70), (1, 300), (86, 5), (86, 200)])
def test_dense_tail_of_padded_rows(setup_golden, dtype, copies, n_tail):
    """A left-padded batch with a tail, a row with nothing but its tail among it, few rows and more than there are SMs."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    starts = [0, 41, 70] * copies
    store = PackedStore(codec, len(starts), 2, capacity=72)
    store.pack(vectors((len(starts), 2, 70, 128), 1, dtype), vectors((len(starts), 2, 70, 128), 2, dtype))
    store.set_seq_start(torch.tensor(starts, dtype=torch.int32, device="cuda"))
    q = query((len(starts), 6, 1), 3, dtype)
    tk, tv = vectors((len(starts), 2, n_tail, 128), 4, dtype), vectors((len(starts), 2, n_tail, 128), 5, dtype)
    assert rel_inf(store.decode_attn(q, tail_k=tk, tail_v=tv), attend_tail64(store, p, q, 3, tk, tv, starts)) <= ATTN_TOL[dtype]


@pytest.mark.parametrize("dtype", [BF16, F32])
def test_tail_alone_after_a_step(setup_golden, dtype):
    """A tail without packed tokens, right behind a step of another layer whose last kernel starts its successor early and
    whose output is the tail's newest token: attended as it is after that step."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(4, True, setup_golden)
    first, second = PackedStore(codec, 1, 4, capacity=40), PackedStore(codec, 1, 4, capacity=8)
    first.pack(vectors((1, 4, 33, 128), 1, dtype), vectors((1, 4, 33, 128), 2, dtype))
    qs, tv = [query((1, 4, 1), 10 + i, dtype) for i in range(20)], vectors((1, 4, 5, 128), 4, dtype)
    q, tk = query((1, 4, 1), 3, dtype), vectors((1, 4, 5, 128), 5, dtype)
    got, tails = [], []
    for x in qs:
        row = torch.empty(1, 4, 1, 128, dtype=dtype, device="cuda")
        first.decode_attn(x, out=row)
        got.append(second.decode_attn(q, tail_k=row, tail_v=tv[:, :, :1]))
        tails.append(row)
        got.append(second.decode_attn(row, tail_k=tk, tail_v=tv))
    torch.cuda.synchronize()
    for i, row in enumerate(tails):
        assert torch.equal(got[2 * i], tv[:, :, :1])  # one token: its value
        again = second.decode_attn(row, tail_k=tk, tail_v=tv)
        torch.cuda.synchronize()
        assert torch.equal(got[2 * i + 1], again)


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("splits", [1, 2, 8, 9, 31, 32, 33, 41, 70])
def test_split_merge(setup_golden, dtype, splits):
    """Split counts around the merge's batches of 8 and 32 partials (fp32: as many partials; bf16: fewer, see the next)."""
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


MODES = [(2, False), (3, False), (4, False), (2, True), (3, True), (4, True)]


# The unrounded 16-bit kernels against 64 bits, relative to the largest output: weights and value centres are f16 (2^-11 each),
# key centres too, which moves a logit of order 1 by a few 2^-12: 2e-3 in all.  Typical is a tenth of it, since roundings of many
# tokens cancel.
UNROUNDED_TOL = 2e-3


@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("groups", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("dtype", [BF16, F16])
def test_16bit_attention_unrounded(setup_golden, bits, qjl, groups, dtype):
    """The tensor-core kernels at every code width, on both sides of and at a tile of 16 tokens, a warp's 32 and a step of 512."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    store = PackedStore(codec, 2, 3, capacity=513)
    for n in (1, 6, 15, 16, 17, 31, 32, 33, 130, 511, 512, 513):
        store.length = 0
        store.pack(vectors((2, 3, n, 128), 5 + n, dtype), vectors((2, 3, n, 128), 6 + n, dtype))
        q = query((2, 3 * groups, 1), 7 + n, dtype)
        assert rel_inf(store.decode_attn_f32(q), attend64(store, p, q, groups)) <= UNROUNDED_TOL, n


@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("groups", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("dtype", [BF16, F16])
def test_16bit_attention_of_long_rows(setup_golden, bits, qjl, groups, dtype):
    """Up to ten iterations a warp under growing logits, so that the accumulators are rescaled again and again; whole rows to a CTA
    and rows cut by chunks, with the last steps empty for some warps."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    n = 5003
    k = vectors((1, 3, n, 128), 1, F32) * torch.linspace(0.2, 1.2, n, device="cuda")[:, None]
    store = PackedStore(codec, 1, 3, capacity=n)
    store.pack(k.to(dtype), vectors((1, 3, n, 128), 2, dtype))
    q = query((1, 3 * groups, 1), 3, dtype)
    want = attend64(store, p, q, groups)
    for splits in (1, 3, 4, None):
        assert rel_inf(store.decode_attn_f32(q, splits=splits), want) <= UNROUNDED_TOL, splits
    assert codec.device_status() == 0


@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("groups", [2, 4, 5, 8])
@pytest.mark.parametrize("dtype", [BF16, F16])
def test_16bit_attention_of_many_rows(setup_golden, bits, qjl, groups, dtype):
    """More rows than SMs and a ragged length: a CTA goes from one row to the next and merges its warps for each of them."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    store = PackedStore(codec, 41, 8, capacity=700)
    for n in (67, 700):
        store.length = 0
        store.pack(vectors((41, 8, n, 128), 5 + n, dtype), vectors((41, 8, n, 128), 6 + n, dtype))
        q = query((41, 8 * groups, 1), 7 + n, dtype)
        assert rel_inf(store.decode_attn_f32(q), attend64(store, p, q, groups)) <= UNROUNDED_TOL, n
    assert codec.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("shape", [(1, 1, 1024), (1, 8, 129), (3, 5, 127)])
def test_prefill_encoder(setup_golden, bits, qjl, dtype, shape):
    """The tcgen05 encoder from its smallest size on: whole tiles, one vector over, one vector short."""
    from helpers import check_packed
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    k, v = vectors((*shape, 128), 1, dtype, "cpu"), vectors((*shape, 128), 2, dtype, "cpu")
    k[:, :, 5] = 0
    store = PackedStore(codec, shape[0], shape[1], capacity=shape[2] + 9)
    store.pack(k.cuda(), v.cuda())
    assert codec.device_status() == 0
    check_packed(store, O.pack_layer(k, v, p), k, v, p, f"{bits} {qjl} {dtype} {shape}")


def with_boundaries(monkeypatch, setup_golden, bits, qjl, kind):
    """A codec whose codebooks are not Lloyd-Max ones: what a caller of the C interface may bring."""
    from types import SimpleNamespace

    import numpy as np
    from tq_local_b200.runtime import codec as codec_module

    lloyd = codec_module.build_scalar_codebook

    def build(dim, n_bits, grid_size):
        book = lloyd(dim, n_bits, grid_size)
        bnd = np.array(book.boundaries, dtype=np.float64)
        if kind == "close":  # two boundaries a ten-thousandth of the width apart
            bnd[1] = bnd[0] + 1e-4 * (bnd[-1] - bnd[0])
        elif kind == "geometric":
            half = 0.2 * 3.0 ** -np.arange(len(bnd) // 2)
            bnd = np.concatenate((-half, [0.0], half[::-1]))
        return SimpleNamespace(centers=book.centers, boundaries=bnd)

    monkeypatch.setattr(codec_module, "build_scalar_codebook", build)
    return make_codec(bits, qjl, setup_golden)


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("bits,qjl", [(3, False), (4, False), (3, True), (4, True)])
@pytest.mark.parametrize("kind", ["close", "geometric"])
def test_prefill_encoder_of_other_codebooks(setup_golden, monkeypatch, dtype, bits, qjl, kind):
    """Codebooks that no uniform grid separates (the geometric one of seven boundaries: one does): codes against 64 bits, and at
    the tensor cores' speed (the CUDA-core encoder takes more than ten times as long for these vectors)."""
    import numpy as np
    from tq_local_b200.runtime.packed_store import PackedStore

    plain, codec = make_codec(bits, qjl, setup_golden), with_boundaries(monkeypatch, setup_golden, bits, qjl, kind)
    k, v = vectors((1, 8, 9000, 128), 1, dtype), vectors((1, 8, 9000, 128), 2, dtype)
    store = PackedStore(codec, 1, 8, 9000)
    store.pack(k, v)
    for x, codes, n_bits, rot, bnd in ((k, store.k_codes, codec.key_bits, codec.rot_k, codec.bnd_k), (v, store.v_codes, bits, codec.rot_v, codec.bnd_v)):
        rows, edges = x.double().view(-1, 128), torch.from_numpy(bnd).double().cuda()
        z = (rows / rows.norm(dim=1, keepdim=True)) @ torch.from_numpy(np.asarray(rot)).double().cuda().T
        got = torch.from_numpy(O.unpack_codes(codes.reshape(-1, codes.shape[-1]).cpu().numpy(), n_bits, 128).astype(np.int64)).cuda()
        off = got != torch.bucketize(z, edges)
        assert not (off & ((z.unsqueeze(-1) - edges).abs().amin(-1) >= 1e-6)).any()
        assert off.float().mean() < 1e-4
    assert codec.device_status() == 0

    def fastest(c):
        s, best = PackedStore(c, 1, 8, 9000), float("inf")
        for _ in range(12):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            s.length = 0
            begin.record()
            s.pack(k, v)
            end.record()
            torch.cuda.synchronize()
            best = min(best, begin.elapsed_time(end))
        return best

    assert fastest(codec) <= 3 * fastest(plain)


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("qjl", [False, True])
def test_prefill_encoder_extreme_rows(setup_golden, dtype, qjl):
    """Rows whose norm underflows, overflows or is undefined: what the CUDA-core encoder gives (which takes the same
    rows when they are not 16-byte aligned)."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(4, qjl, setup_golden)
    k, v = vectors((1, 2, 1100, 128), 1, dtype), vectors((1, 2, 1100, 128), 2, dtype)
    for x in (k, v):
        x[:, :, 3] *= 1e-5 if dtype == F16 else 1e-30  # squares vanish (fp16: a norm that is subnormal in fp16)
        x[:, :, 4] = 0
        if dtype != F16:
            x[:, :, 10] *= 1e18
            x[:, :, 11] *= 1e22  # squares overflow
        x[:, :, 12, 7] = float("inf")
        x[:, :, 13, 100] = float("nan")
        x[:, :, 14, 1] = -float("inf")
    fast, exact = PackedStore(codec, 1, 2, 1100), PackedStore(codec, 1, 2, 1100)
    fast.pack(k, v)
    exact.pack(off_by_one(k), off_by_one(v))
    rows = [3, 4, 10, 11, 12, 13, 14]
    for name, a, b in zip(("k", "kn", "ks", "kr", "v", "vn") if qjl else ("k", "kn", "v", "vn"), fast.streams(), exact.streams()):
        a, b = a[:, :, rows], b[:, :, rows]
        if a.dtype == torch.float16:  # one ulp, as between any two orders of summation; undefined where undefined
            assert torch.equal(a.isnan(), b.isnan()), name
            a, b = a.nan_to_num(), b.nan_to_num()
            assert (a.view(torch.int16).int() - b.view(torch.int16).int()).abs().max() <= 1, name
        else:
            assert torch.equal(a, b), name


@pytest.mark.parametrize("form", ["transposed", "keys unaligned", "both unaligned"])
def test_prefill_encoder_operand_forms(setup_golden, form):
    """Strides and alignments the kernel takes or hands on: the same codes as from contiguous tensors, outside the 1e-6
    band where the two encoders may differ."""
    from helpers import check_packed
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    k, v = vectors((2, 3, 200, 128), 1, BF16, "cpu"), vectors((2, 3, 200, 128), 2, BF16, "cpu")
    kd, vd = k.cuda(), v.cuda()
    if form == "transposed":
        kd, vd = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (kd, vd))
    else:
        kd = off_by_one(kd)
        vd = off_by_one(vd) if form == "both unaligned" else vd
    store = PackedStore(codec, 2, 3, capacity=216)
    store.pack(vectors((2, 3, 3, 128), 3, BF16), vectors((2, 3, 3, 128), 4, BF16))  # (an odd position to append at)
    store.pack(kd, vd)
    view = PackedStore(codec, 2, 3, capacity=200)
    for a, b in zip(view.streams(), store.streams()):
        a[:, :, :200] = b[:, :, 3:203]
    view.length = 200
    check_packed(view, O.pack_layer(k, v, p), k, v, p, form)


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("shape", [(1, 1, 1024), (1, 8, 129), (3, 5, 127)])
def test_dequantisation(setup_golden, bits, qjl, dtype, shape):
    """The tcgen05 dequantisation from its smallest size on, and the CUDA-core one below it (a slice of few tokens)."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(bits, qjl, setup_golden), make_codec(bits, qjl, setup_golden)
    store = PackedStore(codec, shape[0], shape[1], capacity=shape[2] + 9)
    store.pack(vectors((*shape, 128), 1, dtype), vectors((*shape, 128), 2, dtype))
    layer = store_to_layer(store, p, torch.float32)
    # fp32 sums of 128 products against the oracle's, relative to the largest element; a 16-bit result may in addition
    # be a neighbour of the oracle's, and a key's two rounded parts one each
    ulp = {F32: 0.0, F16: 2.0 ** -10, BF16: 2.0 ** -7}[dtype]
    for which, want in (("keys", O.dequant_keys(layer)), ("values", O.dequant_values(layer))):
        for lo in (0, shape[2] - 3):
            got = store.dequant(which, lo, dtype=dtype).cpu().float()
            ref = want[:, :, lo:]
            room = 2e-6 * ref.abs().max() + ulp * (ref.abs() + 0.5 * ref.abs().amax(dim=-1, keepdim=True) * (which == "keys" and qjl))
            assert ((got - ref).abs() <= room).all(), (which, lo, float((got - ref).abs().max()))
    assert codec.device_status() == 0


@pytest.mark.parametrize("bits,qjl", MODES)
@pytest.mark.parametrize("rows", ["gaussian", "one large element", "few large coordinates"])
def test_fp32_dequantisation_is_as_exact_as_fp32_sums(setup_golden, bits, qjl, rows):
    """fp32 results against 64 bits, also where every product of a sum has the same sign (codes that follow a row of the
    rotation, as those of a vector with one large element do): the 2-norm of the errors stays below what 128 fp32
    multiply-adds one after the other leave, 2.0e-7 of the result (measured over such rows: 1.96e-7 to 2.2e-7)."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec, n = make_codec(bits, qjl, setup_golden), 1 << 16
    gen = torch.Generator(device="cuda").manual_seed(11)
    store = PackedStore(codec, 1, 1, n)
    store.length = n
    to64 = lambda a: torch.from_numpy(a).double().cuda()

    def pack_bits(idx, b):
        words = (idx.view(-1, 16, 8) << (b * torch.arange(8, device="cuda"))).sum(-1)
        return torch.stack([(words >> (8 * i)) & 255 for i in range(b)], -1).to(torch.uint8).view(-1, 16 * b)

    for which, b, rot, cen, codes, norms in (("keys", codec.key_bits, to64(codec.rot_k), to64(codec.cen_k), store.k_codes, store.k_norms),
                                             ("values", bits, to64(codec.rot_v), to64(codec.cen_v), store.v_codes, store.v_norms)):
        if rows == "gaussian":
            z = torch.randn(n, 128, generator=gen, device="cuda", dtype=torch.float64) * 128 ** -0.5
        elif rows == "one large element":
            z = 4 * rot.T[torch.randint(0, 128, (n,), generator=gen, device="cuda")]
        else:
            x = torch.zeros(n, 128, device="cuda", dtype=torch.float64)
            x.scatter_(1, torch.randint(0, 128, (n, 4), generator=gen, device="cuda"), torch.randn(n, 4, generator=gen, device="cuda", dtype=torch.float64))
            z = x / x.norm(dim=1, keepdim=True) @ rot.T
        idx = torch.bucketize(z, (cen[1:] + cen[:-1]) / 2)
        norm = (11.3 * torch.exp(0.5 * torch.randn(n, generator=gen, device="cuda"))).half()
        codes[0, 0].copy_(pack_bits(idx, b)), norms[0, 0].copy_(norm)
        want = (cen[idx] @ rot) * norm.double()[:, None]
        if which == "keys" and qjl:
            sign = torch.randint(0, 2, (n, 128), generator=gen, device="cuda")
            rnorm = (2 * torch.exp(0.5 * torch.randn(n, generator=gen, device="cuda"))).half()
            store.k_signs[0, 0].copy_(pack_bits(sign, 1)), store.k_rnorms[0, 0].copy_(rnorm)
            want += (2 * sign - 1).double() @ to64(codec.qjl) * (math.sqrt(math.pi / 2) / 128) * rnorm.double()[:, None]
        got = store.dequant(which, dtype=F32)[0, 0].double()
        assert float((got - want).norm() / want.norm()) <= 1.9e-7, which
    assert codec.device_status() == 0


MANY = (1, 8, 16001)  # 1001 tiles of 128 vectors, the last of 8: three tiles and more for each group of warps of either kernel


def unpack_on_gpu(codes, bits):
    """[..., 16 * bits] code bytes -> [vectors, 128] indices."""
    b = codes.reshape(-1, 16, bits).long()
    words = sum(b[..., i] << (8 * i) for i in range(bits))
    return ((words.unsqueeze(-1) >> (bits * torch.arange(8, device=codes.device))) & ((1 << bits) - 1)).reshape(-1, 128)


def tables64(codec):
    return {name: torch.from_numpy(getattr(codec, name)).double().cuda() for name in ("rot_k", "rot_v", "cen_k", "cen_v", "bnd_k", "bnd_v")}


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("bits,qjl", MODES)
def test_prefill_encoder_of_many_tiles(setup_golden, bits, qjl, dtype):
    """Every group of warps walks several tiles: codes and norms against 64 bits; signs and residual norms against the
    CUDA-core encoder (which takes the same vectors when they are not 16-byte aligned).  A tile's rows under another tile's
    number, or a tile encoded twice, differ in half of the sign bits and in most codes."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(bits, qjl, setup_golden)
    t = tables64(codec)
    k, v = vectors((*MANY, 128), 1, dtype), vectors((*MANY, 128), 2, dtype)
    store, exact = (PackedStore(codec, MANY[0], MANY[1], MANY[2] + 3) for _ in range(2))
    for s in (store, exact):
        s.pack(k[:, :, :3], v[:, :, :3])  # (an odd position to append at)
    store.pack(k, v)
    exact.pack(off_by_one(k), off_by_one(v))
    same = torch.ones(k[..., 0].numel(), dtype=torch.bool, device="cuda")
    for x, codes, norms, n_bits, rot, edges in ((k, store.k_codes, store.k_norms, codec.key_bits, t["rot_k"], t["bnd_k"]),
                                                (v, store.v_codes, store.v_norms, bits, t["rot_v"], t["bnd_v"])):
        rows = x.double().view(-1, 128)
        norm = rows.norm(dim=1)
        z = rows / norm[:, None] @ rot.T
        off = unpack_on_gpu(codes[:, :, 3:MANY[2] + 3], n_bits) != torch.bucketize(z, edges)
        assert not (off & ((z.unsqueeze(-1) - edges).abs().amin(-1) >= 1e-6)).any() and off.float().mean() < 1e-4
        ulps = norms[:, :, 3:MANY[2] + 3].reshape(-1).view(torch.int16).int() - norm.half().view(torch.int16).int()
        assert ulps.abs().max() <= 1
    if qjl:
        cut = lambda s, name: getattr(s, name)[:, :, 3:MANY[2] + 3]
        same = (cut(store, "k_codes") == cut(exact, "k_codes")).all(-1) & (cut(store, "k_norms") == cut(exact, "k_norms"))
        flips = (unpack_on_gpu(cut(store, "k_signs"), 1) != unpack_on_gpu(cut(exact, "k_signs"), 1)).sum(-1).view(same.shape)
        ulps = (cut(store, "k_rnorms").view(torch.int16).int() - cut(exact, "k_rnorms").view(torch.int16).int()).abs()
        # (a residual whose reconstruction rounds to the other neighbour in a few of its elements: some signs near zero)
        assert same.float().mean() > 0.99 and flips[same].max() <= 16 and flips[same].float().mean() < 0.128
        assert (ulps[same] <= 1).float().mean() > 0.999
    assert codec.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("rows", ["gaussian", "four outlier channels", "four coordinates of 128"])
def test_prefill_encoder_is_as_exact_as_three_terms(setup_golden, dtype, rows):
    """How often the encoder's fp32-like sums decide otherwise than 64 bits do, over 16.8 M coordinates.  Measured over twice as
    many, any of these rows: 3 to 17 codes and 51 to 80 signs (fp32 rows, which round no reconstruction, 9 to 14); with operands
    in three bf16 terms 5 to 89 codes and 257 to 410 signs (38 to 53).  The limits lie between, for half as many."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec, n = make_codec(4, True, setup_golden), 1 << 17
    t = tables64(codec)
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(n, 128, generator=gen, device="cuda")
    if rows == "four outlier channels":
        x[:, [3, 40, 77, 101]] *= 30
    elif rows == "four coordinates of 128":
        x = torch.zeros_like(x).scatter_(1, torch.randint(0, 128, (n, 4), generator=gen, device="cuda"), x[:, :4])
    x = x.to(dtype)
    store = PackedStore(codec, 1, 1, n)
    store.pack(x.view(1, 1, n, 128), x.view(1, 1, n, 128))
    x64 = x.double()
    unit = x64 / x64.norm(dim=1, keepdim=True)
    key_codes = unpack_on_gpu(store.k_codes, codec.key_bits)
    assert int((key_codes != torch.bucketize(unit @ t["rot_k"].T, t["bnd_k"])).sum()) <= 20
    assert int((unpack_on_gpu(store.v_codes, 4) != torch.bucketize(unit @ t["rot_v"].T, t["bnd_v"])).sum()) <= 20
    rec = ((t["cen_k"][key_codes] @ t["rot_k"]) * store.k_norms.view(-1, 1).double()).float().to(dtype).double()
    projected = (x64 - rec) @ torch.from_numpy(codec.qjl).double().cuda().T
    off = int((unpack_on_gpu(store.k_signs, 1).bool() != (projected >= 0)).sum())
    assert off <= (16 if dtype == F32 else 80)
    assert codec.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
@pytest.mark.parametrize("bits,qjl", MODES)
def test_dequantisation_of_many_tiles(setup_golden, bits, qjl, dtype):
    """The same for the dequantisation, every element against 64 bits, from an odd token on."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(bits, qjl, setup_golden)
    t = tables64(codec)
    store = PackedStore(codec, MANY[0], MANY[1], MANY[2] + 3)
    store.pack(vectors((MANY[0], MANY[1], MANY[2] + 3, 128), 1, dtype), vectors((MANY[0], MANY[1], MANY[2] + 3, 128), 2, dtype))
    cut = lambda x: x[:, :, 3:MANY[2] + 3]
    unit = {F32: 2.0 ** -24, F16: 2.0 ** -11, BF16: 2.0 ** -8}[dtype]
    for which, b, rot, cen, codes, norms in (("keys", codec.key_bits, t["rot_k"], t["cen_k"], store.k_codes, store.k_norms),
                                             ("values", bits, t["rot_v"], t["cen_v"], store.v_codes, store.v_norms)):
        want = (cen[unpack_on_gpu(cut(codes), b)] @ rot) * cut(norms).reshape(-1, 1).double()
        rounded = want.abs()  # what is rounded to the type on the way
        if which == "keys" and qjl:
            part = 2.0 * unpack_on_gpu(cut(store.k_signs), 1).double() - 1.0
            part = part @ torch.from_numpy(codec.qjl).double().cuda() * (math.sqrt(math.pi / 2) / 128) * cut(store.k_rnorms).reshape(-1, 1).double()
            want = want + part
            rounded += part.abs() + want.abs()
        got = store.dequant(which, 3, dtype=dtype).double().view(-1, 128)
        # fp32 sums of 128 products (as in test_dequantisation), half a place of every rounding, fp16 subnormals
        room = 2e-6 * want.abs().max() + 1.01 * unit * rounded + 2.0 ** -24
        assert ((got - want).abs() <= room).all(), which
    assert codec.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("partials", [1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 64, 65])
def test_merge_of_every_number_of_partials(setup_golden, dtype, partials):
    """One long row cut into exactly that many partials: the kernel's step times ``partials`` tokens (the last partial of few)
    and one split more, so that a CTA takes one step."""
    from tq_local_b200.runtime import ffi
    from tq_local_b200.runtime.packed_store import PackedStore

    step = ffi.lib().tq_decode_tokens_per_step()
    p, codec = oracle_params(3, True, setup_golden), make_codec(3, True, setup_golden)
    n = step * (partials - 1) + 3
    store = PackedStore(codec, 1, 1, capacity=n)
    store.pack(vectors((1, 1, n, 128), 1, dtype), vectors((1, 1, n, 128), 2, dtype))
    q = query((1, 5, 1), 3, dtype)
    # 16-bit: the plan needs at least ceil(step / (splits - 1)) tokens a partial; fp32: splits partials
    splits = partials + 1 if dtype == BF16 else partials
    assert rel_inf(store.decode_attn(q, splits=splits), attend64(store, p, q, 5)) <= ATTN_TOL[dtype]


@pytest.mark.parametrize("batch,tokens", [(23, 2100), (10, 5582), (3, 23964)])
def test_merge_of_rows_cut_at_different_places(setup_golden, batch, tokens):
    """Chunks that begin inside rows, so that rows have different numbers of partials: two and three, four and five (on
    both sides of what is merged at once), sixteen and seventeen, with 148 SMs."""
    from tq_local_b200.runtime.packed_store import PackedStore

    p, codec = oracle_params(4, True, setup_golden), make_codec(4, True, setup_golden)
    store = PackedStore(codec, batch, 3, capacity=tokens)
    store.pack(vectors((batch, 3, tokens, 128), 1, BF16), vectors((batch, 3, tokens, 128), 2, BF16))
    q = query((batch, 15, 1), 3, BF16)
    want = attend64(store, p, q, 5)
    for splits in (None, 2, 7):
        assert rel_inf(store.decode_attn(q, splits=splits), want) <= ATTN_TOL[BF16], splits


@pytest.mark.parametrize("dtype", [BF16, F16, F32])
def test_append_encoder_staging(setup_golden, dtype):
    """Appends of no more vectors than SMs keep the matrices in shared memory, larger ones read them from L2: the same
    bits."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(4, True, setup_golden)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms // 4  # tokens of two heads, keys and values: 4 n blocks
    assert 4 * n <= sms < 4 * (n + 1)
    k, v = vectors((1, 2, n + 1, 128), 1, dtype), vectors((1, 2, n + 1, 128), 2, dtype)
    few, more = PackedStore(codec, 1, 2, n + 8), PackedStore(codec, 1, 2, n + 8)
    few.pack(k[:, :, :n], v[:, :, :n])
    more.pack(k, v)
    for a, b in zip(few.streams(), more.streams()):
        assert torch.equal(a[:, :, :n], b[:, :, :n])
    assert codec.device_status() == 0


@pytest.mark.parametrize("batch,heads,tokens", [(1, 2, 33), (1, 8, 4099), (4, 8, 2000), (8, 8, 1500)])
def test_recorded_steps_of_several_layers(setup_golden, batch, heads, tokens):
    """Chained steps that release their successors early (few rows and tokens: idle SMs) and that do not: every layer's
    replayed output and stored bytes are those of the same calls made one at a time."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec, layers = make_codec(4, True, setup_golden), 4
    draw = lambda h, t, s: vectors((batch, h, t, 128), s, BF16)
    stores, plain, new = [], [], []
    for i in range(layers):
        k, v = draw(heads, tokens, 10 * i), draw(heads, tokens, 10 * i + 1)
        for group in (stores, plain):
            group.append(PackedStore(codec, batch, heads, tokens + 8))
            group[-1].pack(k, v)
        new.append((query((batch, 4 * heads, 1), 10 * i + 2, BF16), draw(heads, 1, 10 * i + 3), draw(heads, 1, 10 * i + 4)))
    pos = torch.tensor([tokens], dtype=torch.int32, device="cuda")
    step = lambda: [s.decode_step_dev(*x, pos) for s, x in zip(stores, new)]
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = step()
    for n in range(3):
        pos.fill_(tokens + n)
        graph.replay()
        torch.cuda.synchronize()
        for s, p, out, (q, k, v) in zip(stores, plain, outs, new):
            p.pack(k, v)
            torch.cuda.synchronize()
            assert torch.equal(out, p.decode_attn(q, splits=s.suggest_splits(s.capacity)))
            for a, b in zip(s.streams(), p.streams()):
                assert torch.equal(a[:, :, :tokens + n + 1], b[:, :, :tokens + n + 1])
    assert codec.device_status() == 0


@pytest.mark.parametrize("bits,qjl,batch,heads,groups,tokens", [(4, True, 4, 8, 4, 500), (4, True, 4, 8, 4, 1000), (4, True, 1, 8, 4, 8191),
                                                              (4, False, 16, 2, 8, 77), (4, True, 6, 8, 4, 16), (3, True, 4, 4, 7, 2000)])
def test_chained_attention_calls(setup_golden, bits, qjl, batch, heads, groups, tokens):
    """Attention calls in a row, on both sides of the line up to which one starts the next early: each gives what it gives alone."""
    from tq_local_b200.runtime.packed_store import PackedStore

    codec = make_codec(bits, qjl, setup_golden)
    stores = [PackedStore(codec, batch, heads, tokens) for _ in range(3)]
    for i, store in enumerate(stores):
        store.pack(vectors((batch, heads, tokens, 128), 2 * i, BF16), vectors((batch, heads, tokens, 128), 2 * i + 1, BF16))
    qs = [query((batch, heads * groups, 1), 50 + i, BF16) for i in range(12)]
    alone = []
    for i, q in enumerate(qs):
        alone.append(stores[i % 3].decode_attn(q))
        torch.cuda.synchronize()
    chained = [stores[i % 3].decode_attn(q) for i, q in enumerate(qs)]
    for a, b in zip(alone, chained):
        assert torch.equal(a, b)
    assert codec.device_status() == 0


@pytest.mark.parametrize("batch,heads", [(1, 1), (1, 8), (7, 4), (16, 8), (75, 4)])
def test_split_count_within_a_kernel_step(setup_golden, batch, heads):
    """What an attention call may keep: the suggested split count changes only between multiples of the kernel's step."""
    from tq_local_b200.runtime import ffi
    from tq_local_b200.runtime.packed_store import PackedStore

    store, step = PackedStore(make_codec(4, True, setup_golden), batch, heads, 8), ffi.lib().tq_decode_tokens_per_step()
    for k in list(range(40)) + [100, 255]:
        assert len({store.suggest_splits(n) for n in (k * step + 1, k * step + 2, k * step + step // 2, k * step + step - 1, (k + 1) * step)}) == 1
