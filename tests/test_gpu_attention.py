"""tcgen05 flash-attention forward against the fp32 CPU oracle (masks, causal, ragged lengths)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from zenith_b200 import _capi, ops

pytestmark = pytest.mark.gpu


def rng(seed):
    return np.random.default_rng(seed)


def run(cuda, B, H, S, D, causal=False, lens=None, seed=0, dtype=np.float16):
    q, k, v = (rng(seed + i).standard_normal((B, H, S, D)).astype(dtype) for i in range(3))
    kl = None if lens is None else np.array(lens, np.int32)
    o = ops.flash_attention(*(torch.from_numpy(a).to(cuda) for a in (q, k, v)), causal=causal,
                            kv_lens=None if kl is None else torch.from_numpy(kl).to(cuda))
    want = O.attention(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), kl, causal)
    return o, want


@pytest.mark.parametrize("B,H,S,D,causal,lens", [
    (1, 12, 32, 64, False, None),            # the shape of benchmarks/flash_attention_benchmark.py:129-153
    (2, 3, 128, 64, False, [128, 96]),       # key-padding mask as in the encoder
    (1, 2, 256, 64, True, None), (1, 2, 200, 64, False, None), (1, 1, 129, 64, True, None),
    (1, 1, 128, 128, False, None), (2, 2, 384, 128, True, [384, 200]), (1, 2, 1024, 64, True, None),
    (1, 1, 1, 64, False, None), (2, 1, 300, 128, False, [1, 299])])
def test_attention_fp16(cuda, B, H, S, D, causal, lens):
    o, want = run(cuda, B, H, S, D, causal, lens)
    got = o.float().cpu().numpy()
    assert o.dtype == torch.float16 and not np.isnan(got).any()
    # fp16 path within 1e-2 (relative to the output scale) of the fp32 path
    assert np.max(np.abs(got - want)) < 1e-2 * max(1.0, np.abs(want).max())
    assert np.mean(np.abs(got - want)) < 2e-4


@pytest.mark.parametrize("S,D", [(129, 64), (255, 128), (257, 64), (383, 128), (385, 128), (640, 64), (2048, 64), (2049, 64),
                                 (3072, 64), (3073, 64), (4097, 64)])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_at_tile_edges(cuda, S, D, causal):
    """Ends of query tiles and key blocks, a tile without keys of its own, both tile counts per CTA (beyond 2048 tokens at
    head size 64 the count follows the waves), key lengths at and next to a block's end; the last query rows against the oracle."""
    lens = [S, max(1, S - 127), 128, 0] if S < 1000 else [S, S - 1, 1025, 128]
    r = rng(S + D)
    q, k, v = (r.standard_normal((4, 2, S, D)).astype(np.float16) for _ in range(3))
    kl = np.array(lens, np.int32)
    o = ops.flash_attention(*(torch.from_numpy(a).to(cuda) for a in (q, k, v)), causal=causal, kv_lens=torch.from_numpy(kl).to(cuda))
    got = o.float().cpu().numpy()
    assert not np.isnan(got).any()
    rows = np.unique(np.clip([0, 1, 127, 128, S // 2, S - 129, S - 128, S - 1], 0, S - 1))
    want = O.attention_rows(q.astype(np.float32), k.astype(np.float32), v.astype(np.float32), rows, kl, causal)
    assert np.max(np.abs(got[:, :, rows] - want)) < 1e-2


@pytest.mark.parametrize("S", [129, 191, 192, 193, 256, 257, 321, 385, 1025])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_with_four_tiles_per_sm(cuda, S, causal):
    """Head size 64 with tiles enough for the four-tile kernel: ends of its 64-key blocks, sequences without keys, rows whose
    maximum grows past the rescaling threshold late; the edge rows of two heads of every sequence against the oracle."""
    B = 8
    H = -(-1400 // (B * ((S + 127) // 128)))
    r = rng(S)
    q, k, v = (r.standard_normal((B, H, S, 64)).astype(np.float16) for _ in range(3))
    k[:, :, -S // 4:] *= 6
    kl = np.array([S, S - 1, 0, 1, 64, 65, 128, S - 64], np.int32)
    o = ops.flash_attention(*(torch.from_numpy(a).to(cuda) for a in (q, k, v)), causal=causal, kv_lens=torch.from_numpy(kl).to(cuda))
    assert _capi.device_status() == 0
    rows = np.unique(np.clip([0, 1, 31, 32, 63, 64, 127, 128, S // 2, S - 65, S - 64, S - 2, S - 1], 0, S - 1))
    for h in (0, H - 1):
        f = [a[:, h:h + 1].astype(np.float32) for a in (q, k, v)]
        want = O.attention_rows(*f, rows, kl, causal)
        assert np.max(np.abs(o[:, h:h + 1].float().cpu().numpy()[:, :, rows] - want)) < 1e-2
    assert torch.isfinite(o).all() and torch.all(o[2] == 0)


@pytest.mark.parametrize("S", [129, 191, 192, 193, 256, 300, 385, 640])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_with_int8_copy_does_not_depend_on_the_batch(cuda, S, causal):
    """A batch of enough tiles for three CTAs per SM against the same sequences two at a time (the kernel of few tiles): the same
    bits, int8 copy included, at ends of 32-, 64- and 128-key pieces, without keys, with maxima that grow late."""
    heads, B = 12, 2 * (-(-310 // (12 * ((S + 127) // 128))) + 1)
    H = heads * 64
    qkv = torch.from_numpy(rng(S).standard_normal((B * S, 3 * H)).astype(np.float16)).to(cuda)
    qkv.view(B, S, 3 * H)[:, -S // 4:, H:2 * H] *= 6
    lens = torch.from_numpy(np.array([S, S - 1, 0, 1, 33, 64, 65, 96, 127, 128, max(1, S - 64)] * B, np.int32)[:B]).to(cuda)
    st, so = (S * 3 * H, 64, 3 * H), (S * H, 64, H)
    out = [torch.zeros((B * S, H), dtype=torch.float16, device=cuda) for _ in range(2)]
    quant = [torch.zeros((B * S, H), dtype=torch.int8, device=cuda) for _ in range(2)]
    for step, o, oq in zip((B, 2), out, quant):
        for b in range(0, B, step):
            x, rows = qkv[b * S:(b + step) * S], slice(b * S, (b + step) * S)
            ops.flash_attention_strided(x, x[:, H:], x[:, 2 * H:], o[rows], step, heads, S, 64, st, st, st, so, kv_lens=lens[b:b + step],
                                        causal=causal, out_q=oq[rows], out_scale=0.02)
    assert _capi.device_status() == 0
    assert torch.equal(out[0], out[1]) and torch.equal(quant[0], quant[1]) and torch.isfinite(out[0]).all()


@pytest.mark.parametrize("S,causal", [(129, False), (200, True), (300, False), (513, True)])
def test_pinned_attention_does_not_depend_on_the_batch(cuda, S, causal):
    """``keys``: the bits of a sequence alone, in a large batch, packed, and with another max_seqlen; 128 are the bits beside an
    int8 copy, and the two differ.  No value of it changes what there is one form of (short sequences, head size 128)."""
    B, H = 64, 12
    assert _capi.lib().zen_attention_plan(B, H, S, 64, causal, 0) == _capi.ATTN_KEYS_64
    qkv = torch.from_numpy(rng(S).standard_normal((B * S, 3 * H * 64)).astype(np.float16)).to(cuda)
    q, k, v = (t.contiguous() for t in qkv.view(B, S, 3, H, 64).permute(2, 0, 3, 1, 4))
    cu = torch.arange(0, B * S + 1, S, dtype=torch.int32, device=cuda)
    rows = lambda o: o.transpose(1, 2).reshape(B * S, H * 64)
    full = {keys: ops.flash_attention(q, k, v, causal=causal, keys=keys) for keys in (None, 64, 128)}
    assert torch.equal(full[None], full[64]) and not torch.equal(full[64], full[128])
    for keys in (64, 128):
        for b in (0, B - 1):
            part = [t[b:b + 1] for t in (q, k, v)]
            assert torch.equal(ops.flash_attention(*part, causal=causal, keys=keys), full[keys][b:b + 1])
        for max_seqlen in (S, 4 * S):
            assert torch.equal(ops.flash_attention_unpadded(qkv, cu, H, 64, max_seqlen, causal=causal, keys=keys), rows(full[keys]))
    assert torch.equal(ops.flash_attention_unpadded(qkv, cu, H, 64, S, causal=causal, out_scale=0.02, keys=64)[0], rows(full[128]))
    for shape in ((2, 3, 128, 64), (2, 3, 300, 128)):
        x, y, z = (torch.randn(shape, device=cuda, dtype=torch.float16) for _ in range(3))
        assert torch.equal(ops.flash_attention(x, y, z, keys=64), ops.flash_attention(x, y, z, keys=128))


@pytest.mark.parametrize("B,H,S,D,causal", [(3, 2, 700, 128, False), (2, 11, 18432, 64, False), (3, 16, 8320, 128, True)])
def test_attention_does_not_depend_on_the_order_of_tiles(cuda, B, H, S, D, causal):
    """Every order of query tiles, heads and batches (tiles first: full, d = 128 or K and V beyond L2; tiles before batches:
    causal, K and V beyond twice that): the bits of one sequence and of one head on their own."""
    g = torch.Generator(device=cuda).manual_seed(S)
    q, k, v = (torch.randn((B, H, S, D), generator=g, device=cuda, dtype=torch.float16) for _ in range(3))
    lens = torch.tensor([S, S - 129, 77][:B], dtype=torch.int32, device=cuda)
    o = ops.flash_attention(q, k, v, causal=causal, kv_lens=lens)
    for b, h in ((0, H - 1), (B - 1, 0), (1, 1)):
        part = [t[b:b + 1, h:h + 1].contiguous() for t in (q, k, v)]
        assert torch.equal(o[b:b + 1, h:h + 1], ops.flash_attention(*part, causal=causal, kv_lens=lens[b:b + 1]))


@pytest.mark.parametrize("B,H,S,causal", [(16, 16, 2048, False), (16, 16, 4096, True), (26, 16, 1920, True)])
def test_four_tile_kernel_does_not_depend_on_the_order_of_tiles(cuda, B, H, S, causal):
    """Tiles of a head together (full, K and V beyond L2), heads before tiles (causal, beyond twice that), heads and batches first
    (causal, within): the bits of one sequence and of one head on their own."""
    assert _capi.lib().zen_attention_plan(B, H, S, 64, causal, 0) == _capi.ATTN_KEYS_64
    g = torch.Generator(device=cuda).manual_seed(S)
    q, k, v = (torch.randn((B, H, S, 64), generator=g, device=cuda, dtype=torch.float16) for _ in range(3))
    lens = torch.tensor([max(0, S - 129 * b) for b in range(B)], dtype=torch.int32, device=cuda)
    o = ops.flash_attention(q, k, v, causal=causal, kv_lens=lens)
    for b, h in ((0, H - 1), (B - 1, 0), (1, 1)):
        part = [t[b:b + 1, h:h + 1].contiguous() for t in (q, k, v)]
        assert torch.equal(o[b:b + 1, h:h + 1], ops.flash_attention(*part, causal=causal, kv_lens=lens[b:b + 1], keys=64))
    assert _capi.device_status() == 0


@pytest.mark.parametrize("B,heads,S,causal", [(100, 12, 640, False), (26, 16, 2048, True), (90, 12, 640, True)])
def test_three_tile_kernel_does_not_depend_on_the_order_of_tiles(cuda, B, heads, S, causal):
    """The same with an int8 copy, from a fused projection and from packed rows: both results of single sequences."""
    H = heads * 64
    g = torch.Generator(device=cuda).manual_seed(S + B)
    qkv = torch.randn((B * S, 3 * H), generator=g, device=cuda, dtype=torch.float16)
    cu = torch.arange(0, B * S + 1, S, dtype=torch.int32, device=cuda)
    st, so = (S * 3 * H, 64, 3 * H), (S * H, 64, H)

    def padded(x, n, **kw):
        o, oq = (torch.zeros((n * S, H), dtype=t, device=cuda) for t in (torch.float16, torch.int8))
        ops.flash_attention_strided(x, x[:, H:], x[:, 2 * H:], o, n, heads, S, 64, st, st, st, so, causal=causal, out_q=oq, out_scale=0.02, **kw)
        return o, oq

    for whole in (padded(qkv, B), ops.flash_attention_unpadded(qkv, cu, heads, 64, S, causal=causal, out_scale=0.02)):
        for b in (0, 1, B - 1):
            rows = slice(b * S, (b + 1) * S)
            for got, want in zip(whole, padded(qkv[rows], 1)):
                assert torch.equal(got[rows], want)
    assert _capi.device_status() == 0


@pytest.mark.parametrize("order", ["heads", "tiles"])
def test_packed_attention_does_not_depend_on_the_order_of_tiles(cuda, order):
    """Packed rows at head size 64, K and V (by max_seqlen) within and beyond what takes the tiles of a head together; both key
    block sizes."""
    heads, S = 12, 1100
    B = 24 if order == "heads" else 48
    assert (4e-6 * B * heads * S * 64 > 100) == (order == "tiles")
    H = heads * 64
    lens = [(S, 1, 257, 640, 0, 1099)[b % 6] for b in range(B)]
    cu = torch.tensor([0] + list(np.cumsum(lens)), dtype=torch.int32, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(B)
    qkv = torch.randn((sum(lens), 3 * H), generator=g, device=cuda, dtype=torch.float16)
    for keys in (64, 128):
        o = ops.flash_attention_unpadded(qkv, cu, heads, 64, S, keys=keys)
        for b in (0, 1, 2, B - 1):
            lo, n = int(cu[b]), lens[b]
            part = [t.contiguous() for t in qkv[lo:lo + n].view(n, 3, heads, 64).permute(1, 2, 0, 3).unsqueeze(1)]
            pad = [torch.nn.functional.pad(t, (0, 0, 0, max(0, 129 - n))) for t in part]  # (short sequences have a kernel of their own)
            want = ops.flash_attention(*pad, kv_lens=torch.tensor([n], dtype=torch.int32, device=cuda), keys=keys)[:, :, :n]
            assert torch.equal(o[lo:lo + n], want.transpose(1, 2).reshape(n, H))
    assert _capi.device_status() == 0


@pytest.mark.parametrize("S,causal", [(1536, False), (2049, False), (3072, False), (2047, True), (4096, True)])
def test_four_tile_kernel_of_long_sequences(cuda, S, causal):
    """Up to the longest sequences that come there by default, key lengths at ends of 64-key blocks, maxima that grow late; the
    edge rows against the oracle."""
    r = rng(S)
    q, k, v = (r.standard_normal((4, 2, S, 64)).astype(np.float16) for _ in range(3))
    k[:, :, -S // 3:] *= 6
    kl = np.array([S, S - 1, S - 64, 1025], np.int32)
    o = ops.flash_attention(*(torch.from_numpy(a).to(cuda) for a in (q, k, v)), causal=causal, kv_lens=torch.from_numpy(kl).to(cuda), keys=64)
    assert _capi.device_status() == 0
    rows = np.unique([0, 63, 64, 127, 128, 1024, 1025, S // 2, S - 65, S - 64, S - 2, S - 1])
    want = O.attention_rows(*(a.astype(np.float32) for a in (q, k, v)), rows, kl, causal)
    assert np.max(np.abs(o.float().cpu().numpy()[:, :, rows] - want)) < 1e-2


@pytest.mark.parametrize("S", [129, 192, 300, 700, 2048])
@pytest.mark.parametrize("causal", [False, True])
def test_smaller_key_blocks_are_no_further_from_64_bits(cuda, S, causal):
    """Relative error of the result with 64 keys at a time against that with 128, both from softmax in 64 bits: 0.04 to 1.4 % smaller
    over 72 shapes and seeds (its second block moves the reference maximum, so the largest probability is 1 in both)."""
    g = torch.Generator(device=cuda).manual_seed(S)
    q, k, v = (torch.randn((2, 8, S, 64), generator=g, device=cuda, dtype=torch.float16) for _ in range(3))
    lens = torch.tensor([S, S - min(32, S // 4)], dtype=torch.int32, device=cuda)
    pos = torch.arange(S, device=cuda)
    keep = (pos[None, :] < lens[:, None])[:, None, None, :]
    if causal:
        keep = keep & (pos[None, :] <= pos[:, None])
    s = (q.double() @ k.double().transpose(2, 3)) / 8
    want = torch.softmax(s.masked_fill(~keep, float("-inf")), -1) @ v.double()
    err = [(ops.flash_attention(q, k, v, causal=causal, kv_lens=lens, keys=keys).double() - want).norm() / want.norm() for keys in (64, 128)]
    assert err[0] <= err[1] < 4e-4


def test_fully_masked_batch_yields_zeros(cuda):
    o, want = run(cuda, 2, 2, 200, 64, lens=[0, 77])
    assert torch.all(o[0] == 0) and np.all(want[0] == 0)
    assert np.max(np.abs(o[1].float().cpu().numpy() - want[1])) < 1e-2


def test_fp32_binding_shape_and_dtype(cuda):
    """The reference binding takes and returns fp32 [batch, heads, seq, dim] (cuda_bindings.cpp:90-106)."""
    o, want = run(cuda, 1, 12, 32, 64, dtype=np.float32, seed=42)
    assert o.dtype == torch.float32 and tuple(o.shape) == (1, 12, 32, 64)
    assert np.max(np.abs(o.cpu().numpy() - want)) < 1e-2


def test_strided_qkv_and_int8_copy(cuda):
    """Q, K, V read in place from a fused [tokens, 3*hidden] projection; output written as [tokens, hidden]
    with an int8 copy, as the encoder does."""
    B, S, nh, hd = 2, 128, 4, 64
    H = nh * hd
    qkv = rng(1).standard_normal((B * S, 3 * H)).astype(np.float16)
    lens = np.array([128, 50], np.int32)
    t = torch.from_numpy(qkv).to(cuda)
    out = torch.empty((B * S, H), dtype=torch.float16, device=cuda)
    outq = torch.empty((B * S, H), dtype=torch.int8, device=cuda)
    qs, os_ = (S * 3 * H, hd, 3 * H), (S * H, hd, H)
    ops.flash_attention_strided(t, t[:, H:], t[:, 2 * H:], out, B, nh, S, hd, qs, qs, qs, os_,
                                kv_lens=torch.from_numpy(lens).to(cuda), out_q=outq, out_scale=0.02)
    f = qkv.astype(np.float32)
    split = lambda a: np.ascontiguousarray(a.reshape(B, S, nh, hd).transpose(0, 2, 1, 3))
    want = O.attention(split(f[:, :H]), split(f[:, H:2 * H]), split(f[:, 2 * H:]), lens)
    want = want.transpose(0, 2, 1, 3).reshape(B * S, H)
    got = out.float().cpu().numpy()
    assert np.max(np.abs(got - want)) < 1e-2
    assert np.array_equal(outq.cpu().numpy(), O.quantize(got, 0.02))


@pytest.mark.parametrize("S,lens,causal", [
    (128, [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 127], False),  # every kind of boundary inside a 32-key chunk
    (100, [100, 99, 37, 5], False), (100, [100, 64, 33, 1], True), (17, [17, 3], True), (128, [128, 96, 32, 0], True)])
def test_single_block_kernel_key_length_boundaries(cuda, S, lens, causal):
    """Sequences of at most 128 keys (the encoder's kernel): chunk-level masking and the shortened P V product."""
    o, want = run(cuda, len(lens), 2, S, 64, causal, lens, seed=7)
    got = o.float().cpu().numpy()
    assert not np.isnan(got).any()
    assert np.max(np.abs(got - want)) < 1e-2 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("S,hd", [(128, 128), (96, 128), (384, 64), (300, 128)])
def test_int8_copy_equals_quantized_output(cuda, S, hd):
    """Both kernels (one key block / pipelined), both head sizes, strided in and out with key lengths: the int8
    copy is exactly the quantization of the fp16 output beside it."""
    B, nh = 3, 2
    H = nh * hd
    qkv = rng(S + hd).standard_normal((B * S, 3 * H)).astype(np.float16)
    lens = np.array([S, max(1, S // 3), S - 1], np.int32)
    t = torch.from_numpy(qkv).to(cuda)
    out = torch.empty((B * S, H), dtype=torch.float16, device=cuda)
    outq = torch.empty((B * S, H), dtype=torch.int8, device=cuda)
    qs, os_ = (S * 3 * H, hd, 3 * H), (S * H, hd, H)
    ops.flash_attention_strided(t, t[:, H:], t[:, 2 * H:], out, B, nh, S, hd, qs, qs, qs, os_,
                                kv_lens=torch.from_numpy(lens).to(cuda), out_q=outq, out_scale=0.013)
    f = qkv.astype(np.float32)
    split = lambda a: np.ascontiguousarray(a.reshape(B, S, nh, hd).transpose(0, 2, 1, 3))
    want = O.attention(split(f[:, :H]), split(f[:, H:2 * H]), split(f[:, 2 * H:]), lens).transpose(0, 2, 1, 3).reshape(B * S, H)
    got = out.float().cpu().numpy()
    assert np.max(np.abs(got - want)) < 1e-2
    assert np.array_equal(outq.cpu().numpy(), O.quantize(got, 0.013))


def test_properties_at_encoder_size(cuda):
    """B = 32, H = 12, S = 128, d = 64 (too large for the CPU oracle in a test): rows of P sum to one, so
    V = 1 gives O = 1; permuting the keys (with their values) changes nothing beyond fp16 rounding; a key
    length is the same as truncating K and V."""
    B, H, S, D = 32, 12, 128, 64
    g = torch.Generator(device="cpu").manual_seed(3)
    q, k, v = (torch.randn(B, H, S, D, generator=g).half().to(cuda) for _ in range(3))
    ones = ops.flash_attention(q, k, torch.ones_like(v))
    assert (ones.float() - 1).abs().max().item() < 2e-3
    base = ops.flash_attention(q, k, v)
    perm = torch.randperm(S, generator=g).to(cuda)
    assert (ops.flash_attention(q, k[:, :, perm], v[:, :, perm]).float() - base.float()).abs().max().item() < 4e-3
    lens = torch.full((B,), 77, dtype=torch.int32, device=cuda)
    cut = ops.flash_attention(q, k, v, kv_lens=lens)
    # the truncated call has 77 query rows as well (the binding wants equal shapes); compare those rows
    ref = ops.flash_attention(q[:, :, :77].contiguous(), k[:, :, :77].contiguous(), v[:, :, :77].contiguous())
    assert (cut[:, :, :77].float() - ref.float()).abs().max().item() < 2e-3


@pytest.mark.parametrize("S,D,causal", [(1, 64, False), (128, 128, True), (129, 64, True), (300, 64, False)])
def test_fp32_binding_rounds_like_the_fp16_call(cuda, S, D, causal):
    q, k, v = (torch.from_numpy(rng(S + i).standard_normal((2, 3, S, D)).astype(np.float32)).to(cuda) for i in range(3))
    lens = torch.tensor([S, max(1, S // 2)], dtype=torch.int32, device=cuda)
    got = ops.flash_attention(q, k, v, causal=causal, kv_lens=lens)
    want = ops.flash_attention(q.half(), k.half(), v.half(), causal=causal, kv_lens=lens).float()
    assert got.dtype == torch.float32
    assert torch.equal(got, want)  # the same kernels, with fp32 stores


@pytest.mark.parametrize("B,H,S,D,causal,kernels", [
    (3, 5, 257, 128, True, 1), (2, 37, 129, 64, False, 1), (3, 25, 129, 64, False, 2), (2, 16, 513, 64, True, 2), (61, 8, 97, 64, False, 1),
    (40, 9, 128, 128, True, 1), (150, 3, 15, 64, True, 1)])
def test_fp32_operands_converted_by_the_attention_kernel(cuda, B, H, S, D, causal, kernels):
    """Both sides of the line (one tile per SM, of 148), many short items per CTA, sequences without keys: the bits of the fp16
    call, and nothing but finite values where rows end with the allocation."""
    q, k, v = (torch.from_numpy(rng(S + i).standard_normal((B, H, S, D)).astype(np.float32)).to(cuda) for i in range(3))
    lens = torch.tensor([max(0, S - 13 * b) for b in range(B)], dtype=torch.int32, device=cuda)
    before = ops.launch_count
    got = ops.flash_attention(q, k, v, causal=causal, kv_lens=lens)
    if torch.cuda.get_device_properties(cuda).multi_processor_count == 148:
        assert ops.launch_count - before == kernels
    assert torch.equal(got, ops.flash_attention(q.half(), k.half(), v.half(), causal=causal, kv_lens=lens).float())
    assert torch.isfinite(got).all()


@pytest.mark.parametrize("scale", [0.0, -0.125, -1.5, 0.5])
@pytest.mark.parametrize("S,D,causal", [(40, 64, False), (128, 128, True), (100, 64, True), (200, 64, False), (300, 128, True), (2100, 64, False)])
def test_any_scale_with_masked_keys(cuda, S, D, causal, scale):
    """A scale of zero (the mean of the valid keys' values) and negative ones: masked keys stay without weight."""
    q, k, v = (torch.from_numpy(rng(S + i).standard_normal((2, 2, S, D)).astype(np.float16)).to(cuda) for i in range(3))
    lens = torch.tensor([S, max(1, S - 39)], dtype=torch.int32, device=cuda)
    got = ops.flash_attention(q, k, v, causal=causal, kv_lens=lens, scale=scale).double()
    s = scale * (q.double() @ k.double().transpose(2, 3))
    pos = torch.arange(S, device=cuda)
    keep = (pos[None, :] < lens[:, None])[:, None, None, :]
    if causal:
        keep = keep & (pos[None, :] <= pos[:, None])
    want = torch.softmax(s.masked_fill(~keep, float("-inf")), -1) @ v.double()
    assert not torch.isnan(got).any()
    assert (got - want).abs().max().item() < 1e-2 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("which", [(0,), (1,), (2,), (0, 1, 2)])
@pytest.mark.parametrize("S,D,offset", [(1, 64, 1), (33, 64, 2), (128, 128, 3), (197, 64, 1), (300, 128, 5)])
def test_fp32_binding_takes_views_off_a_16_byte_boundary(cuda, S, D, offset, which):
    """Contiguous operands that start at an odd element of a larger tensor: the bits of the aligned call."""
    q, k, v = (torch.from_numpy(rng(S + i).standard_normal((2, 3, S, D)).astype(np.float32)).to(cuda) for i in range(3))

    def shifted(t):
        big = torch.full((t.numel() + offset,), float("nan"), device=cuda)
        big[offset:] = t.flatten()
        return big[offset:].view(t.shape)

    args = [shifted(t) if i in which else t for i, t in enumerate((q, k, v))]
    assert any(t.data_ptr() % 16 for t in args) and all(t.is_contiguous() for t in args)
    assert torch.equal(ops.flash_attention(*args), ops.flash_attention(q, k, v))


@pytest.mark.parametrize("B,H,S,D,causal", [(110, 9, 33, 64, False), (50, 9, 128, 64, True), (37, 9, 100, 128, False)])
def test_single_block_kernel_many_items(cuda, B, H, S, D, causal):
    """More (head, batch) items than the SMs take at a time: tiles, columns and barriers are used again, empty sequences
    between full ones."""
    o, want = run(cuda, B, H, S, D, causal, [(7 * b) % (S + 1) for b in range(B)], seed=3)
    got = o.float().cpu().numpy()
    assert not np.isnan(got).any()
    assert np.max(np.abs(got - want)) < 1e-2 * max(1.0, np.abs(want).max())
