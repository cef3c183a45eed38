"""The small-product GEMM (K split two or four ways over a cluster; other splits and the tile-width flag are taken as the
nearest) and the two-launch LayerNorm form, forced through the call flags at the edges of their tiles, against the CPU
oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from zenith_b200 import _capi, ops
from zenith_b200._capi import ACT_GELU, ACT_NONE, DT_F16, DT_F32, DT_S8, DT_S32, GEMM_NARROW, gemm_split_k

pytestmark = pytest.mark.gpu
# the kernel's two forms (K split two and four ways) under all the names that the flags have for them
FORMS = [gemm_split_k(k) for k in (1, 2, 4, 8)] + [gemm_split_k(k) | GEMM_NARROW for k in (1, 2, 4)]


def rng(seed):
    return np.random.default_rng(seed)


def dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def call(fn, *args):
    _capi.call(fn, *[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args], torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("flags", FORMS)
@pytest.mark.parametrize("M,N,K", [(1, 32, 1024), (24, 768, 768), (129, 72, 1040), (200, 130, 2048)])
def test_int8_bit_exact_in_every_form(cuda, M, N, K, flags):
    x = rng(M).integers(-128, 128, (M, K), dtype=np.int8)
    w = rng(N).integers(-128, 128, (N, K), dtype=np.int8)
    ws = ((rng(1).random(N) + 0.5) * 3e-4).astype(np.float32)
    b = (rng(2).standard_normal(N) * 0.1).astype(np.float32)
    for dt, td, name, act in ((DT_S32, torch.int32, "s32", ACT_NONE), (DT_F32, torch.float32, "f32", ACT_NONE),
                              (DT_F16, torch.float16, "f16", ACT_NONE), (DT_S8, torch.int8, "s8", ACT_GELU)):
        out = torch.zeros((M, N), dtype=td, device=cuda)
        call("zen_linear_i8_ex", dev(x, cuda), K, dev(w, cuda), K, M, N, K, 0.02, dev(ws, cuda), dev(b, cuda), act, dt, 0.03, 0, out, N,
             None, 0, None, 0, flags)
        if dt == DT_S32:
            want = O.gemm_s8(x, w)
        else:
            want = O.linear_int8(x, w, 0.02, ws, b, "gelu" if act else "none", name, 0.03)
        assert np.array_equal(out.cpu().numpy(), want), name
    assert _capi.device_status() == 0


@pytest.mark.parametrize("flags", FORMS)
def test_fp16_in_every_form(cuda, flags):
    M, N, K = 130, 200, 1536
    x = rng(1).standard_normal((M, K)).astype(np.float16)
    w = (rng(2).standard_normal((N, K)) * 0.05).astype(np.float16)
    out = torch.zeros((M, N), dtype=torch.float32, device=cuda)
    call("zen_linear_f16_ex", dev(x, cuda), K, dev(w, cuda), K, M, N, K, None, ACT_NONE, DT_F32, out, N, flags)
    want = O.gemm_f32_nt(x.astype(np.float32), w.astype(np.float32))
    assert np.max(np.abs(out.cpu().numpy() - want)) < 1e-3 * np.abs(want).max()
    assert _capi.device_status() == 0


@pytest.mark.parametrize("flags", [gemm_split_k(k) | GEMM_NARROW for k in (2, 4)] + [gemm_split_k(14), gemm_split_k(15), 0])
@pytest.mark.parametrize("M,N,K", [(1, 768, 768), (129, 768, 1536), (300, 1024, 4096), (1025, 768, 128)])
def test_layernorm_forms(cuda, M, N, K, flags):
    x = rng(M).integers(-128, 128, (M, K), dtype=np.int8)
    w = rng(K).integers(-128, 128, (N, K), dtype=np.int8)
    ws = ((rng(1).random(N) + 0.5) * 2e-4).astype(np.float32)
    b = (rng(2).standard_normal(N) * 0.1).astype(np.float32)
    res = rng(3).standard_normal((M, N)).astype(np.float16)
    g = (1 + 0.1 * rng(4).standard_normal(N)).astype(np.float16)
    be = (0.1 * rng(5).standard_normal(N)).astype(np.float16)
    y = torch.zeros((M, N), dtype=torch.float16, device=cuda)
    yq = torch.zeros((M, N), dtype=torch.int8, device=cuda)
    scratch = torch.empty((M, N), dtype=torch.float32, device=cuda)
    call("zen_linear_i8_add_layernorm_ws", dev(x, cuda), K, dev(w, cuda), K, M, N, K, 0.02, dev(ws, cuda), dev(b, cuda), dev(res, cuda), N,
         dev(g, cuda), dev(be, cuda), 1e-12, y, yq, 0.03, 0, scratch, scratch.numel() * 4, flags)
    t = O.linear_int8(x, w, 0.02, ws, b, "none", "f32") + res.astype(np.float32)
    want = O.layernorm(t, g.astype(np.float32), be.astype(np.float32), 1e-12)
    got = y.float().cpu().numpy()
    assert np.max(np.abs(got - want)) < 4e-3
    assert np.array_equal(yq.cpu().numpy(), O.quantize(got, 0.03))
    assert _capi.device_status() == 0


@pytest.mark.parametrize("offset", [(1, 0), (0, 2), (3, 3)])
@pytest.mark.parametrize("elem,M,N,K", [(1, 1, 768, 768), (1, 300, 1024, 1024), (1, 1025, 768, 128), (2, 1025, 768, 128)])
def test_layernorm_parameters_may_start_anywhere(cuda, elem, M, N, K, offset):
    """gamma and beta as views at an odd element of a larger vector, in sizes that run as two launches when they are aligned:
    the same bits."""
    x, w = (torch.from_numpy(rng(s).integers(-100, 100, (n, K), dtype=np.int8)).to(cuda) for s, n in ((M, M), (K, N)))
    res = torch.from_numpy(rng(3).standard_normal((M, N)).astype(np.float16)).to(cuda)
    vectors = [torch.from_numpy(rng(s).standard_normal(N + 8).astype(np.float16)).to(cuda) for s in (4, 5)]
    moved = [torch.cat((v.new_zeros(o), v[:N]))[o:] for v, o in zip(vectors, offset)]
    assert any(v.data_ptr() % 8 for v in moved)

    def run(g, b):
        if elem == 2:
            return (ops.linear_fp16_add_layernorm(x.half() * 0.02, w.half() * 0.001, None, res, g, b, 1e-12),)
        return ops.linear_int8_add_layernorm(x, w, 0.02, None, None, res, g, b, 1e-12, out_scale=0.03)

    for got, want in zip(run(*moved), run(*(v[:N] for v in vectors))):
        assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K", [(1, 768, 768), (129, 768, 3072), (300, 1024, 1024), (1025, 768, 768), (4300, 768, 128)])
def test_layernorm_forms_give_the_same_bits(cuda, M, N, K):
    """One kernel, two launches, two launches with K split: a batch that crosses a rule's line keeps its rows' bits (int8; fp16
    where K is not split).  4300 rows are more than one round of the clusters."""
    x, w = (torch.from_numpy(rng(s).integers(-128, 128, (n, K), dtype=np.int8)).to(cuda) for s, n in ((M, M), (K, N)))
    ws, b = dev(((rng(1).random(N) + 0.5) * 2e-4).astype(np.float32), cuda), dev(rng(2).standard_normal(N).astype(np.float32), cuda)
    res = dev((rng(3).standard_normal((M, N)) * 3).astype(np.float16), cuda)
    g, be = (dev(rng(s).standard_normal(N).astype(np.float16), cuda) for s in (4, 5))
    scratch = torch.empty((M, N), dtype=torch.float32, device=cuda)

    def run(flags, elem):
        y, yq = torch.zeros((M, N), dtype=torch.float16, device=cuda), torch.zeros((M, N), dtype=torch.int8, device=cuda)
        tail = (b, res, N, g, be, 1e-12, y, yq, 0.03, 0, scratch, scratch.numel() * 4, flags)
        if elem == 1:
            call("zen_linear_i8_add_layernorm_ws", x, K, w, K, M, N, K, 0.02, ws, *tail)
        else:
            call("zen_linear_f16_add_layernorm_ws", x.half() * 0.02, K, w.half() * 0.001, K, M, N, K, *tail)
        return y, yq

    for elem, flags in ((1, [14, 2, 4]), (2, [14])):
        want = run(gemm_split_k(15), elem)
        for f in flags:
            got = run(gemm_split_k(f) | (GEMM_NARROW if f < 14 else 0), elem)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (elem, f)


def test_layernorm_form_follows_the_resident_clusters(cuda):
    """A row block more than the clusters that are resident at once (fewer than SMs / 4) is a second round."""
    form = lambda blocks, K: (_capi.lib().zen_gemm_plan(1, blocks * 128, 768, K, 1) >> 20) & 0xf
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for K in (768, 3072):
        line = next(n for n in range(26, sms // 4 + 2) if form(n, K) != 15)
        assert line <= sms // 4 and all(form(n, K) == 14 for n in range(line, sms // 4 + 2))


@pytest.mark.parametrize("M,N,K", [(1, 8, 192), (3, 64, 200), (130, 72, 264), (256, 1024, 768), (257, 1024, 768), (64, 3072, 768), (65, 3072, 768),
                                   (384, 1024, 1024), (385, 1024, 1024), (512, 1024, 2048), (513, 1024, 2048), (48, 4096, 1016)])
def test_matmul_of_row_major_operands_at_the_lines_of_its_rule(cuda, M, N, K):
    """wmma_matmul on both sides of every line between the K splits and the large tiles.  fp16 products are exact in fp32, and
    sums of K of them in any order lie within K * 2^-24 of the sum of magnitudes; the bound leaves 2^-19 (K <= 2048: 2^-13)."""
    a, b = (torch.from_numpy(rng(s).standard_normal(sh).astype(np.float16)).to(cuda) for s, sh in ((M, (M, K)), (N, (K, N))))
    got = ops.wmma_matmul(a, b)
    want, scale = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    assert bool(((got - want).abs() <= 2.0**-19 * scale).all())


@pytest.mark.parametrize("M,N,K,offset", [(1, 1, 4, 0), (128, 32, 32, 0), (129, 33, 36, 1), (385, 78, 96, 0), (500, 1000, 100, 3), (1100, 100, 2120, 0),
                                          (200, 1088, 1000, 2), (130, 1120, 128, 0), (257, 1536, 512, 1), (257, 1537, 300, 0), (129, 2369, 512, 0)])
def test_fp32_matmul_transposes_b_on_its_way_in(cuda, M, N, K, offset):
    """Both sides of every line of its rule (33 and 66 tiles of 128 x 32, 74 of 128 x 64; fewer k-blocks than ways), ragged edges, and a B
    that starts off the 16-byte grid.  TF32 drops 13 bits of each operand, a relative error below 2^-10 each, so a result is within
    (2^-9 + 2^-20) sum |a||b| of the exact one, and the fp32 sums add less than 2^-16 of that (K < 2^8 x 32 ordered terms)."""
    a = torch.from_numpy(rng(M).standard_normal((M, K)).astype(np.float32)).to(cuda)
    b = torch.empty(N * K + offset, device=cuda)[offset:].view(K, N)
    b.copy_(torch.from_numpy(rng(N).standard_normal((K, N)).astype(np.float32)))
    c = torch.full((M, N), float("nan"), device=cuda)
    ws = torch.empty(4 * N * K, dtype=torch.uint8, device=cuda)
    call("zen_matmul_f32", a, b, c, M, N, K, ws, ws.numel())
    bound = (a.double().abs() @ b.double().abs()) * (2.0**-9 + 2.0**-15)
    assert bool(((c.double() - a.double() @ b.double()).abs() <= bound).all())
    assert _capi.device_status() == 0


@pytest.mark.parametrize("M,N,K,direct", [(128, 1000, 4096, True), (860, 100, 2120, True), (385, 400, 96, True), (384, 352, 132, True),
                                          (256, 544, 132, True), (384, 704, 264, True), (128, 2144, 264, True), (129, 2368, 512, True),
                                          (129, 2369, 512, False), (128, 4736, 64, True), (128, 4737, 64, False), (1000, 1000, 68, False)])
def test_fp32_matmul_at_the_lines_of_its_rule(cuda, M, N, K, direct):
    """Which products are one launch, and their results: 32 and 28 tiles with more k-blocks than the deep ring has stages, 52 tiles of a
    K that goes to 64 columns, 33 / 34 and 66 / 67 tiles of 128 x 32, 74 of 128 x 64 and one more.  The one launch's result is
    zen_matmul_f32's, bit for bit; the bound against 64 bits as above."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines lie elsewhere")
    a = torch.from_numpy(rng(M).standard_normal((M, K)).astype(np.float32)).to(cuda)
    b = torch.from_numpy(rng(N).standard_normal((K, N)).astype(np.float32)).to(cuda)
    one, c = (torch.full((M, N), float("nan"), device=cuda) for _ in range(2))
    ws = torch.empty(4 * N * K, dtype=torch.uint8, device=cuda)
    status = _capi.lib().zen_matmul_f32_direct(a.data_ptr(), b.data_ptr(), one.data_ptr(), M, N, K, torch.cuda.current_stream().cuda_stream)
    assert status == (_capi.OK if direct else _capi.ERR_NEEDS_WORKSPACE)
    call("zen_matmul_f32", a, b, c, M, N, K, ws, ws.numel())
    bound = (a.double().abs() @ b.double().abs()) * (2.0**-9 + 2.0**-15)
    assert bool(((c.double() - a.double() @ b.double()).abs() <= bound).all())
    assert torch.equal(one, c) if direct else bool(one.isnan().all())
    assert _capi.device_status() == 0
