"""Encoder drivers on the device against the CPU oracles.

fp16 encoder  : within 1e-2 (relative to the activation scale) of the fp32 oracle encoder.
int8 encoder  : every int8 GEMM of every layer is checked BIT-EXACTLY against the oracle on the int8
                inputs the device really produced (teacher forcing), the int8 copies are the exact
                quantization of the fp16 tensors beside them, and the final hidden states track the
                oracle's int8 encoder and the fp32 encoder.
"""
import ctypes
import threading

import numpy as np
import pytest
import torch

from oracle import encoder_ref as ER
from oracle import oracle as O
from zenith_b200 import _capi, ops
from zenith_b200.calibrate import activation_scales_from_ranges, calibrate, quantize_weights
from zenith_b200.encoder import EncoderConfig, Fp16Encoder, Int8Encoder, Int8Scales, init_params

pytestmark = pytest.mark.gpu

CFG = EncoderConfig(layers=3, hidden=256, heads=4, ffn=512, vocab=2000, max_pos=128)


def rng(seed):
    return np.random.default_rng(seed)


def batch(seed, B=3, S=96):
    r = rng(seed)
    ids = r.integers(0, CFG.vocab, (B, S))
    lens = (S - r.integers(0, 33, B)).astype(np.int32)
    return ids, lens


def tdev(ids, lens, cuda):
    return torch.from_numpy(ids).to(cuda), torch.from_numpy(lens).to(cuda)


@pytest.fixture(scope="module")
def params():
    return init_params(CFG, 7, random_affine=True)


def test_fp16_encoder_tracks_fp32_oracle(cuda, params):
    enc = Fp16Encoder(CFG, params, cuda)
    ids, lens = batch(1)
    got = enc.forward(*tdev(ids, lens, cuda)).float().cpu().numpy()
    want = ER.encoder_fp32(CFG, params, ids, lens)
    assert np.max(np.abs(got - want)) < 1e-2 * np.abs(want).max() * 3  # 3 layers of fp16 storage
    assert np.mean(np.abs(got - want)) < 2e-3
    # CUDA-graph replay reproduces the eager pass bit for bit
    eager = enc.out.clone()
    enc.capture(*ids.shape)
    enc.set_inputs(*tdev(ids, lens, cuda))
    assert torch.equal(enc.replay(), eager)


def test_device_calibration_matches_oracle_calibration(cuda, params):
    batches = [batch(100 + i) for i in range(4)]
    dev_scales = calibrate(CFG, params, [tdev(i, l, cuda) for i, l in batches], cuda)
    cpu_scales = ER.calibrate_on_oracle(CFG, params, batches, quantize_weights, activation_scales_from_ranges, Int8Scales)
    for a, b in zip(dev_scales.act, cpu_scales.act):
        for k in a:
            assert abs(a[k] - b[k]) / b[k] < 0.03  # fp16 vs fp32 activations
    for a, b in zip(dev_scales.weights, cpu_scales.weights):
        for k in a:
            assert np.array_equal(a[k][0], b[k][0]) and np.array_equal(a[k][1], b[k][1])


def test_int8_encoder_gemms_bit_exact_and_output_tracks_oracle(cuda, params):
    batches = [batch(100 + i) for i in range(4)]
    scales = ER.calibrate_on_oracle(CFG, params, batches, quantize_weights, activation_scales_from_ranges, Int8Scales)
    enc = Int8Encoder(CFG, params, scales, cuda, fuse_layernorm=False, keep_qkv=True)
    ids, lens = batch(2)
    np_ = lambda t: t.cpu().numpy()
    for li, buf in enc.forward_layerwise(*tdev(ids, lens, cuda)):
        a, wq, lp = scales.act[li], scales.weights[li], params["layers"][li]
        # int8 copies == quantization of the fp16 tensor written beside them
        assert np.array_equal(np_(buf["xq"]), O.quantize(np_(buf["x"].float()), a["x"]))
        assert np.array_equal(np_(buf["ctxq"]), O.quantize(np_(buf["ctx"].float()), a["ctx"]))
        assert np.array_equal(np_(buf["h1q"]), O.quantize(np_(buf["h1"].float()), a["h1"]))
        # each GEMM, on the device's own int8 inputs, bit-exact through its fused epilogue
        want = O.linear_int8(np_(buf["xq"]), wq["wqkv"][0], a["x"], wq["wqkv"][1], lp["bqkv"], "none", "f16")
        assert np.array_equal(np_(buf["qkv"]).view(np.uint16), want.view(np.uint16))
        want = O.linear_int8(np_(buf["ctxq"]), wq["wo"][0], a["ctx"], wq["wo"][1], lp["bo"], "none", "f16")
        assert np.array_equal(np_(buf["ao"]).view(np.uint16), want.view(np.uint16))
        want = O.linear_int8(np_(buf["h1q"]), wq["w1"][0], a["h1"], wq["w1"][1], lp["b1"], "gelu", "s8", a["gelu"])
        assert np.array_equal(np_(buf["gq"]), want)
        want = O.linear_int8(np_(buf["gq"]), wq["w2"][0], a["gelu"], wq["w2"][1], lp["b2"], "none", "f16")
        assert np.array_equal(np_(buf["o"]).view(np.uint16), want.view(np.uint16))
        # float kernels on the device's own inputs, within tolerance
        f16 = lambda k: lp[k].astype(np.float16).astype(np.float32)
        want = O.add_layernorm(np_(buf["ao"].float()), np_(buf["x"].float()), f16("ln1_g"), f16("ln1_b"), CFG.eps)
        assert np.max(np.abs(np_(buf["h1"].float()) - want)) < 1e-2
    got = np_(enc.out.float())
    want8 = ER.encoder_int8(CFG, params, scales, ids, lens).astype(np.float32)
    want32 = ER.encoder_fp32(CFG, params, ids, lens)
    assert np.mean(np.abs(got - want8)) < 5e-3 and np.max(np.abs(got - want8)) < 0.1
    assert np.mean(np.abs(got - want32)) < 3e-2
    # graph replay == eager
    eager = enc.out.clone()
    enc.capture(*ids.shape)
    enc.set_inputs(*tdev(ids, lens, cuda))
    assert torch.equal(enc.replay(), eager)
    # QKV projection and attention as two kernels instead of one: bit-identical
    two = Int8Encoder(CFG, params, scales, cuda, fuse_layernorm=False, fuse_attention=False)
    assert torch.equal(two.forward(*tdev(ids, lens, cuda)), eager)
    assert two.launches_per_layer == 7 and enc.launches_per_layer == 6
    # concurrent micro-batches (sequences are independent): bit-identical, eager and replayed
    for n in (2, 3):
        enc_m = Int8Encoder(CFG, params, scales, cuda, micro_batches=n, fuse_layernorm=False)
        assert torch.equal(enc_m.forward(*tdev(ids, lens, cuda)), eager)
        enc_m.capture(*ids.shape)
        enc_m.set_inputs(*tdev(ids, lens, cuda))
        assert torch.equal(enc_m.replay(), eager)


def test_int8_encoder_with_fused_layernorm_kernels(cuda):
    """hidden 768: attention-output and FFN2 run as GEMM + residual + LayerNorm kernels (5 launches / layer)."""
    cfg = EncoderConfig(layers=2, hidden=768, heads=12, ffn=1024, vocab=2000, max_pos=128)
    params = init_params(cfg, 11, random_affine=True)
    mk = lambda s: (rng(s).integers(0, cfg.vocab, (2, 96)), np.array([96, 70], np.int32))
    scales = ER.calibrate_on_oracle(cfg, params, [mk(s) for s in range(3)], quantize_weights,
                                    activation_scales_from_ranges, Int8Scales)
    ids, lens = mk(50)
    enc = Int8Encoder(cfg, params, scales, cuda)
    assert enc.fuse_layernorm
    np_ = lambda t: t.cpu().numpy()
    for li, buf in enc.forward_layerwise(*tdev(ids, lens, cuda)):
        a, wq, lp = scales.act[li], scales.weights[li], params["layers"][li]
        f16 = lambda k: lp[k].astype(np.float16).astype(np.float32)
        # the fused kernel on the device's own inputs: LayerNorm(dequant(ctx_q . Wo) + bo + x)
        t = O.linear_int8(np_(buf["ctxq"]), wq["wo"][0], a["ctx"], wq["wo"][1], lp["bo"], "none", "f32") + np_(buf["x"].float())
        want = O.layernorm(t, f16("ln1_g"), f16("ln1_b"), cfg.eps)
        assert np.max(np.abs(np_(buf["h1"].float()) - want)) < 1e-2
        assert np.array_equal(np_(buf["h1q"]), O.quantize(np_(buf["h1"].float()), a["h1"]))
        want = O.linear_int8(np_(buf["h1q"]), wq["w1"][0], a["h1"], wq["w1"][1], lp["b1"], "gelu", "s8", a["gelu"])
        assert np.array_equal(np_(buf["gq"]), want)
        t = O.linear_int8(np_(buf["gq"]), wq["w2"][0], a["gelu"], wq["w2"][1], lp["b2"], "none", "f32") + np_(buf["h1"].float())
        want = O.layernorm(t, f16("ln2_g"), f16("ln2_b"), cfg.eps)
        assert np.max(np.abs(np_(buf["x_next"].float()) - want)) < 1e-2
    got = np_(enc.out.float())
    want8 = ER.encoder_int8(cfg, params, scales, ids, lens, fused_layernorm=True).astype(np.float32)
    assert np.mean(np.abs(got - want8)) < 5e-3 and np.max(np.abs(got - want8)) < 0.1
    assert enc.launches_per_layer == 4  # QKV + attention, attention-out + LN, FFN1, FFN2 + LN
    unfused = Int8Encoder(cfg, params, scales, cuda, fuse_layernorm=False).forward(*tdev(ids, lens, cuda)).float()
    assert (unfused - enc.out.float()).abs().mean().item() < 5e-3
    two = Int8Encoder(cfg, params, scales, cuda, fuse_attention=False)
    assert torch.equal(two.forward(*tdev(ids, lens, cuda)), enc.out) and two.launches_per_layer == 5
    eager = enc.out.clone()
    enc.capture(*ids.shape)
    enc.set_inputs(*tdev(ids, lens, cuda))
    assert torch.equal(enc.replay(), eager)


def test_host_pipeline_returns_every_batch(cuda):
    """HostPipeline: different batches streamed back to back from pinned host memory come back, in host
    memory, equal to what a plain forward pass gives for each of them."""
    from zenith_b200.serve import HostPipeline

    cfg = EncoderConfig(layers=2, hidden=768, heads=12, ffn=1024, vocab=2000, max_pos=128)
    params = init_params(cfg, 11, random_affine=True)
    mk = lambda s: (rng(s).integers(0, cfg.vocab, (4, 64)), rng(s + 100).integers(1, 65, 4).astype(np.int32))
    scales = ER.calibrate_on_oracle(cfg, params, [mk(s) for s in range(2)], quantize_weights,
                                    activation_scales_from_ranges, Int8Scales)
    enc = Int8Encoder(cfg, params, scales, cuda)
    batches = [mk(20 + i) for i in range(5)]
    want = [enc.forward(*tdev(i, l, cuda)).cpu().clone() for i, l in batches]
    pipe = HostPipeline(enc, 4, 64)
    host = [(torch.from_numpy(i).pin_memory(), torch.from_numpy(l).pin_memory()) for i, l in batches]
    got, prev = [], None
    for ids_h, lens_h in host:
        t = pipe.submit(ids_h, lens_h)
        if prev is not None:
            got.append(pipe.result(prev).clone())
        prev = t
    got.append(pipe.result(prev).clone())
    pipe.drain()
    for g, w in zip(got, want):
        assert torch.equal(g, w)
    with pytest.raises(ValueError):
        pipe.result(0)  # its slot has been reused
    assert _capi.device_status() == 0


@pytest.mark.parametrize("micro_batches", [1, 2])
def test_capture_slots_have_their_own_inputs_and_results(cuda, micro_batches):
    """capture(..., slots=2): two graphs of the same pass, each with its own input block and result buffer; a slot's
    replay leaves the other slot's result alone and gives the bits of a plain forward pass."""
    cfg = EncoderConfig(layers=2, hidden=768, heads=12, ffn=1024, vocab=2000, max_pos=128)
    params = init_params(cfg, 11, random_affine=True)
    mk = lambda s: (rng(s).integers(0, cfg.vocab, (4, 64)), rng(s + 100).integers(1, 65, 4).astype(np.int32))
    scales = ER.calibrate_on_oracle(cfg, params, [mk(s) for s in range(2)], quantize_weights,
                                    activation_scales_from_ranges, Int8Scales)
    enc = Int8Encoder(cfg, params, scales, cuda, micro_batches=micro_batches)
    (ia, la), (ib, lb) = mk(31), mk(32)
    want_a = enc.forward(*tdev(ia, la, cuda)).clone()
    want_b = enc.forward(*tdev(ib, lb, cuda)).clone()
    enc.capture(4, 64, slots=2)
    pack = lambda i, l: torch.from_numpy(np.concatenate([i.reshape(-1), l]).astype(np.int32)).to(cuda)
    enc.inputs_of(0).copy_(pack(ia, la))
    enc.inputs_of(1).copy_(pack(ib, lb))
    ra = enc.replay(0)
    rb = enc.replay(1)
    assert ra.data_ptr() != rb.data_ptr() and ra.data_ptr() == enc.result_of(0).data_ptr()
    assert torch.equal(ra, want_a) and torch.equal(rb, want_b)
    enc.inputs_of(0).copy_(pack(ib, lb))
    assert torch.equal(enc.replay(0), want_b) and torch.equal(enc.result_of(1), want_b)
    if micro_batches != 1:
        return  # the unpadded form runs as one micro-batch
    # the unpadded form takes slots the same way
    cap = Int8Encoder.unpadded_capacity(la.tolist(), 64)
    enc.capture_unpadded(4, 64, max(cap, Int8Encoder.unpadded_capacity(lb.tolist(), 64)), slots=2)
    enc.inputs_of(1).copy_(pack(ia, la))
    got = enc.replay(1)
    rows = torch.from_numpy(np.concatenate([b * 64 + np.arange(int(n)) for b, n in enumerate(la)])).to(cuda)
    assert torch.equal(got[rows], want_a[rows])
    assert _capi.device_status() == 0


def test_fp16_encoder_with_fused_layernorm_kernels(cuda):
    """hidden 768: the fp16 encoder runs attention-output and FFN2 as GEMM + residual + LayerNorm kernels."""
    cfg = EncoderConfig(layers=2, hidden=768, heads=12, ffn=1024, vocab=2000, max_pos=128)
    params = init_params(cfg, 11, random_affine=True)
    ids = rng(50).integers(0, cfg.vocab, (2, 96))
    lens = np.array([96, 70], np.int32)
    enc = Fp16Encoder(cfg, params, cuda)
    assert enc.fuse_layernorm and enc.launches_per_layer == 5
    got = enc.forward(*tdev(ids, lens, cuda)).float().cpu().numpy()
    want = ER.encoder_fp32(cfg, params, ids, lens)
    assert np.max(np.abs(got - want)) < 3e-2 and np.mean(np.abs(got - want)) < 2e-3
    unfused = Fp16Encoder(cfg, params, cuda, fuse_layernorm=False).forward(*tdev(ids, lens, cuda)).float().cpu().numpy()
    assert np.mean(np.abs(unfused - got)) < 2e-3
    eager = enc.out.clone()
    enc.capture(*ids.shape)
    enc.set_inputs(*tdev(ids, lens, cuda))
    assert torch.equal(enc.replay(), eager)
    taps = enc.forward_with_taps(*tdev(ids, lens, cuda))
    assert len(taps["h1"]) == cfg.layers and all(lo < hi for lo, hi in taps["h1"])


@pytest.mark.parametrize("micro_batches", [1, 2])
def test_repeated_plain_calls_equal_the_first(cuda, params, micro_batches):
    """From its third consecutive call for a shape on ``forward`` replays a recorded graph: same bits as the launches it recorded, for
    new inputs, after a change of shape, on another stream, and inside a caller's own capture."""
    enc, ref = (Fp16Encoder(CFG, params, cuda, micro_batches=micro_batches) for _ in range(2))
    mk = lambda s, B, S: tdev(rng(s).integers(0, CFG.vocab, (B, S)), (S - rng(s).integers(0, S // 2, B)).astype(np.int32), cuda)
    for B, S in ((3, 40), (2, 64), (3, 40)):
        for i in range(5):
            ids, lens = mk(10 * B + i, B, S)
            ref._plain_calls = 0  # the reference never records
            assert torch.equal(enc.forward(ids, lens), ref.forward(ids, lens)), (B, S, i)
        assert enc._pass_graph is not None and ref._pass_graph is None
    ids, lens = mk(77, 3, 40)
    want = ref.forward(ids, lens).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = enc.forward(ids, lens).clone()
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(got, want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = enc.forward(ids, lens)
    out.zero_()
    g.replay()
    assert torch.equal(out, want)


@pytest.mark.parametrize("S,micro_batches", [(256, 2), (256, 5), (144, 3)])
def test_fp16_micro_batches_keep_the_bits_of_the_batch(cuda, S, micro_batches):
    """A batch of tiles enough for 64 keys at a time in attention, cut into parts that have too few by themselves."""
    cfg = EncoderConfig(layers=2, hidden=768, heads=12, ffn=1024, vocab=2000, max_pos=256)
    params = init_params(cfg, 3, random_affine=True)
    B = 32
    plan = _capi.lib().zen_attention_plan
    assert plan(B, 12, S, 64, 0, 0) == _capi.ATTN_KEYS_64 and plan(B // micro_batches, 12, S, 64, 0, 0) == _capi.ATTN_KEYS_128
    ids, lens = tdev(rng(1).integers(0, cfg.vocab, (B, S)), (S - rng(2).integers(0, S, B)).astype(np.int32), cuda)
    want = Fp16Encoder(cfg, params, cuda).forward(ids, lens)
    enc = Fp16Encoder(cfg, params, cuda, micro_batches=micro_batches)
    assert torch.equal(enc.forward(ids, lens), want)
    enc.capture(B, S)
    enc.set_inputs(ids, lens)
    assert torch.equal(enc.replay(), want)


def third_call(enc, ids, lens, during):
    """The call that records, with ``during()`` run between two of the recorded launches."""
    issue, calls = enc._issue, []

    def patched(launches, stream):
        issue(launches[:3], stream)
        calls.append(stream)
        if len(calls) == 1:
            during()
        issue(launches[3:], stream)

    enc._issue = patched
    try:
        return enc.forward(ids, lens)
    finally:
        del enc._issue


@pytest.mark.parametrize("error", [RuntimeError, KeyboardInterrupt, _capi.ZenithError])
def test_a_recording_that_fails_is_closed(cuda, params, error):
    enc = Fp16Encoder(CFG, params, cuda)
    ids, lens = tdev(rng(5).integers(0, CFG.vocab, (2, 40)), np.array([40, 17], np.int32), cuda)
    want = enc.forward(ids, lens).clone()
    enc.forward(ids, lens)

    def fail():
        raise error("zen_x", 2, "refused") if error is _capi.ZenithError else error("stopped")

    enc.out.zero_()
    if error is _capi.ZenithError:  # the library refused: the call runs as plain launches
        assert torch.equal(third_call(enc, ids, lens, fail), want)
    else:
        with pytest.raises(error, match="stopped"):
            third_call(enc, ids, lens, fail)
    assert enc._pass_graph is None and not torch.cuda.is_current_stream_capturing()
    for _ in range(4):
        enc.out.zero_()
        assert torch.equal(enc.forward(ids, lens), want)
    enc.forward(ids[:1], lens[:1])
    for _ in range(4):
        assert torch.equal(enc.forward(ids, lens), want)
    assert enc._pass_graph is not None  # another shape in between: recorded anew


@pytest.mark.parametrize("calls_before", [2, 3, 6])
def test_a_pass_goes_into_the_callers_recording(cuda, params, calls_before):
    """Between zen_record_begin and zen_record_end of the caller, whatever call it is: one that would record itself (the third),
    or that would launch what an earlier one has recorded."""
    enc = Fp16Encoder(CFG, params, cuda)
    ids, lens = tdev(rng(8).integers(0, CFG.vocab, (2, 40)).astype(np.int32), np.array([40, 17], np.int32), cuda)
    want = enc.forward(ids, lens).clone()
    for _ in range(calls_before - 1):
        enc.forward(ids, lens)
    lib, graph = _capi.lib(), ctypes.c_void_p()
    assert lib.zen_record_begin() == _capi.OK and lib.zen_record_begin() == _capi.ERR_INVALID_ARG
    out = enc.forward(ids, lens)
    assert lib.zen_memcpy_async(out.data_ptr(), want.data_ptr(), 16, None) == _capi.ERR_UNSUPPORTED
    assert lib.zen_record_end(ctypes.byref(graph)) == _capi.OK and lib.zen_record_end(None) == _capi.ERR_INVALID_ARG
    out.zero_()
    enc.inputs.zero_()
    _capi.call("zen_graph_launch", graph, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(out, want)
    _capi.call("zen_graph_destroy", graph)
    for _ in range(4):  # and plain calls go on
        assert torch.equal(enc.forward(ids, lens), want)


def other_threads_work():
    """What another thread of a program does at any time: random numbers, allocations, pooled streams, synchronisation."""
    torch.randn(8, device="cuda")
    torch.empty(1 << 28, device="cuda")
    filled = []
    for i in range(64):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            filled.append((s, torch.full((64,), i, device="cuda")))
    for i, (s, t) in enumerate(filled):
        s.synchronize()
        assert bool((t == i).all())
    torch.cuda.synchronize()


@pytest.mark.parametrize("micro_batches", [1, 2])
def test_recording_leaves_other_threads_alone(cuda, params, micro_batches):
    enc = Fp16Encoder(CFG, params, cuda, micro_batches=micro_batches)
    ids, lens = tdev(rng(6).integers(0, CFG.vocab, (3, 40)), np.array([40, 17, 9], np.int32), cuda)
    want = enc.forward(ids, lens).clone()
    enc.forward(ids, lens)
    errors = []

    def body():
        try:
            other_threads_work()
        except BaseException as e:
            errors.append(e)

    def during():
        t = threading.Thread(target=body)
        t.start()
        t.join()

    enc.out.zero_()
    assert torch.equal(third_call(enc, ids, lens, during), want)
    assert not errors and enc._pass_graph is not None
    enc.out.zero_()
    assert torch.equal(enc.forward(ids, lens), want)
    del enc  # the graph and its buffers go while it may still run
    torch.cuda.synchronize()
    assert _capi.device_status() == 0


@pytest.mark.parametrize("B,S,packed,workspace", [(1, 24, None, True), (16, 128, None, False), (3, 60, 128, True), (20, 100, 1920, False)])
def test_a_new_shape_prepares_only_what_its_pass_uses(cuda, monkeypatch, B, S, packed, workspace):
    """Kernel choices once per GEMM and not once per layer, LayerNorm scratch only where a choice is two launches, zeros only
    where rows of no sequence exist."""
    cfg = EncoderConfig(layers=3, hidden=768, heads=12, ffn=896, vocab=500, max_pos=128)
    enc = Fp16Encoder(cfg, init_params(cfg, 3), cuda)
    plans, zeros = [], []
    plan, make = _capi.lib().zen_gemm_plan, torch.zeros
    monkeypatch.setattr(_capi.lib(), "zen_gemm_plan", lambda *a: plans.append(a) or plan(*a))
    monkeypatch.setattr(torch, "zeros", lambda *a, **k: zeros.append(a[0]) or make(*a, **k))
    enc._prepare(B, S, packed)
    assert len(plans) == len(set(plans)) and len(plans) <= (6 if packed is None else 8)
    assert (enc.ln_ws is not None) == workspace
    assert ((packed or B * S, 768) in zeros) == (packed is not None)


@pytest.mark.parametrize("B,S,fused,calls,kernels", [(1, 24, True, 5, 7), (16, 128, True, 5, 5), (1, 24, False, 7, 7)])
def test_launch_counts_count_kernels(cuda, B, S, fused, calls, kernels):
    """A projection + LayerNorm of few rows is one call and two kernels; plain calls, recorded ones and replays count alike."""
    cfg = EncoderConfig(layers=3, hidden=768, heads=12, ffn=896, vocab=500, max_pos=128)
    enc = Fp16Encoder(cfg, init_params(cfg, 3), cuda, fuse_layernorm=fused)
    ids, lens = tdev(rng(5).integers(0, cfg.vocab, (B, S)).astype(np.int32), np.full(B, S, np.int32), cuda)
    for _ in range(4):
        before = ops.launch_count
        enc.forward(ids, lens)
        assert ops.launch_count - before == 1 + enc.kernels_per_forward  # and the one that takes the inputs
    assert enc.launches_per_forward == 1 + 3 * calls and enc.kernels_per_forward == 1 + 3 * kernels
    enc.capture(B, S)
    before = ops.launch_count
    enc.replay()
    assert ops.launch_count - before == enc.kernels_per_forward


@pytest.mark.parametrize("B,S,launches", [(1, 48, 5), (1, 49, 4), (112, 6, 5), (112, 16, 4), (150, 8, 5)])
def test_int8_encoder_attention_form_by_size(cuda, params, B, S, launches):
    """Few rows, or many rounds of mostly empty tiles: projection and attention as two launches, with the same bits."""
    scales = Int8Scales(act=[dict(x=0.03, ctx=0.01, h1=0.03, gelu=0.02)] * CFG.layers, weights=quantize_weights(params))
    ids, lens = tdev(rng(B).integers(0, CFG.vocab, (B, S)), rng(S).integers(1, S + 1, B).astype(np.int32), cuda)
    mk = lambda f: Int8Encoder(CFG, params, scales, cuda, fuse_layernorm=False, fuse_attention=f)
    enc = mk(None)
    out = enc.forward(ids, lens)
    assert enc.launches_per_layer == launches + 2  # LayerNorms not fused
    assert torch.equal(out, mk(True).forward(ids, lens)) and torch.equal(out, mk(False).forward(ids, lens))


@pytest.mark.parametrize("B,S", [(1, 1), (3, 85), (5, 120)])
def test_inputs_reach_the_static_buffers(cuda, params, B, S):
    """int32 ids and lengths on the device (one launch), other types and the host (copies), no lengths."""
    enc = Fp16Encoder(CFG, params, cuda)
    ids, lens = tdev(rng(S).integers(0, CFG.vocab, (B, S)).astype(np.int32), rng(B).integers(0, S + 1, B).astype(np.int32), cuda)
    full = torch.full_like(lens, S)
    for a, l, want in ((ids, lens, lens), (ids.long(), lens.long(), lens), (ids.cpu(), lens, lens), (ids.T.contiguous().T, lens, lens),
                       (ids, None, full)):
        enc.set_inputs(a, l)
        assert torch.equal(enc.ids.view(B, S), ids) and torch.equal(enc.kv_lens, want)
        enc.inputs.zero_()
