"""GPU parity of the factored-LSTM kernels, called through the C ABI.

Bar (f16 tensor-core contraction, f32 accumulate in an unspecified order): cell state within
1e-2 of the oracle, no int8 hidden code off by more than 1; across a recurrent layer the same
bar holds per step while the fraction of differing codes stays small. Batch shards reproduce
the unsharded result bit for bit.
"""
import ctypes

import numpy as np
import pytest
import torch

from fluke_b200 import lib as L, ops, prep
from fluke_b200.lstm import FactoredLstmLayer, StackPipeline, run_stack, run_stack_c
from fluke_b200.shard import shard_range
from oracle import port

pytestmark = pytest.mark.gpu
DEV = "cuda"


# name -> (mode for fluke_set_lstm_persistent, form fluke_sm100_lstm_last_form then reports)
LSTM_MODES = {"small_clusters": (1, 3), "cluster": (4, 1), "persistent_l2": (2, 2), "per_step": (0, 0)}


@pytest.fixture(params=list(LSTM_MODES))
def lstm_mode(request, flib):
    """Runs a test with each form of the layer recurrence: one launch with few chunk rows per thread-block cluster
    (the default), one with the exchange inside larger clusters, one with the exchange through L2, and two
    launches per step."""
    flib.fluke_set_lstm_persistent(LSTM_MODES[request.param][0])
    yield request.param
    flib.fluke_set_lstm_persistent(1)


@pytest.fixture(autouse=True)
def _default_form_afterwards(flib):
    """A test that fails between two forms leaves the next one the default."""
    yield
    flib.fluke_set_lstm_persistent(1)


@pytest.mark.parametrize("B,H,Kc", [(256, 1024, 256), (128, 768, 256), (100, 768, 256), (200, 96, 128), (1, 64, 64), (1024, 768, 256)])
def test_step_vs_oracle(B, H, Kc):
    g = torch.Generator().manual_seed(B + H)
    A = (torch.randn(B, Kc, generator=g) * 0.3).half(); W = (torch.randn(4 * H, Kc, generator=g) * 0.1).half()
    bias = torch.randn(4 * H, generator=g) * 0.1; c = torch.randn(B, H, generator=g) * 0.1
    cg = c.clone().to(DEV)
    hg = ops.factored_lstm_step_i8(A.to(DEV), W.to(DEV), bias.to(DEV), cg)
    ce, he = port.lstm_step(A.numpy(), W.numpy(), bias.numpy(), c.numpy())
    assert np.abs(cg.cpu().numpy() - ce).max() < 1e-4
    d = np.abs(hg.cpu().numpy().astype(np.int32) - he.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() < 1e-3


@pytest.mark.parametrize("B,H", [(1, 768), (129, 768), (257, 768), (641, 768), (769, 768), (1281, 512), (2000, 768), (640, 96), (300, 48)])
def test_step_of_every_unit_width_vs_oracle(B, H):
    """Rows and hidden sizes on either side of where the kernel changes between 16, 32, 48 and 64 units per
    block on a B200, ragged last row tiles. Cells: 256 products of f16 values summed in f32, then one
    fma, 2^-24 * 256 relative to sums of order 1; a code differs where 127 h lies at a rounding boundary."""
    g = torch.Generator().manual_seed(B + H)
    A = (torch.randn(B, 256, generator=g) * 0.3).half(); W = (torch.randn(4 * H, 256, generator=g) * 0.1).half()
    bias = torch.randn(4 * H, generator=g) * 0.1; c = torch.randn(B, H, generator=g) * 0.1
    cg = c.clone().to(DEV)
    hg = ops.factored_lstm_step_i8(A.to(DEV), W.to(DEV), bias.to(DEV), cg)
    ce, he = port.lstm_step(A.numpy(), W.numpy(), bias.numpy(), c.numpy())
    assert np.abs(cg.cpu().numpy() - ce).max() < 1e-4
    d = np.abs(hg.cpu().numpy().astype(np.int32) - he.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() < 1e-3


def test_step_golden_from_reference_test(golden_tests):
    g = golden_tests
    H = g["lstm_c"].shape[1]
    A = np.concatenate([g["lstm_hh_down"], g["lstm_x_down"]], 1).astype(np.float16)
    W = np.concatenate([np.concatenate([g["lstm_up_hh"][k * H:(k + 1) * H], g["lstm_up_ih"][k * H:(k + 1) * H]], 1) for k in range(4)], 0).astype(np.float16)
    bias = (g["lstm_bhh"] + g["lstm_bih"]).astype(np.float32)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    c = T(g["lstm_c"])
    h = ops.factored_lstm_step_i8(T(A), T(W), T(bias), c)
    assert (c.cpu() - torch.from_numpy(g["lstm_c_ref"])).abs().max() < 0.08   # ABS_TOL of cute/test_factored_lstm.py
    assert (h.float().cpu() / 127.0 - torch.from_numpy(g["lstm_h_ref"])).abs().max() < 0.08


def test_fp8_export_step_golden_from_fly_reference_test(golden_tests):
    """The fused step of the reference's fp8 export (fly/rdna4/factored_lstm/rdna_fp8_factored_lstm.py)
    against the torch reference of fly/test_factored_lstm.py on inputs drawn as that test draws
    them; its bar (:66-72): cell < 1e-2, every int8 code within one level."""
    g = golden_tests
    T = lambda k: torch.from_numpy(np.ascontiguousarray(g[k])).to(DEV)
    c = T("flstm8_c0")
    h = ops.factored_lstm_step_i8(T("flstm8_A"), T("flstm8_W"), T("flstm8_bias"), c, fp8_export_name=True)
    assert (c.cpu() - torch.from_numpy(g["flstm8_c_ref"])).abs().max() < 1e-2
    d = (h.cpu().int() - torch.from_numpy(g["flstm8_h_ref"]).int()).abs()
    assert int(d.max()) <= 1
    # and the oracle on the same inputs: same bar against the reference, tighter against the kernel
    ce, he = port.lstm_step(g["flstm8_A"], g["flstm8_W"], g["flstm8_bias"], g["flstm8_c0"])
    assert np.abs(ce - g["flstm8_c_ref"]).max() < 1e-2 and np.abs(he.astype(np.int32) - g["flstm8_h_ref"].astype(np.int32)).max() <= 1
    assert np.abs(c.cpu().numpy() - ce).max() < 1e-4


@pytest.mark.parametrize("M", [48, 128, 1024, 300])
def test_fp8_down_projection_vs_oracle_and_fly_reference(golden_tests, M):
    """fluke_down_proj_fp8_gpu (N = R = 128, K = H = 768): against the oracle within 1e-2 of the
    output RMS (f32 accumulation order), against the reference construction of the fly tests
    within their 5e-2, and into a wider buffer (row stride)."""
    gt = golden_tests
    if M == 48:   # the fixture built with the reference's own fp8 quantisers
        a8, sa = torch.from_numpy(gt["dp8_A"]), torch.from_numpy(gt["dp8_sa"])
        w8 = torch.from_numpy(np.ascontiguousarray(gt["dp8_B_kn"].T)); sb = torch.from_numpy(gt["dp8_sb"])
    else:
        g = torch.Generator().manual_seed(M)
        a, sa = prep.quantize_fp8_rows(torch.randn(M, 768, generator=g) * 0.3)
        w, sb = prep.quantize_fp8_rows(torch.randn(128, 768, generator=g) / 768 ** 0.5)
        a8, w8 = a.view(torch.uint8), w.view(torch.uint8)
    buf = torch.full((M, 256), 3.0, dtype=torch.float16, device=DEV)
    ops.down_proj_fp8(a8.to(DEV), w8.to(DEV), sa.to(DEV), sb.to(DEV), out=buf[:, :128])
    got = buf[:, :128].float().cpu().numpy()
    assert bool((buf[:, 128:] == 3.0).all())
    exp = port.down_proj_fp8(a8.numpy(), w8.numpy(), sa.numpy(), sb.numpy()).astype(np.float32)
    assert np.abs(got - exp).max() <= 1e-2 * np.sqrt((exp ** 2).mean())
    if M == 48:
        assert np.abs(got - gt["dp8_expected"].astype(np.float32)).max() < 5e-2
    # a preshuffled weight, as the fp8 ABI passes it, goes through the re-ordering kernel once
    wsh = prep.preshuffle_fp8_weight(w8)
    plain = ops.fp8_unshuffle(wsh.to(DEV), 128, 768)
    again = ops.down_proj_fp8(a8.to(DEV), plain, sa.to(DEV), sb.to(DEV))
    assert torch.equal(again, buf[:, :128])


def test_per_step_entry_points_with_an_explicit_stream(flib):
    """The `_stream` forms of the two per-step kernels launch on the stream they are given (here a
    side stream while the thread's own setting stays the default stream) and give the bytes of the
    forms without it; a step loop driven this way equals the layer entry point's per-step mode."""
    T, B, H, R = 4, 200, 768, 128
    layer, x, xs = _layer_case(T, B, H, R, 21, False)
    X, XS = x.to(DEV), xs.to(DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    A = torch.empty(B, 2 * R, dtype=torch.float16, device=DEV)
    outs = []
    w = [layer.w_up.data_ptr() + g * H * 2 * R * 2 for g in range(4)]
    bs = [layer.bias.data_ptr() + g * H * 4 for g in range(4)]
    assert flib.fluke_get_stream() is None
    with torch.cuda.stream(side):
        for t in range(T):
            assert flib.fluke_down_proj_i8_stream_gpu(A.data_ptr(), 2 * R, h.data_ptr(), layer.dn_hh.data_ptr(), 0,
                                                      layer.dn_hh_scale.data_ptr(), B, R, H, side.cuda_stream) == 0
            assert flib.fluke_down_proj_i8_stream_gpu(A.data_ptr() + 2 * R, 2 * R, X[t].data_ptr(), layer.dn_ih.data_ptr(),
                                                      XS[t * B:(t + 1) * B].data_ptr(), layer.dn_ih_scale.data_ptr(), B, R, H,
                                                      side.cuda_stream) == 0
            hn = torch.empty(B, H, dtype=torch.int8, device=DEV)
            assert flib.fluke_factored_lstm_step_i8_stream_gpu(A.data_ptr(), w[0], w[1], w[2], w[3], bs[0], bs[1], bs[2], bs[3],
                                                               c.data_ptr(), hn.data_ptr(), B, H, 2 * R, side.cuda_stream) == 0
            h = hn
            outs.append(hn)
    side.synchronize()
    flib.fluke_set_lstm_persistent(0)
    c2 = torch.zeros(B, H, device=DEV); h2 = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    want = ops.factored_lstm_layer_i8(X, XS, layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up, layer.bias, c2, h2)
    flib.fluke_set_lstm_persistent(1)
    assert torch.equal(torch.stack(outs), want) and torch.equal(c, c2)


def test_hidden_quantiser_rounds_half_away_from_zero():
    """Gates forced open (large o bias, zero weights): h = tanh(c); codes at +-k.5/127 round away."""
    B, H, Kc = 128, 64, 64
    ks = torch.arange(0, 64).float()
    target = (ks + 0.5) / 127.0
    c_prev = torch.atanh(target.clamp(max=0.999)).repeat(B, 1)
    c_prev[::2] *= -1
    A = torch.zeros(B, Kc, dtype=torch.float16); W = torch.zeros(4 * H, Kc, dtype=torch.float16)
    bias = torch.zeros(4 * H); bias[H:2 * H] = 10.0; bias[3 * H:] = 10.0   # f = 1, o = 1, i*g = 0.5*0
    cg = c_prev.clone().to(DEV)
    h = ops.factored_lstm_step_i8(A.to(DEV), W.to(DEV), bias.to(DEV), cg).cpu()
    _, he = port.lstm_step(A.numpy(), W.numpy(), bias.numpy(), c_prev.numpy())
    assert np.abs(h.numpy().astype(np.int32) - he.astype(np.int32)).max() <= 1
    assert torch.equal(h[0], -h[1])  # symmetric rounding


def _layer_case(T, B, H, R, seed, reverse):
    g = torch.Generator().manual_seed(seed)
    layer = FactoredLstmLayer.random(H, R, reverse, g, DEV)
    x, xs = prep.quantize_int8_rows(torch.randn(T * B, H, generator=g))
    return layer, x.view(T, B, H), xs


def _run_oracle_layer(layer, x, xs, reverse, c0=None, h0=None):
    B, H = x.shape[1], x.shape[2]
    c0 = np.zeros((B, H), np.float32) if c0 is None else c0
    h0 = np.zeros((B, H), np.int8) if h0 is None else h0
    n = lambda t: t.cpu().numpy()
    return port.lstm_layer(x.numpy(), None if xs is None else xs.numpy(), n(layer.dn_ih), n(layer.dn_ih_scale), n(layer.dn_hh),
                           n(layer.dn_hh_scale), n(layer.w_up), n(layer.bias), c0, h0, reverse)


@pytest.mark.parametrize("T,B,reverse", [(12, 200, False), (12, 200, True), (40, 128, False), (3, 1, True),
                                         (6, 330, True), (5, 60, False)])
def test_layer_vs_oracle(T, B, reverse, lstm_mode):
    H, R = 768, 128
    layer, x, xs = _layer_case(T, B, H, R, 42 + T, reverse)
    c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    ho = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                    layer.w_up, layer.bias, c, h, reverse=reverse)
    assert L.load().fluke_sm100_lstm_last_form() == LSTM_MODES[lstm_mode][1]  # each form covers this shape
    he, ce, hf = _run_oracle_layer(layer, x, xs, reverse)
    d = np.abs(ho.cpu().numpy().astype(np.int32) - he.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() < 5e-3
    assert np.abs(c.cpu().numpy() - ce).max() < 1e-2
    last = 0 if reverse else T - 1
    assert torch.equal(h, ho[last])  # final hidden state = last written step


def test_layer_resumes_from_state_and_fixed_scale_input(lstm_mode):
    """Two halves run back to back (state carried in c/h) equal one run; input at the fixed
    1/127 scale (x_scale NULL) as for layers fed by a previous layer."""
    T, B, H, R = 10, 130, 768, 128
    layer, x, _ = _layer_case(T, B, H, R, 7, False)
    run = lambda xx, c, h: ops.factored_lstm_layer_i8(xx.to(DEV), None, layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                                      layer.w_up, layer.bias, c, h)
    c1 = torch.zeros(B, H, device=DEV); h1 = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    whole = run(x, c1, h1)
    c2 = torch.zeros(B, H, device=DEV); h2 = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    first = run(x[:5].contiguous(), c2, h2); second = run(x[5:].contiguous(), c2, h2)
    assert torch.equal(whole, torch.cat([first, second])) and torch.equal(c1, c2) and torch.equal(h1, h2)
    he, _, _ = _run_oracle_layer(layer, x, None, False)
    assert np.abs(whole.cpu().numpy().astype(np.int32) - he.astype(np.int32)).max() <= 1


def test_stack_alternating_directions_and_batch_shards(lstm_mode):
    """3-layer stack (odd layer reversed): sharding the chunk axis over 2 'ranks' reproduces
    the unsharded output bit for bit; the stack agrees with the oracle stack within one code
    per layer input."""
    T, B, H, R = 8, 192, 768, 128
    g = torch.Generator().manual_seed(1)
    layers = [FactoredLstmLayer.random(H, R, bool(i % 2), g, DEV) for i in range(3)]
    x, xs = prep.quantize_int8_rows(torch.randn(T * B, H, generator=g))
    x = x.view(T, B, H); xs2 = xs.view(T, B)
    full, _ = run_stack(layers, x.to(DEV), xs.to(DEV))
    full = full.clone()
    parts = []
    for rank in range(2):
        b0, b1 = shard_range(B, rank, 2)
        out, _ = run_stack(layers, x[:, b0:b1].contiguous().to(DEV), xs2[:, b0:b1].contiguous().view(-1).to(DEV))
        parts.append(out.clone())
    assert torch.equal(full, torch.cat(parts, dim=1))
    # oracle stack, feeding each layer the ORACLE's own previous output
    cur, cur_s = x, xs
    for layer in layers:
        he, _, _ = _run_oracle_layer(layer, cur, cur_s, layer.reverse)
        cur, cur_s = torch.from_numpy(he), None
    d = np.abs(full.cpu().numpy().astype(np.int32) - cur.numpy().astype(np.int32))
    assert d.max() <= 2 and (d > 1).mean() < 1e-3 and (d != 0).mean() < 2e-2


def test_stack_entry_point_equals_layer_by_layer(flib):
    """fluke_factored_lstm_stack_i8_gpu (one C call per pass) gives the bytes and the final state
    of the layer-by-layer loop; 4 layers (even count: the first layer writes the scratch buffer)
    and a single layer (no scratch buffer needed)."""
    T, B, H, R = 6, 200, 768, 128
    g = torch.Generator().manual_seed(5)
    x, xs = prep.quantize_int8_rows(torch.randn(T * B, H, generator=g))
    X, XS = x.view(T, B, H).to(DEV), xs.to(DEV)
    for n_layers in (4, 1, 3):
        layers = [FactoredLstmLayer.random(H, R, bool(i % 2), g, DEV) for i in range(n_layers)]
        want, state = run_stack(layers, X, XS)
        got, (c, h) = run_stack_c(layers, X, XS)
        assert torch.equal(got, want)
        for i in range(n_layers):
            assert torch.equal(c[i], state[i][0]) and torch.equal(h[i], state[i][1])
    assert flib.fluke_factored_lstm_stack_i8_gpu(None, 0, T, B, H, R, 0, 0, 0, 0, 0, 0, 0, 0) != 0  # bad arguments: refused


@pytest.mark.parametrize("mode", [0, 1, 2, 4])
def test_hidden_output_that_is_not_16_byte_aligned_is_refused(flib, mode):
    """No form launches for an h_out that its 16-byte stores could not write: the call returns an error,
    the buffer and the state stay as they are."""
    T, B, H, R = 2, 200, 768, 128
    layer, x, xs = _layer_case(T, B, H, R, 3, False)
    raw = torch.full((T * B * H + 16,), 5, dtype=torch.int8, device=DEV)
    c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    flib.fluke_set_lstm_persistent(mode)
    try:
        for off in (1, 4, 8):
            with pytest.raises(RuntimeError, match="misaligned"):
                ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                           layer.w_up, layer.bias, c, h, h_out=raw[off:off + T * B * H].view(T, B, H))
    finally:
        flib.fluke_set_lstm_persistent(1)
    assert bool((raw == 5).all()) and not c.any() and not h.any()


def test_persistent_and_per_step_layers_agree(flib):
    """Same layer through all three drivers: the only difference is the accumulation order of the two
    K halves, so codes differ by at most one, rarely. Also other hidden sizes (1024, 384 with an odd
    number of 128-byte K blocks, 512), batches that are not a multiple of the 128-row tile and one
    with more row tiles than one single-launch kernel holds."""
    for (T, B, H) in [(16, 300, 768), (6, 130, 1024), (5, 1024, 768), (4, 140, 384), (4, 70, 512), (3, 1100, 768)]:
        layer, x, xs = _layer_case(T, B, H, 128, 11 + B, False)
        outs = []
        for mode in (4, 2, 0):
            flib.fluke_set_lstm_persistent(mode)
            c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
            outs.append((ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh,
                                                    layer.dn_hh_scale, layer.w_up, layer.bias, c, h).clone(), c, h))
        flib.fluke_set_lstm_persistent(1)
        for other in (outs[1], outs[2]):
            d = (outs[0][0].int() - other[0].int()).abs()
            assert int(d.max()) <= 1 and float((d != 0).float().mean()) < 5e-3
            assert float((outs[0][1] - other[1]).abs().max()) < 1e-2
            assert torch.equal(outs[0][2], outs[0][0][-1]) and torch.equal(other[2], other[0][-1])
        he, ce, _ = _run_oracle_layer(layer, x, xs, False)
        d = np.abs(outs[0][0].cpu().numpy().astype(np.int32) - he.astype(np.int32))
        assert d.max() <= 1 and (d != 0).mean() < 5e-3


def test_cluster_form_runs_in_rounds_when_nothing_else_covers_the_shape(flib):
    """H = 192 is outside the L2-exchange form (H % 128) and 17 row tiles are more clusters than
    fit at once, so the cluster form runs them in rounds; a ragged last tile as well."""
    T, B, H, R = 4, 2100, 192, 128
    layer, x, xs = _layer_case(T, B, H, R, 5, True)
    c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    flib.fluke_set_lstm_persistent(4)
    ho = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                    layer.w_up, layer.bias, c, h, reverse=True)
    flib.fluke_set_lstm_persistent(1)
    assert flib.fluke_sm100_lstm_last_form() == 1
    he, ce, _ = _run_oracle_layer(layer, x, xs, True)
    d = np.abs(ho.cpu().numpy().astype(np.int32) - he.astype(np.int32))
    assert d.max() <= 1 and (d != 0).mean() < 5e-3
    assert np.abs(c.cpu().numpy() - ce).max() < 1e-2


def test_layer_config_size_properties(lstm_mode):
    """H = 768, R = 128, B = 1024 (T cut to 24): codes stay in [-127, 127], the first step of a
    zero state matches the single-step kernel on [0 | x_down], and the reversed layer on
    time-flipped input equals the flipped forward output."""
    T, B, H, R = 24, 1024, 768, 128
    layer, x, xs = _layer_case(T, B, H, R, 3, False)
    X, XS = x.to(DEV), xs.to(DEV)
    args = (layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up, layer.bias)
    c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    fwd = ops.factored_lstm_layer_i8(X, XS, *args, c, h, reverse=False).clone()
    form = L.load().fluke_sm100_lstm_last_form()
    assert form == LSTM_MODES[lstm_mode][1]
    assert int(fwd.min()) >= -127
    c2 = torch.zeros(B, H, device=DEV); h2 = torch.zeros(B, H, dtype=torch.int8, device=DEV)
    rev = ops.factored_lstm_layer_i8(X.flip(0).contiguous(), XS.view(T, B).flip(0).contiguous().view(-1), *args, c2, h2, reverse=True)
    assert torch.equal(rev.flip(0), fwd) and torch.equal(c, c2)
    xd = ops.down_proj_i8(X[0], layer.dn_ih, XS[:B].contiguous(), layer.dn_ih_scale)
    A = torch.cat([torch.zeros(B, R, dtype=torch.float16, device=DEV), xd], dim=1).contiguous()
    c3 = torch.zeros(B, H, device=DEV)
    h3 = ops.factored_lstm_step_i8(A, layer.w_up, layer.bias, c3)
    d = (h3.int() - fwd[0].int()).abs()   # the persistent kernel uses the fast-exp tanh: rare one-code ties
    assert int(d.max()) <= 1 and float((d != 0).float().mean()) < 1e-3
    if lstm_mode == "per_step":
        assert torch.equal(h3, fwd[0])


def test_two_batches_side_by_side_config_size(flib):
    """Two benchmark-size batches (2 x 1024 chunks, H = 768, R = 128; T cut to 24) in one layer
    call, which the wide L2-exchange configuration runs in a single launch of 16 row tiles, give
    the bytes of the two batches run on their own (narrow configuration, 8 row tiles each)."""
    T, B, H, R = 24, 1024, 768, 128
    flib.fluke_set_lstm_persistent(2)
    layer, x, xs = _layer_case(T, 2 * B, H, R, 9, True)
    X, XS = x.to(DEV), xs.to(DEV)
    args = (layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up, layer.bias)
    c = torch.zeros(2 * B, H, device=DEV); h = torch.zeros(2 * B, H, dtype=torch.int8, device=DEV)
    both = ops.factored_lstm_layer_i8(X, XS, *args, c, h, reverse=True).clone()
    assert flib.fluke_sm100_lstm_last_form() == 2
    for j in range(2):
        xj = X[:, j * B:(j + 1) * B].contiguous()
        xsj = XS.view(T, 2 * B)[:, j * B:(j + 1) * B].contiguous().view(-1)
        cj = torch.zeros(B, H, device=DEV); hj = torch.zeros(B, H, dtype=torch.int8, device=DEV)
        one = ops.factored_lstm_layer_i8(xj, xsj, *args, cj, hj, reverse=True)
        assert torch.equal(one, both[:, j * B:(j + 1) * B])
        assert torch.equal(cj, c[j * B:(j + 1) * B]) and torch.equal(hj, h[j * B:(j + 1) * B])
    flib.fluke_set_lstm_persistent(1)


@pytest.mark.parametrize("passes_per_launch,time_chunks", [(1, 1), (2, 1), (2, 3), (1, 4)])
def test_streaming_pipeline_equals_pass_by_pass(passes_per_launch, time_chunks):
    """Five passes with different inputs through the three-stream driver (copy-in, layers,
    copy-out overlapped across groups of passes) give the bytes of run_stack on each input alone;
    with two passes per launch the fifth is a group of its own that `drain` runs; with time chunks
    the first and the last layer run block by block between their copies."""
    T, B, H, R, NL = 6, 200, 768, 128, 3
    g = torch.Generator().manual_seed(77)
    layers = [FactoredLstmLayer.random(H, R, bool(i % 2), g, DEV) for i in range(NL)]
    pipe = StackPipeline(layers, T, B, DEV, passes_per_launch=passes_per_launch, time_chunks=time_chunks)
    ins, outs = [], []
    for k in range(5):
        x, xs = prep.quantize_int8_rows(torch.randn(T * B, H, generator=g))
        ins.append((x.view(T, B, H).contiguous().pin_memory(), xs.contiguous().pin_memory()))
        outs.append(torch.empty(T, B, H, dtype=torch.int8).pin_memory())
    for k in range(5):
        pipe.submit(ins[k][0], ins[k][1], outs[k])
    pipe.drain()
    torch.cuda.synchronize()
    for k in range(5):
        ref, _ = run_stack(layers, ins[k][0].to(DEV), ins[k][1].to(DEV))
        assert torch.equal(outs[k], ref.cpu())


def test_streaming_pipeline_launches_full_groups_and_flush_launches_a_partial_one():
    """With two passes per launch, `submit` of a lone pass only queues it (its output buffer stays
    untouched however long one waits); `flush` launches it without blocking, and the bytes are
    those of the pass alone."""
    T, B, H, R, NL = 4, 130, 768, 128, 2
    g = torch.Generator().manual_seed(78)
    layers = [FactoredLstmLayer.random(H, R, bool(i % 2), g, DEV) for i in range(NL)]
    pipe = StackPipeline(layers, T, B, DEV, passes_per_launch=2, time_chunks=2)
    x, xs = prep.quantize_int8_rows(torch.randn(T * B, H, generator=g))
    x, xs = x.view(T, B, H).contiguous().pin_memory(), xs.contiguous().pin_memory()
    out = torch.full((T, B, H), 77, dtype=torch.int8).pin_memory()
    pipe.submit(x, xs, out)
    torch.cuda.synchronize()
    assert bool((out == 77).all())          # nothing was launched
    pipe.flush()
    pipe.drain()
    ref, _ = run_stack(layers, x.to(DEV), xs.to(DEV))
    assert torch.equal(out, ref.cpu())
    pipe.close()


def test_wide_l2_configuration_matches_the_narrow_one(flib):
    """The L2-exchange form with 48 units per gate CTA and one worker per row tile (chosen by itself
    when a layer has more row tiles than a narrow launch holds) computes every element in the same
    order as the narrow configuration: identical bytes. Shapes: ragged tiles, H = 384, and a batch
    of 2100 chunks (17 row tiles: one full wide launch and a second one)."""
    for (T, B, H) in [(6, 300, 768), (5, 130, 384), (3, 2100, 768), (4, 1, 768)]:
        layer, x, xs = _layer_case(T, B, H, 128, 3 + B, False)
        res = []
        for wide in (0, 1, -1):
            flib.fluke_set_lstm_persistent(2)
            flib.fluke_sm100_set_lstm_wide(wide)
            c = torch.zeros(B, H, device=DEV); h = torch.zeros(B, H, dtype=torch.int8, device=DEV)
            out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh,
                                             layer.dn_hh_scale, layer.w_up, layer.bias, c, h)
            assert flib.fluke_sm100_lstm_last_form() == 2
            res.append((out.clone(), c.clone(), h.clone()))
        flib.fluke_sm100_set_lstm_wide(-1)
        flib.fluke_set_lstm_persistent(1)
        for other in res[1:]:
            assert torch.equal(res[0][0], other[0]) and torch.equal(res[0][1], other[1]) and torch.equal(res[0][2], other[2])
        he, ce, _ = _run_oracle_layer(layer, x, xs, False)
        d = np.abs(res[1][0].cpu().numpy().astype(np.int32) - he.astype(np.int32))
        assert d.max() <= 1 and (d != 0).mean() < 5e-3


@pytest.mark.parametrize("H,B", [(768, 1), (768, 45), (768, 352), (768, 353), (768, 506), (768, 507), (768, 704), (768, 705),
                                 (768, 858), (768, 859), (768, 1056), (768, 1057), (256, 300), (256, 2900), (384, 47), (384, 1600),
                                 (384, 2048), (512, 1000), (512, 1600), (640, 90), (640, 1200), (896, 500), (896, 800), (1024, 33),
                                 (1024, 470), (1024, 481)])
@pytest.mark.parametrize("T", [1, 2, 3, 4])
def test_small_cluster_form_gives_the_bytes_of_the_l2_form(flib, H, B, T):
    """The default form (few chunk rows per cluster, operands swapped) against the L2-exchange form,
    which shares none of its data movement: same arithmetic in the same order, so equal bytes from a
    non-zero state. Batches around the row counts per cluster where the kernel's column count (16, 32, 48),
    the number of groups or the number of waves changes on a B200, one row, ragged last clusters (an
    empty second group among them), every cluster size from 2 to 8 CTAs; one step (no barrier is armed again, the
    final state leaves at once) to four."""
    R = 128
    layer, x, xs = _layer_case(T, B, H, R, H + B, B % 2 == 1)
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                         layer.w_up, layer.bias, c, h, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    for got, want in zip(*res):
        assert torch.equal(got, want)


@pytest.mark.parametrize("H,B", [(256, 1), (256, 528), (256, 529), (384, 3), (384, 391), (384, 393), (512, 287), (512, 290), (640, 175), (640, 185),
                                 (768, 2), (768, 44), (768, 175), (768, 176), (768, 177), (768, 1023), (896, 143), (896, 145), (1024, 5),
                                 (1024, 144), (1024, 145), (1024, 577), (1024, 863)])
@pytest.mark.parametrize("T", [1, 2, 5, 10])
def test_small_cluster_form_of_few_rows_and_of_two_groups_gives_the_bytes_of_the_l2_form(flib, H, B, T):
    """As above, at the row counts per cluster where the form that contracts the x rows of two steps at once ends (8 on a B200),
    its ring of five slots (steps 4, 5 and 8, 9 reuse them), and one wave of 33 to 48 rows at H = 1024. Exact."""
    layer, x, xs = _layer_case(T, B, H, 128, H + B, B % 2 == 1)
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                         layer.w_up, layer.bias, c, h, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    for got, want in zip(*res):
        assert torch.equal(got, want)


@pytest.mark.parametrize("H,B", [(768, 44), (768, 150), (768, 300), (768, 700), (768, 727), (768, 1000), (1024, 100), (1024, 700), (256, 400)])
def test_infinite_gate_weights_reach_their_own_unit_and_row_only(flib, H, B):
    """An infinite weight makes a pre-activation infinite, so the gate saturates (NaN only where the row's own factor is zero or
    two infinities meet), whatever the other rows of the cluster are. Every number of rows per cluster from which the small-cluster
    form has another kernel (727: nothing in the last cluster's second group), weights of all four gates and both halves, against the L2-exchange form, which multiplies
    every weight by the row's own values alone: the same bytes, NaN at the same places."""
    T, R = 7, 128
    layer, x, xs = _layer_case(T, B, H, R, H + B, False)
    w = layer.w_up.clone()
    for i, (unit, k) in enumerate([(3, 5), (40, 127), (H - 1, 64), (129, 0), (70, 130), (H - 100, 255)]):
        w[(i % 4) * H + unit, k] = float("inf") if i % 2 else float("-inf")
    w[2 * H + 17, 33] = 65504.0
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, w, layer.bias, c, h)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    (out, c, h), (out_l2, c_l2, h_l2) = res
    assert torch.equal(torch.isnan(c), torch.isnan(c_l2)) and not torch.isnan(c).all(0).all()
    assert torch.equal(c.nan_to_num(7.0), c_l2.nan_to_num(7.0)) and torch.equal(out, out_l2) and torch.equal(h, h_l2)


@pytest.mark.parametrize("H,B", [(256, 600), (384, 32), (768, 44), (768, 300), (896, 144), (1024, 30), (1024, 200)])
def test_one_timestep_per_call_gives_the_bytes_of_one_call(flib, H, B):
    """A caller's own time loop over calls of one timestep, state carried over in place: the final hidden codes of a call are stored
    where the cluster's CTAs load the initial ones of all units from. Rows per cluster where they do. Exact."""
    T = 48
    layer, x, xs = _layer_case(T, B, H, 128, H + B, False)
    x, xs = x.to(DEV), xs.to(DEV)
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    args = (layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up, layer.bias)
    c, h = c0.clone(), h0.clone()
    want = ops.factored_lstm_layer_i8(x, xs, *args, c, h)
    assert flib.fluke_sm100_lstm_last_form() == 3
    c1, h1 = c0.clone(), h0.clone()
    got = torch.cat([ops.factored_lstm_layer_i8(x[t:t + 1], xs.view(T, B)[t], *args, c1, h1) for t in range(T)])
    assert torch.equal(got, want) and torch.equal(c1, c) and torch.equal(h1, h)


@pytest.mark.parametrize("H,B", [(256, 3), (256, 64), (256, 527), (256, 528), (384, 32), (384, 130), (384, 343), (384, 344), (384, 345)])
@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8, 9, 17])
@pytest.mark.parametrize("infinite", [False, True])
def test_four_steps_per_contraction_give_the_bytes_of_the_l2_form(flib, H, B, T, infinite):
    """Clusters of two and three with up to 8 rows each (528 and 344 chunks on a B200) contract the x rows of four steps at once, from a
    ring of eight slots: fewer steps than that, the ring's wrap, both directions, ragged last clusters; and weights that are not finite, for
    which every step contracts its own. Against the L2-exchange form. Exact."""
    layer, x, xs = _layer_case(T, B, H, 128, H + B + T, T % 2 == 1)
    w = layer.w_up.clone()
    if infinite:
        for i, (unit, k) in enumerate([(3, 5), (40, 127), (H - 1, 64), (129, 0), (70, 130), (H - 100, 255)]):
            w[(i % 4) * H + unit, k] = float("inf") if i % 2 else float("-inf")
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, w, layer.bias,
                                         c, h, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    for got, want in zip(*res):
        if got.is_floating_point():
            assert torch.equal(torch.isnan(got), torch.isnan(want))
            got, want = got.nan_to_num(7.0), want.nan_to_num(7.0)
        assert torch.equal(got, want)


@pytest.mark.parametrize("H,B", [(256, 1057), (256, 2112), (384, 689), (384, 1376), (512, 513), (512, 1024), (640, 443), (640, 832), (768, 353), (768, 704),
                                 (896, 289), (896, 544), (1024, 300), (256, 1056), (384, 345), (384, 688), (512, 257), (512, 512)])
@pytest.mark.parametrize("T", [1, 2, 3, 6, 7])
def test_two_steps_per_contraction_of_more_than_eight_rows_give_the_bytes_of_the_l2_form(flib, H, B, T):
    """17 to 32 rows per cluster on a B200 (clusters of up to seven) and 9 to 16 (up to four), the fewest and the most: two steps' x rows per contraction, windows that
    begin before the first step and end behind the last, both parities and directions; pieces that stay in a CTA. Against the L2-exchange form. Exact."""
    layer, x, xs = _layer_case(T, B, H, 128, H + B + T, T % 2 == 0)
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-128, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                         layer.w_up, layer.bias, c, h, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    for got, want in zip(*res):
        assert torch.equal(got, want)


@pytest.mark.parametrize("B", [120, 121, 127, 135, 136, 151, 166, 180, 181, 211, 226, 240, 241])
@pytest.mark.parametrize("T", [1, 2, 3, 9])
def test_rows_projected_by_pair_give_the_bytes_of_the_l2_form(flib, B, T):
    """H = 1024, around and within the 9 to 16 rows per cluster (15 clusters on a B200) that are projected by pairs of CTAs: one to four rows
    per pair, pairs and quarters without rows in the last cluster. Against the L2-exchange form. Exact."""
    H = 1024
    layer, x, xs = _layer_case(T, B, H, 128, B + T, B % 2 == 1)
    g = torch.Generator().manual_seed(B)
    c0 = (torch.randn(B, H, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (B, H), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, h = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale,
                                         layer.w_up, layer.bias, c, h, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, h))
    flib.fluke_set_lstm_persistent(1)
    for got, want in zip(*res):
        assert torch.equal(got, want)


@pytest.mark.parametrize("h", [1088, 1152, 1280, 2048])
@pytest.mark.parametrize("b", [16, 3000])
def test_layers_of_more_than_1024_units_are_refused_without_a_launch(flib, h, b):
    """The down-projection's contraction is limited to 1024; a layer beyond it is refused by the library's own check whichever kernel
    its number of rows would take, also during a stream capture, which goes on."""
    t = 2
    layer = FactoredLstmLayer.random(h, 128, False, torch.Generator().manual_seed(h), DEV)
    x = torch.zeros(t, b, h, dtype=torch.int8, device=DEV)
    c, hs = torch.ones(b, h, device=DEV), torch.ones(b, h, dtype=torch.int8, device=DEV)
    out = torch.full_like(x, 5)
    ws = torch.empty(flib.fluke_factored_lstm_layer_workspace(t, b, h, 128), dtype=torch.uint8, device=DEV)

    def layer_is_refused():
        with pytest.raises(RuntimeError):
            ops.factored_lstm_layer_i8(x, None, layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up,
                                       layer.bias, c, hs, h_out=out, workspace=ws)

    layer_is_refused()
    y = torch.randn(40, 512, device=DEV).half()
    want = ops.silu_mul(y)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        ops.set_stream(stream)
        try:
            layer_is_refused()
            got = ops.silu_mul(y)
        finally:
            ops.set_stream(None)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert bool((c == 1).all()) and bool((hs == 1).all()) and bool((out == 5).all())


def _small_clusters(flib, t, b, h):
    """(chunk rows per cluster, steps whose x rows one contraction covers) of the small-cluster form on this device."""
    steps = ctypes.c_int(0)
    return flib.fluke_sm100_lstm_small_clusters(t, b, h, ctypes.byref(steps)), steps.value


def _chunk_counts(flib, h, rows):
    """So many rows in every cluster that the device runs at once, and as few as the last one can have beside them."""
    per_cluster = lambda b: _small_clusters(flib, 1, b, h)[0]
    clusters = next(n for n in range(1, 256) if per_cluster(48 * n) == 48 and per_cluster(48 * n + 1) < 48)
    return clusters * rows, clusters * rows - min(rows, clusters) + 1


def _assert_default_form_gives_the_bytes_of_the_l2_form(flib, t, b, h, infinite):
    """Of both directions' layers from a non-zero state; infinite: weights of all gates and both halves, as above. Exact, NaN at the same places."""
    layer, x, xs = _layer_case(t, b, h, 128, h + b + t, (t + b) % 2 == 1)
    w = layer.w_up.clone()
    if infinite:
        for i, (unit, k) in enumerate([(3, 5), (40, 127), (h - 1, 64), (129, 0), (70, 130), (h - 100, 255)]):
            w[(i % 4) * h + unit, k] = float("inf") if i % 2 else float("-inf")
    g = torch.Generator().manual_seed(b)
    c0 = (torch.randn(b, h, generator=g) * 0.3).to(DEV)
    h0 = torch.randint(-127, 128, (b, h), generator=g, dtype=torch.int8).to(DEV)
    res = []
    for mode, form in ((1, 3), (2, 2)):
        flib.fluke_set_lstm_persistent(mode)
        c, hs = c0.clone(), h0.clone()
        out = ops.factored_lstm_layer_i8(x.to(DEV), xs.to(DEV), layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, w, layer.bias,
                                         c, hs, reverse=layer.reverse)
        assert flib.fluke_sm100_lstm_last_form() == form
        res.append((out, c, hs))
    (out, c, hs), (out_l2, c_l2, hs_l2) = res
    assert torch.equal(torch.isnan(c), torch.isnan(c_l2)) and torch.equal(c.nan_to_num(7.0), c_l2.nan_to_num(7.0))
    assert torch.equal(out, out_l2) and torch.equal(hs, hs_l2)


@pytest.mark.parametrize("h,rows,steps", [(256, 8, 4), (384, 6, 4), (512, 8, 2), (256, 9, 2), (256, 16, 2), (384, 14, 2), (512, 12, 2), (640, 16, 1), (1024, 16, 1),
                                          (256, 17, 2), (512, 32, 2), (896, 24, 2), (1024, 32, 1), (768, 33, 1)])
@pytest.mark.parametrize("infinite", [False, True])
def test_every_kernel_of_the_small_clusters_gives_the_bytes_of_the_l2_form(flib, h, rows, steps, infinite):
    """Rows per cluster on this device, and the steps per contraction of the kernel they take, are asked for and asserted. All clusters full, and the
    last one short of rows; also weights that are not finite in windows of two steps of more than 8 rows."""
    t = 18
    for b in _chunk_counts(flib, h, rows):
        assert _small_clusters(flib, t, b, h) == (rows, steps)
        _assert_default_form_gives_the_bytes_of_the_l2_form(flib, t, b, h, infinite)


@pytest.mark.parametrize("h,rows", [(256, 33), (384, 40), (512, 47), (640, 33), (768, 47), (896, 36), (1024, 33), (1024, 48)])
@pytest.mark.parametrize("t", [1, 2, 3])
def test_infinite_gate_weights_in_layers_of_few_steps(flib, h, rows, t):
    """Two groups of 24 rows, whose MMAs for such weights are others: one step (no barrier is armed again) to three; an empty second group in the last cluster."""
    for b in _chunk_counts(flib, h, rows):
        assert _small_clusters(flib, t, b, h) == (rows, 1)
        _assert_default_form_gives_the_bytes_of_the_l2_form(flib, t, b, h, True)


@pytest.mark.parametrize("h,rows,few,enough", [(256, 8, 7, 8), (384, 6, 7, 8), (384, 7, 18, None), (256, 16, 15, 16), (384, 14, 15, 16), (384, 15, 18, None), (512, 12, 15, 16),
                                               (512, 13, 18, None), (256, 17, 7, 8), (640, 32, 7, 8), (896, 32, 15, 16)])
def test_layers_of_few_steps_take_the_kernel_of_fewer_steps_per_contraction(flib, h, rows, few, enough):
    """On either side of the numbers of timesteps (and of rows: None) from which a contraction covers more of them. Exact."""
    b = _chunk_counts(flib, h, rows)[1]
    fewest = 2 if rows <= 8 else 1
    for t in range(max(1, few - 1), few + 1):
        assert _small_clusters(flib, t, b, h) == (rows, fewest)
        _assert_default_form_gives_the_bytes_of_the_l2_form(flib, t, b, h, False)
    if enough:
        assert _small_clusters(flib, enough, b, h) == (rows, 2 * fewest)
        _assert_default_form_gives_the_bytes_of_the_l2_form(flib, enough, b, h, False)


def test_a_short_layer_is_captured_after_a_long_one_has_run(flib):
    """The kernel of a layer of few steps is another one than that of a longer layer; it is configured with it, in front of the capture."""
    h, rows, t = 640, 20, 9
    b = _chunk_counts(flib, h, rows)[0]
    assert _small_clusters(flib, t, b, h)[1] != _small_clusters(flib, 3, b, h)[1]
    layer, x, xs = _layer_case(t, b, h, 128, 5, False)
    x, xs = x.to(DEV), xs.to(DEV)
    args = (layer.dn_ih, layer.dn_ih_scale, layer.dn_hh, layer.dn_hh_scale, layer.w_up, layer.bias)
    state = lambda: (torch.zeros(b, h, device=DEV), torch.zeros(b, h, dtype=torch.int8, device=DEV))
    ws = torch.empty(flib.fluke_factored_lstm_layer_workspace(t, b, h, 128), dtype=torch.uint8, device=DEV)
    ops.factored_lstm_layer_i8(x, xs, *args, *state(), workspace=ws)
    c, hs = state()
    out = torch.empty(3, b, h, dtype=torch.int8, device=DEV)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        ops.set_stream(stream)
        try:
            ops.factored_lstm_layer_i8(x[:3], xs[:3 * b], *args, c, hs, h_out=out, workspace=ws)
        finally:
            ops.set_stream(None)
    graph.replay()
    torch.cuda.synchronize()
    c2, hs2 = state()
    want = ops.factored_lstm_layer_i8(x[:3], xs[:3 * b], *args, c2, hs2)
    assert torch.equal(out, want) and torch.equal(c, c2) and torch.equal(hs, hs2)
