"""Learned proposal on the GPU: network kernels against the FP64 oracle, the plane sweep and the proposal-gated run
start bit for bit against the CPU oracle, the random-init fallback, the propose pipeline and training.

Tolerances: the sweep and every PatchStereo run are integer-exact (zero tolerance, parity build).  The network runs in
BF16 with FP32 accumulation: a single convolution is compared with FP64 at 1e-5 of the output's max magnitude (1e-4
for the weight gradient, a sum over all pixels); whole-network gradients against an oracle that rounds to bf16 where
the GPU stores bf16, at 10 % relative L2 and cosine 0.995 per layer (the bf16 noise floor; see the test).
"""
import numpy as np
import pytest
import torch

from oracle import cnn_oracle as O
from oracle import oracle
from cumulus3d_b200 import _lib, proposal, scenes
from cumulus3d_b200.patchstereo import PatchMatchBackend, RunParams, ViewState

pytestmark = pytest.mark.gpu


def _bf16(rng, shape, lo=-1.0, hi=1.0):
    return O.bf16_bits(rng.uniform(lo, hi, shape))


@pytest.mark.parametrize("path", ["tcgen05", "mma"])
@pytest.mark.parametrize("shape", [(2, 9, 13, 48, 32), (1, 8, 8, 32, 8), (1, 12, 20, 224, 96), (3, 5, 7, 16, 64),
                                   (1, 4, 300, 128, 128)])
def test_conv_kernels_match_fp64(shape, path):
    """Forward (tcgen05 for cout in {32, 64, 96, 128}, else mma.sync; or mma.sync only), data and weight gradients."""
    proposal.set_conv_path(path)
    proposal.conv_timeouts(reset=True)
    b, h, w, ci, co = shape
    rng = np.random.default_rng(sum(shape))
    x = _bf16(rng, (b, h, w, ci))
    dy = _bf16(rng, (b, h, w, co))
    wt = rng.uniform(-0.3, 0.3, (co, 9, ci)).astype(np.float32)
    y, dx, dw = proposal.conv_check(x, wt, dy)
    xf, dyf, wf = O.from_bf16_bits(x), O.from_bf16_bits(dy), O.bf16_round(wt)
    y_ref = O.conv(xf, wf)
    dx_ref, dw_ref, _ = O.conv_grads(xf, wf, dyf)
    assert np.abs(y - y_ref).max() <= 1e-5 * np.abs(y_ref).max()
    assert np.abs(dx - dx_ref).max() <= 1e-5 * np.abs(dx_ref).max()
    assert np.abs(dw - dw_ref).max() <= 1e-4 * np.abs(dw_ref).max()
    assert proposal.conv_timeouts() == 0
    proposal.set_conv_path("auto")


@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 8), (2, 8, 16, 32, 64), (1, 9, 17, 40, 24), (3, 25, 33, 96, 48),
                                   (1, 70, 130, 56, 128), (5, 3, 40, 224, 16)])
def test_weight_gradient_tiles_match_fp64(shape):
    """The weight gradient at the edges of its 8 x 16 pixel tiles, 32 input and 16/32/48/64 output channel blocks, with
    one tile and with several per CTA.  Products of bf16 are exact in binary32; each of the P additions rounds once, so
    the error is at most P * 2^-24 of the sum of magnitudes (twice that is allowed)."""
    b, h, w, ci, co = shape
    rng = np.random.default_rng(7 + sum(shape))
    x, dy = _bf16(rng, (b, h, w, ci)), _bf16(rng, (b, h, w, co))
    _, _, dw = proposal.conv_check(x, np.zeros((co, 9, ci), np.float32), dy)
    xf, dyf = O.from_bf16_bits(x), O.from_bf16_bits(dy)
    _, ref, _ = O.conv_grads(xf, np.zeros((co, 9, ci)), dyf)
    _, mag, _ = O.conv_grads(np.abs(xf), np.zeros((co, 9, ci)), np.abs(dyf))
    assert (np.abs(dw - ref) <= b * h * w * 2.0 ** -23 * mag + 1e-30).all()


@pytest.mark.parametrize("shape", [(1, 1, 1, 8, 8), (2, 8, 16, 32, 64), (1, 9, 17, 40, 24), (3, 25, 33, 96, 48),
                                   (1, 70, 130, 56, 128), (5, 3, 40, 224, 16), (2, 64, 129, 32, 16)])
def test_weight_gradient_counts_every_pixel_once(shape):
    """Inputs and gradients in {-1, 0, 1}: every product and partial sum is a whole number below 2^24, exact in binary32
    in any order, so a pixel left out or taken twice anywhere shows, whatever the number of pixels."""
    b, h, w, ci, co = shape
    rng = np.random.default_rng(70 + sum(shape))
    x, dy = (rng.integers(-1, 2, (b, h, w, c)).astype(np.float32) for c in (ci, co))
    _, _, dw = proposal.conv_check(O.bf16_bits(x), np.zeros((co, 9, ci), np.float32), O.bf16_bits(dy))
    _, ref, _ = O.conv_grads(x, np.zeros((co, 9, ci)), dy)
    np.testing.assert_array_equal(dw, ref)


def _labels(rng, b, h, w, dr=(25.0, 60.0)):
    lab = np.zeros((b, h, w, 6), np.float32)
    lab[..., 0] = rng.uniform(0, 1, (b, h, w))
    n = rng.normal(size=(b, h, w, 3))
    lab[..., 1:4] = n / np.linalg.norm(n, axis=-1, keepdims=True)
    lab[..., 4] = rng.random((b, h, w)) < 0.8
    d = 1.0 / (1.0 / dr[1] + lab[..., 0] * (1.0 / dr[0] - 1.0 / dr[1]))
    lab[..., 5] = d * (1 + rng.normal(0, 0.01, (b, h, w)))
    lab[lab[..., 4] == 0] = 0
    return lab


def test_network_gradients_match_fp64_oracle():
    rng = np.random.default_rng(7)
    b, h, w = 2, 16, 24
    dr = (25.0, 60.0)
    xb = O.bf16_bits(np.concatenate([rng.uniform(0, 1, (b, h, w, 33)), np.zeros((b, h, w, 15))], axis=-1))
    net = proposal.ProposalNet(0, seed=3)
    params = net.get_params()
    a = O.forward(O.split(params), O.from_bf16_bits(xb), bf16=True)
    # labels: the confidence target |d - d*| < 1 % d* is a step function of the network output; d* is placed 0.3 %
    # or 3 % away from the oracle's depth so that FP32-vs-FP64 differences of the output cannot flip it
    lab = _labels(rng, b, h, w, dr)
    t = 1 / (1 + np.exp(-a["o"][..., 0]))
    d = 1 / (1 / dr[1] + t * (1 / dr[0] - 1 / dr[1]))
    lab[..., 5] = np.where(lab[..., 4] > 0, d * np.where(rng.random((b, h, w)) < 0.5, 1.003, 1.03), 0.0)
    x_t = torch.from_numpy(xb.view(np.int16)).cuda()
    lab_t = torch.from_numpy(lab).cuda()
    loss, g = net.train_step(x_t, lab_t, dr, lr=0.0, grads=True)
    out = torch.empty((b, h, w, 8), dtype=torch.float32, device="cuda")
    net.forward(x_t, out)
    torch.cuda.synchronize()
    fwd = float(np.abs(out.cpu().numpy() - a["o"]).max() / np.abs(a["o"]).max())
    loss_ref, g_o = O.loss_and_grad(a["o"], lab.astype(np.float64), dr)
    g_ref = O.backward(O.split(params), a, g_o, bf16=True)
    rels, coss, o = {}, {}, 0
    for (ci, co), name in zip(proposal.LAYERS, proposal.LAYER_NAMES):
        n = co * 9 * ci + co
        gg, rr = g[o:o + n], g_ref[o:o + n]
        rels[name] = float(np.linalg.norm(gg - rr) / max(np.linalg.norm(rr), 1e-30))
        coss[name] = float(gg @ rr / max(np.linalg.norm(gg) * np.linalg.norm(rr), 1e-30))
        o += n
    cos = float(g @ g_ref / (np.linalg.norm(g) * np.linalg.norm(g_ref)))
    report = {"forward": fwd, "loss": (loss, loss_ref), "cos": cos, "rel": rels, "layer_cos": coss}
    print(report)
    net.close()
    # Bounds from the bf16 noise floor: an activation stored in bf16 flips by one ulp wherever FP32 and FP64
    # accumulation straddle a rounding boundary, which is frequent for outputs that cancel to small values.  On this
    # network the oracle's own bf16-vs-FP64 gradients differ by 8-17 % per layer (cosine 0.9995); a wrong kernel
    # (tap order, transposition, missing term) gives a layer cosine far below 0.99.
    assert fwd < 1e-2, report
    assert abs(loss - loss_ref) <= 1e-3 * abs(loss_ref), report
    assert max(rels.values()) < 0.1, report
    assert min(coss.values()) > 0.995, report
    assert cos > 0.999, report


@pytest.mark.parametrize("wr,size,tuning", [(3, (64, 48), 0), (6, (80, 64), 0), (6, (80, 64), 6), (3, (64, 48), 2)])
def test_sweep_bitwise_vs_oracle(wr, size, tuning):
    """The sweep kernel of the windows 13x13 and the one for any other window (radius 3), under the default tuning word and
    under two words that select the same gathers."""
    wl = scenes.workload_small(size[0], size[1], views=3, window_radius=wr, seed=11)
    be = PatchMatchBackend(0, math="parity", tuning=tuning)
    w, h = size
    with be.begin(wl.input) as s:
        for v in range(3):
            buf = torch.zeros((h, w, 48), dtype=torch.int16, device="cuda")
            torch.cuda.synchronize()  # the session stream does not wait for torch's stream
            s.sweep_volume(0, v, buf.data_ptr(), w)
            s.synchronize()
            got = buf.cpu().numpy().view(np.uint16)
            want = oracle.sweep(wl.input, 0, v)
            np.testing.assert_array_equal(got, want)
    be.close()


def _proposals(wl, seed, keep=0.5):
    rng = np.random.default_rng(seed)
    out = []
    for v, cam in enumerate(wl.cams):
        p = np.zeros((cam.height, cam.width, 4), np.float32)
        n = wl.gt_normal[v].astype(np.float32)
        fx, fy, cx, cy = cam.k
        ys, xs = np.mgrid[0:cam.height, 0:cam.width]
        ray = np.stack([(xs - cx) / fx, (ys - cy) / fy, np.ones_like(xs, dtype=np.float64)], -1)
        n = np.where(((n * ray).sum(-1) > 0)[..., None], -n, n)  # facing the camera
        p[..., :3] = n
        p[..., 3] = wl.gt_depth[v] * (1 + rng.normal(0, 0.003, wl.gt_depth[v].shape))
        p[rng.random((cam.height, cam.width)) > keep] = 0.0
        out.append(p)
    return out


def test_proposal_init_bitwise_vs_oracle():
    wl = scenes.workload_small(96, 64, views=3, window_radius=3, seed=5)
    props = _proposals(wl, 1)
    views = [0, 1, 2]
    be = PatchMatchBackend(0, math="parity")
    st = [ViewState.new(c.width, c.height) for c in wl.cams]
    with be.begin(wl.input) as s:
        s.proposal_upload(0, views, props)
        s.run(views, st, RunParams(0, False, _lib.PS_INIT_PROPOSAL, 2, 1))
    be.close()
    ref = [ViewState.new(c.width, c.height) for c in wl.cams]
    oracle.run(wl.input, views, ref, RunParams(0, False, _lib.PS_INIT_PROPOSAL, 2, 1), proposals=props)
    for a, b in zip(st, ref):
        np.testing.assert_array_equal(a.depth, b.depth)
        np.testing.assert_array_equal(a.normal, b.normal)
        np.testing.assert_array_equal(a.cost, b.cost)


def test_empty_proposal_falls_back_to_random_init_bitwise():
    """Where no plane is proposed the run start draws exactly the plain random hypothesis."""
    wl = scenes.workload_small(96, 64, views=3, window_radius=3, seed=6)
    views = [0, 1, 2]
    empty = [np.zeros((c.height, c.width, 4), np.float32) for c in wl.cams]
    be = PatchMatchBackend(0, math="parity")
    a = [ViewState.new(c.width, c.height) for c in wl.cams]
    b = [ViewState.new(c.width, c.height) for c in wl.cams]
    with be.begin(wl.input) as s:
        s.run(views, a, RunParams(0, False, True, 2, 1))
        s.proposal_upload(0, views, empty)
        s.run(views, b, RunParams(0, False, _lib.PS_INIT_PROPOSAL, 2, 1))
        with pytest.raises(_lib.PsError):  # random_init beyond PS_INIT_PROPOSAL is rejected
            s.run_resident([0], RunParams(0, False, 3, 1, 1))
    be.close()
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x.depth, y.depth)
        np.testing.assert_array_equal(x.normal, y.normal)


def test_propose_pipeline_and_learned_run_vs_oracle():
    """ps_propose = sweep -> network -> decode (checked against the same steps done separately), and the schedule's
    learned run start from those proposals equals the oracle's run from the same proposals bit for bit."""
    wl = scenes.workload_small(100, 60, views=3, window_radius=3, seed=9)  # sizes not multiples of 8: padded input
    views = [0, 1, 2]
    net = proposal.ProposalNet(0, seed=5)
    be = PatchMatchBackend(0, math="parity")
    st = [ViewState.new(c.width, c.height) for c in wl.cams]
    with be.begin(wl.input) as s:
        n_all = s.propose(net, 0, views, conf_threshold=0.0)
        props = s.proposal_download(0, views)
        assert n_all == sum(int((p[..., 3] > 0).sum()) for p, _ in props)
        assert n_all > 0.5 * sum(c.width * c.height for c in wl.cams)
        # the same steps by hand for view 1: sweep into a padded buffer, forward, decode on the host
        w, h = wl.cams[1].width, wl.cams[1].height
        hp, wp = (h + 7) // 8 * 8, (w + 7) // 8 * 8
        xin = torch.zeros((1, hp, wp, 48), dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()  # the session stream does not wait for torch's stream
        s.sweep_volume(0, 1, xin.data_ptr(), wp)
        s.synchronize()
        out = torch.empty((1, hp, wp, 8), dtype=torch.float32, device="cuda")
        net.forward(xin, out)
        torch.cuda.synchronize()
        o = out.cpu().numpy()[0, :h, :w].astype(np.float64)
        conf = 1 / (1 + np.exp(-o[..., 4]))
        np.testing.assert_allclose(props[1][1], conf, rtol=0, atol=1e-5)
        t = 1 / (1 + np.exp(-o[..., 0]))
        d = 1 / (1 / 60.0 + t * (1 / 25.0 - 1 / 60.0))
        m = props[1][0][..., 3] > 0
        np.testing.assert_allclose(props[1][0][..., 3][m], d[m], rtol=1e-5)
        assert s.propose(net, 0, views, conf_threshold=1.0) == 0
        # learned schedule run start from the stored proposals (threshold 0.5)
        s.propose(net, 0, views, conf_threshold=0.5)
        props = [p for p, _ in s.proposal_download(0, views)]
        s.run(views, st, RunParams(0, False, _lib.PS_INIT_PROPOSAL, 1, 1))
    be.close()
    net.close()
    ref = [ViewState.new(c.width, c.height) for c in wl.cams]
    oracle.run(wl.input, views, ref, RunParams(0, False, _lib.PS_INIT_PROPOSAL, 1, 1), proposals=props)
    for a, b in zip(st, ref):
        np.testing.assert_array_equal(a.depth, b.depth)
        np.testing.assert_array_equal(a.normal, b.normal)


def test_training_reduces_loss():
    data = proposal.make_training_set(n_scenes=12, seed=500, crop=64, group=12, log=None)
    assert data.valid_fraction > 0.2
    net = proposal.ProposalNet(0, seed=2)
    losses = proposal.train(net, data, steps=60, batch=4, lr=1e-3, log=None)
    assert all(np.isfinite(losses))
    assert np.mean(losses[-5:]) < 0.85 * np.mean(losses[:5]), (losses[:5], losses[-5:])
    assert net.step == 60
    net.close()


@pytest.mark.parametrize("seed", [90000, 91000])
def test_learned_init_beats_random_init_on_held_out_scenes(seed):
    """The gain of the committed network: on held-out crop scenes (seeds far from the training set's 1000-1599),
    one photometric iteration from the learned proposal agrees with the converged plain result (6 iterations, within
    1 % depth, on the pixels that result trusts) on clearly more pixels than one iteration from random init.  Both
    start from the same seeded draws; the proposal replaces them where the network's confidence reaches
    CONF_THRESHOLD (0.15).  Measured on a B200 (seed 90000): 94.1 % vs 73.9 %, proposals on 97 % of the pixels."""
    net = proposal.ProposalNet(0, weights=proposal.DEFAULT_WEIGHTS)
    try:
        g = proposal.evaluate_gain(net, n_scenes=8, seed=seed, iters=1)
    finally:
        net.close()
    assert g["proposed_fraction"] > 0.5, g
    assert g["learned"] >= g["random"] + 0.08, g


def test_sweep_with_ground_normals_bitwise_vs_oracle():
    """A caller-set sweep normal (the world's up seen from each camera) reaches the kernel and matches the oracle."""
    wl = scenes.workload_small(64, 48, views=3, window_radius=3, seed=12)
    normals = scenes.up_normals(wl.cams)
    be = PatchMatchBackend(0, math="parity", tuning=6)
    with be.begin(wl.input) as s:
        s.set_sweep_normals(normals)
        buf = torch.zeros((48, 64, 48), dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        s.sweep_volume(0, 1, buf.data_ptr(), 64)
        s.synchronize()
        got = buf.cpu().numpy().view(np.uint16)
        with pytest.raises(_lib.PsError):  # a normal facing away from the camera is rejected
            s.set_sweep_normals(-normals)
    be.close()
    np.testing.assert_array_equal(got, oracle.sweep(wl.input, 0, 1, normal=normals[1]))
    assert not np.array_equal(got, oracle.sweep(wl.input, 0, 1))  # and differs from the fronto-parallel sweep


def test_tensor_core_wait_expiry_is_reported_and_recoverable():
    """The tcgen05 convolution's bounded waits: with commits withheld (test switch) the kernel returns, counts the
    expiry, and a blocking forward reports PS_ETIMEOUT; afterwards the same context computes correct results."""
    lib = _lib.engine()
    rng = np.random.default_rng(3)
    x = _bf16(rng, (1, 4, 40, 128))  # 4 input chunks: the stage-reuse wait runs
    dy = _bf16(rng, (1, 4, 40, 64))
    wt = rng.uniform(-0.3, 0.3, (64, 9, 128)).astype(np.float32)
    proposal.conv_timeouts(reset=True)
    assert lib.ps_net_test_stall_convolutions(0, 1) == _lib.PS_OK
    try:
        proposal.conv_check(x, wt, dy)  # returns (results invalid) instead of hanging
        assert proposal.conv_timeouts() > 0
        net = proposal.ProposalNet(0, seed=4)
        xin = torch.zeros((1, 16, 16, 48), dtype=torch.int16, device="cuda")
        out = torch.empty((1, 16, 16, 8), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        with pytest.raises(_lib.PsError) as e:
            net.forward(xin, out)
        assert e.value.code == _lib.PS_ETIMEOUT
        net.close()
    finally:
        assert lib.ps_net_test_stall_convolutions(0, 0) == _lib.PS_OK
        proposal.conv_timeouts(reset=True)
    y, _, _ = proposal.conv_check(x, wt, dy)
    y_ref = O.conv(O.from_bf16_bits(x), O.bf16_round(wt))
    assert np.abs(y - y_ref).max() <= 1e-5 * np.abs(y_ref).max()
    assert proposal.conv_timeouts() == 0
