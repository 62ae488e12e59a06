"""The learned support-point proposal on the GPU against its CPU oracle.

* the training kernels (fp32 forward, backward, correlation loss): loss and
  every gradient against the float64 oracle;
* the tcgen05 inference path: against the oracle's bf16 forward pass;
* the pooled features: bit-exact;
* the learned support sweep: given the GPU's bins, the candidate lattice is
  bit-exact with the oracle's restatement, and the settled / fallback
  counts agree;
* what the trained network gains over the plain sweep and over untrained
  weights on held-out pairs.
"""
import os

import numpy as np
import pytest

import elas_b200 as eb
import oracle
import proposal_oracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t

    return t


def test_training_gradients_match_oracle(torch):
    import proposal

    rng = np.random.default_rng(5)
    hd, wd, D = 6, 24, 63
    xL = po.bf16_round(rng.normal(0, 1, (hd, wd, po.CH)))
    xR = po.bf16_round(rng.normal(0, 1, (hd, wd, po.CH)))
    lab = np.stack([rng.integers(4, wd, 12), rng.integers(0, hd, 12), rng.integers(0, 16, 12)], axis=1)
    theta = po.init_params(7).astype(np.float64)
    theta[po.TAPS * po.CH * po.CH:po.LAYER_PARAMS] = rng.normal(0, 0.1, po.CH)   # non-zero biases
    ref_loss, ref_g, ref_hits = po.loss_and_grad(xL, xR, lab, theta, D)

    net = proposal.Net(torch, hd, wd, 1)
    x = torch.from_numpy(np.stack([xL, xR]).astype(np.float32)).cuda()
    th = torch.from_numpy(theta.astype(np.float32)).cuda()
    g = torch.zeros_like(th)
    labels = torch.from_numpy(np.concatenate([np.zeros((12, 1), np.int64), lab], 1).astype(np.int32)).cuda()
    loss_sum, hits = net.forward_backward(th, g, x, labels, 1, D)
    assert abs(loss_sum / 12 - ref_loss) <= 1e-4 * abs(ref_loss)
    assert hits == ref_hits
    gg = g.cpu().numpy().astype(np.float64)
    scale = np.abs(ref_g).max()
    assert np.abs(gg - ref_g).max() <= 1e-4 * scale, np.abs(gg - ref_g).max() / scale
    for l in range(po.LAYERS):   # every layer's block, relative to its own size
        sl = slice(l * po.LAYER_PARAMS, (l + 1) * po.LAYER_PARAMS)
        assert np.abs(gg[sl] - ref_g[sl]).max() <= 1e-3 * np.abs(ref_g[sl]).max() + 1e-9


@pytest.mark.parametrize("hd,wd", [(5, 300), (3, 64), (4, 128), (2, 257)])
def test_tensor_core_inference_matches_oracle(torch, hd, wd):
    rng = np.random.default_rng(hd * 1000 + wd)
    theta = po.init_params(11).astype(np.float64)
    for l in range(po.LAYERS):
        o = l * po.LAYER_PARAMS + po.TAPS * po.CH * po.CH
        theta[o:o + po.CH] = rng.normal(0, 0.1, po.CH)
    x = po.bf16_round(rng.normal(0, 1, (2, hd, wd, po.CH)))
    ref = po.net_fwd(x, po.unpack(theta), round_bf16=True)[-1]
    e = eb.Elas(eb.params_config(255))
    e.set_proposal(theta.astype(np.float32))
    xin = torch.from_numpy(x.astype(np.float32)).to(torch.bfloat16).cuda()
    out = torch.empty_like(xin)
    e.pn_infer(xin.data_ptr(), out.data_ptr(), hd, wd)
    got = out.float().cpu().numpy().astype(np.float64)
    e.close()
    err = np.abs(got - ref)
    assert err.max() <= 2e-2 * np.abs(ref).max(), err.max() / np.abs(ref).max()
    assert err.mean() <= 2e-3 * np.abs(ref).mean()


def test_features_bit_exact():
    L, R, _, _ = eb.synth_pair(0, 21)
    e = eb.Elas(eb.params_config(63))
    e.set_proposal(po.init_params(1))
    e.process(L, R)
    H, W = L.shape
    hd, wd = H // 4, W // 4
    dl = e.stage("desc_left").reshape(H, W, 16)
    dr = e.stage("desc_right").reshape(H, W, 16)
    f = eb.bf16_to_f32(e.stage("pn_features")).reshape(2, hd, wd, 32)
    e.close()
    assert np.array_equal(f[0], po.features(dl).astype(np.float32))
    assert np.array_equal(f[1], po.features(dr).astype(np.float32))


def _weights_or_random():
    if os.path.exists(eb.PN_WEIGHTS):
        return eb.load_proposal()
    return po.init_params(2)


@pytest.mark.parametrize("preset,seed", [(0, 31), (1, 32)])
def test_learned_support_matches_oracle(preset, seed):
    L, R, _, _ = eb.synth_pair(preset, seed)
    W, H, D = eb.synth_dims(preset)
    p = eb.params_config(D)
    e = eb.Elas(p)
    e.set_proposal(_weights_or_random())
    e.process(L, R)
    step = p.candidate_stepsize
    ch, cw = H // step, W // step
    can_lr = e.stage("can_lr").view(np.int32).reshape(ch, cw)
    bins = e.stage("pn_bins").view(np.uint32).reshape(ch, cw)
    dl = e.stage("desc_left").reshape(H, W, 16)
    dr = e.stage("desc_right").reshape(H, W, 16)
    settled, fell = e.proposal_stats()
    e.close()
    _, _, o = oracle.process(L, R, p, dumps=True)
    exp, s_ref, f_ref = po.learned_can_lr(dl, dr, bins, o["can_lr"], p)
    assert (settled, fell) == (s_ref, f_ref)
    assert np.array_equal(can_lr, exp), np.count_nonzero(can_lr != exp)


def _quality(D1, gt):
    valid = np.isfinite(gt) & (gt > 0)
    bad = (np.abs(D1 - gt) > 2) | (D1 < 0)
    return float(bad[valid].mean())


def test_trained_proposal_gain():
    """Held-out pairs: the trained network settles most candidates (untrained
    weights settle far fewer) at nearly the plain method's bad-2px."""
    if not os.path.exists(eb.PN_WEIGHTS):
        pytest.skip("no trained proposal weights in the package")
    seeds = [300000 + k for k in range(6)]
    p = eb.params_config(255)
    plain = eb.Elas(p)
    learned = eb.Elas(p)
    learned.set_proposal(eb.load_proposal())
    untrained = eb.Elas(p)
    untrained.set_proposal(po.init_params(0))
    fb_t, fb_u, bad_p, bad_l = [], [], [], []
    for s in seeds:
        L, R, gt, _ = eb.synth_pair(1, s)
        d_plain, _ = plain.process(L, R)
        d_learn, _ = learned.process(L, R)
        st, fl = learned.proposal_stats()
        fb_t.append(fl / max(st + fl, 1))
        untrained.process(L, R)
        st, fl = untrained.proposal_stats()
        fb_u.append(fl / max(st + fl, 1))
        bad_p.append(_quality(d_plain, gt))
        bad_l.append(_quality(d_learn, gt))
    for e in (plain, learned, untrained):
        e.close()
    print(f"fallback trained {np.mean(fb_t):.3f} untrained {np.mean(fb_u):.3f}; "
          f"bad-2px plain {np.mean(bad_p):.4f} learned {np.mean(bad_l):.4f}")
    assert np.mean(fb_t) < 0.5
    assert np.mean(fb_u) > np.mean(fb_t) + 0.1
    assert np.mean(bad_l) - np.mean(bad_p) < 0.01


@pytest.mark.parametrize("preset,seed", [(1, 33), (2, 34)])
def test_topk_bins_match_float64_scores(preset, seed):
    """The packed top-4 bins of every candidate, from the GPU's own network
    output: valid, distinct, as many as there are valid bins (up to four),
    and the four best of the float64 scores.  Where two scores lie within
    float rounding of each other either order is accepted, so the check
    compares the scores of the chosen bins, not the bin numbers."""
    L, R, _, _ = eb.synth_pair(preset, seed)
    W, H, D = eb.synth_dims(preset)
    p = eb.params_config(D)
    e = eb.Elas(p)
    e.set_proposal(_weights_or_random())
    e.process(L, R)
    step = p.candidate_stepsize
    ch, cw = H // step, W // step
    hd, wd = H // 4, W // 4
    F = eb.bf16_to_f32(e.stage("pn_output")).reshape(2, hd, wd, 32).astype(np.float64)
    bins = e.stage("pn_bins").view(np.uint32).reshape(ch, cw)
    e.close()
    sh = po.bin_shifts(D)
    cys = np.minimum(np.arange(ch) * step // 4, hd - 1)
    cxs = np.minimum(np.arange(cw) * step // 4, wd - 1)
    worst = 0.0
    for vc in range(ch):
        cy = cys[vc]
        xr = cxs[:, None] - sh[None, :]                       # (cw, 64)
        valid = xr >= 0
        s = po.SCALE * np.einsum("ck,cbk->cb", F[0, cy, cxs], F[1, cy, np.maximum(xr, 0)])
        s = np.where(valid, s, -np.inf)
        exp_sorted = -np.sort(-s, axis=1)[:, :po.TOPK]
        for ci in range(cw):
            got = po.unpack_bins(bins[vc, ci])
            nvalid = int(valid[ci].sum())
            assert len(got) == min(po.TOPK, nvalid)
            assert len(set(got)) == len(got)
            assert all(valid[ci, b] for b in got)
            gs = s[ci, got]
            es = exp_sorted[ci, :len(got)]
            tol = 1e-5 * (1.0 + np.abs(es))
            assert np.all(np.diff(gs) <= tol[1:]), (vc, ci, got, gs)
            if len(got):
                worst = max(worst, float(np.max(np.abs(gs - es) / tol)))
    assert worst <= 1.0, worst


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nimg,hd,wd", [(1, 1, 1), (2, 8, 32), (3, 9, 33), (2, 5, 31), (1, 17, 65),
                                        (7, 100, 200)])
def test_training_convolutions_at_tile_edges(torch, nimg, hd, wd, shift):
    """Forward, input, weight and bias gradients of one layer around the
    kernels' tile sizes (16 x 32 and 4 x 32 cells), with more tiles than the
    GPU takes at once, and with buffers off a
    16-byte boundary (shift floats), against float64.  A sum of n products
    in fp32, in any order, is off by at most n * 2^-23 of the sum of their
    magnitudes."""
    F = torch.nn.functional
    gen = torch.Generator().manual_seed(1000 * hd + wd + shift)

    def buf(n, data=None):
        t = torch.zeros(n + 4, device="cuda")[shift:shift + n]
        if data is not None:
            t.copy_(data.reshape(-1))
        return t

    ch, taps = po.CH, po.TAPS
    x, dy = (torch.randn((nimg, hd, wd, ch), generator=gen) for _ in range(2))
    w, b = torch.randn((taps, ch, ch), generator=gen) * 0.1, torch.randn(ch, generator=gen)
    n = x.numel()
    dx_, dy_, dw_, db_ = buf(n, x), buf(n, dy), buf(w.numel(), w), buf(ch, b)
    y, gx, gw, gb, scratch = buf(n), buf(n), buf(w.numel()), buf(ch), buf(w.numel())
    eb.pn_conv_forward(dx_.data_ptr(), dw_.data_ptr(), db_.data_ptr(), y.data_ptr(), nimg, hd, wd, True)
    eb.pn_conv_backward(dx_.data_ptr(), y.data_ptr(), dw_.data_ptr(), dy_.data_ptr(), gx.data_ptr(), gw.data_ptr(),
                        gb.data_ptr(), scratch.data_ptr(), nimg, hd, wd, True)
    torch.cuda.synchronize()

    def conv(v, k):                       # v [n][h][w][ci], k [tap][ci][co]
        k = k.view(3, 3, ch, ch).permute(3, 2, 0, 1)
        return F.conv2d(v.permute(0, 3, 1, 2), k, padding=1).permute(0, 2, 3, 1)

    xd, wd_, got = x.double(), w.double(), y.cpu().double().view(x.shape)
    ref = conv(xd, wd_) + b.double()
    mag = conv(xd.abs(), wd_.abs()) + b.double().abs()
    assert bool(((got - ref.clamp(min=0)).abs() <= (taps * ch + 1) * 2.0 ** -23 * mag).all())
    g = torch.where(got > 0, dy.double(), torch.zeros_like(got))     # the ReLU mask the kernels used
    flip = wd_.flip(0).transpose(1, 2)
    assert bool(((gx.cpu().double().view(x.shape) - conv(g, flip)).abs()
                 <= taps * ch * 2.0 ** -23 * conv(g.abs(), flip.abs())).all())

    def wgrad(v, u):
        p = F.pad(v, (0, 0, 1, 1, 1, 1))
        return torch.stack([torch.einsum("nhwi,nhwo->io", p[:, t // 3:t // 3 + hd, t % 3:t % 3 + wd], u)
                            for t in range(taps)])

    cells = nimg * hd * wd
    assert bool(((gw.cpu().double().view(w.shape) - wgrad(xd, g)).abs()
                 <= cells * 2.0 ** -23 * wgrad(xd.abs(), g.abs())).all())
    assert bool(((gb.cpu().double() - g.sum((0, 1, 2))).abs() <= cells * 2.0 ** -23 * g.abs().sum((0, 1, 2))).all())


def _conv_pair(torch, nimg, hd, wd, shift, groups):
    """Forward map and input gradient of `nimg` images, `groups` equal calls
    after one another on parts of the same buffers."""
    gen = torch.Generator().manual_seed(100 * hd + wd + shift)
    ch, taps = po.CH, po.TAPS

    def buf(t):
        b = torch.zeros(t.numel() + 4, device="cuda")[shift:shift + t.numel()]
        b.copy_(t.reshape(-1))
        return b

    x, dy = (buf(torch.randn((nimg, hd, wd, ch), generator=gen)) for _ in range(2))
    w, b = buf(torch.randn((taps, ch, ch), generator=gen) * 0.1), buf(torch.randn(ch, generator=gen))
    y, dx = torch.full_like(x, 9.0), torch.full_like(x, 9.0)
    gw, gb, scratch = buf(torch.zeros(taps * ch * ch)), buf(torch.zeros(ch)), buf(torch.zeros(taps * ch * ch))
    n = nimg // groups
    part = 4 * n * hd * wd * ch                 # bytes
    for k in range(groups):
        at = [t.data_ptr() + k * part for t in (x, y, dy, dx)]
        eb.pn_conv_forward(at[0], w.data_ptr(), b.data_ptr(), at[1], n, hd, wd, True)
        eb.pn_conv_backward(at[0], at[1], w.data_ptr(), at[2], at[3], gw.data_ptr(), gb.data_ptr(),
                            scratch.data_ptr(), n, hd, wd, True)
    torch.cuda.synchronize()
    return y, dx


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nimg,hd,wd", [(12800, 1, 1), (60, 8, 32), (30, 16, 32), (50, 9, 33), (90, 5, 31), (12, 17, 65),
                                        (2, 37, 332)])
def test_training_convolutions_equal_over_the_dispatch(torch, nimg, hd, wd, shift):
    """The same images in one call, large enough for the tile kernel, and in
    small calls, which the row kernel takes (37 x 332 cells: the most it
    takes on 148 SMs): the same bits, as both add in the same order."""
    assert nimg * hd * wd > 12284 and nimg * hd * wd // 2 <= 12284
    for a, b in zip(_conv_pair(torch, nimg, hd, wd, shift, 1), _conv_pair(torch, nimg, hd, wd, shift, 2)):
        assert torch.equal(a, b), int((a != b).sum())


def test_small_training_convolutions_take_less_time(torch):
    """A layer on 1 x 16 x 32 cells takes less than 0.6 of the time of one on
    73 times as many (2 x 60 x 310), each the fastest of 20 times 20 calls."""
    ms = []
    for nimg, hd, wd in [(1, 16, 32), (2, 60, 310)]:
        n = nimg * hd * wd * po.CH
        x, y = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
        w, b = torch.zeros(po.TAPS * po.CH * po.CH, device="cuda"), torch.zeros(po.CH, device="cuda")
        times = []
        for _ in range(20):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            for _ in range(20):
                eb.pn_conv_forward(x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), nimg, hd, wd, True)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        ms.append(min(times))
    assert ms[0] < 0.6 * ms[1], ms
