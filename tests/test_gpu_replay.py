"""Replayed CUDA graphs against fresh runs: whatever happens to a handle
between two calls with the same sizes, buffers and parameters, a replay must
give what a handle without a graph gives."""
import numpy as np
import pytest

import elas_b200 as eb

pytestmark = pytest.mark.gpu


class Batch:
    """Device buffers of a batch, its inputs, and the call on them."""

    def __init__(self, shapes, seed):
        import torch

        self.torch = torch
        self.dims, self.dmax = [(w, h) for w, h, _ in shapes], [d for _, _, d in shapes]
        self.images = [eb.synth_pair(3, seed + i, width=w, height=h, disp_max=d, gt=False)[:2]
                       for i, (w, h, d) in enumerate(shapes)]
        self.bufs = [[torch.from_numpy(x).cuda() for x in p] + [torch.empty((h, w), device="cuda") for _ in range(2)]
                     for p, (w, h, _) in zip(self.images, shapes)]

    def run(self, e):
        for b in self.bufs:
            b[2].fill_(7.0)
            b[3].fill_(7.0)
        self.torch.cuda.synchronize()
        e.process_batch_device(*[[b[k].data_ptr() for b in self.bufs] for k in range(4)], self.dims, self.dmax)
        self.torch.cuda.synchronize()
        return [b[k].cpu().numpy() for b in self.bufs for k in (2, 3)]


def singles(batch, weights=None):
    out = []
    for (L, R), d in zip(batch.images, batch.dmax):
        e = eb.Elas(eb.params_config(d))
        e.set_graphs(False)
        e.set_proposal(weights)
        out += e.process(L, R)
        e.close()
    return out


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_batch_replays_follow_the_proposal():
    """A batch that was captured without the learned proposal, called again
    with it, with other weights and without it."""
    import proposal_oracle as po

    batch = Batch([(640, 480, 128), (480, 272, 128)], 310)
    sets = [None, eb.load_proposal(), po.init_params(2), None]
    e = eb.Elas(eb.params_config(128))
    try:
        expected = {}
        for k, w in enumerate(sets):
            e.set_proposal(w)
            ref = expected[k] = singles(batch, w)
            for _ in range(3):                  # eager and captured, then replayed twice
                assert same(batch.run(e), ref), k
        assert not same(expected[0], expected[1])       # the proposal does change these maps
    finally:
        e.close()


def test_batch_replays_after_larger_batches():
    """A captured batch called again after batches of larger pairs, host and
    device, have made the workers allocate other workspaces."""
    small, large = Batch([(160, 120, 47), (200, 144, 63)], 330), Batch([(640, 480, 128), (800, 600, 255)], 340)
    ref_small, ref_large = singles(small), singles(large)
    e = eb.Elas(eb.params_config(64))
    try:
        assert same(small.run(e), ref_small) and same(small.run(e), ref_small)
        o1, o2 = e.process_batch([p[0] for p in large.images], [p[1] for p in large.images], large.dmax)
        assert same([x for p in zip(o1, o2) for x in p], ref_large)
        assert same(small.run(e), ref_small) and same(small.run(e), ref_small)
        assert same(large.run(e), ref_large) and same(small.run(e), ref_small)
    finally:
        e.close()


def test_pair_replays_after_the_network_maps_were_reallocated():
    """A captured pair with the proposal called again after elas_b200_pn_infer
    on larger maps has made the handle allocate its feature maps anew."""
    import torch

    W, H, D = 160, 120, 47
    weights = eb.load_proposal()
    e, other = eb.Elas(eb.params_config(D)), eb.Elas(eb.params_config(D))
    other.set_graphs(False)
    for h in (e, other):
        h.set_proposal(weights)
    try:
        for k, (hd, wd) in enumerate([(0, 0), (40, 50), (150, 200), (500, 600)]):
            if hd:
                x = torch.zeros((2, hd, wd, 32), dtype=torch.bfloat16, device="cuda")
                e.pn_infer(x.data_ptr(), torch.empty_like(x).data_ptr(), hd, wd)
            L, R = eb.synth_pair(3, 350 + k, width=W, height=H, disp_max=D, gt=False)[:2]
            ref = other.process(L, R)
            for _ in range(3):
                assert same(e.process(L, R), ref), k
    finally:
        e.close()
        other.close()


def test_batch_latency_belongs_to_the_last_batch():
    """elas_b200_batch_latency after a replay that follows a batch of another
    length: the replayed batch's pairs."""
    three, one = Batch([(160, 120, 47)] * 3, 360), Batch([(96, 64, 31)], 370)
    e = eb.Elas(eb.params_config(64))
    try:
        three.run(e)
        three.run(e)
        L, R = one.images[0]
        e.process_batch([L], [R], one.dmax)
        assert len(e.batch_latency(3)) == 1
        three.run(e)
        lat = e.batch_latency(3)
        assert len(lat) == 3 and (lat > 0).all()
    finally:
        e.close()


def test_pair_survives_a_failed_rebind():
    """A captured pair whose images could be rebound but not its outputs: that
    call and the later ones, on the first and the other buffers, give their
    own images' maps in their own outputs."""
    import torch

    W, H, D = 160, 120, 47
    e, other = eb.Elas(eb.params_config(D)), eb.Elas(eb.params_config(D))
    e.set_test_mode(eb.Elas.TEST_REBIND_FAILS)
    other.set_graphs(False)
    pairs = [eb.synth_pair(3, 380 + k, width=W, height=H, disp_max=D, gt=False)[:2] for k in range(2)]
    refs = [other.process(L, R) for L, R in pairs]
    sets = [[torch.from_numpy(x).cuda() for x in p] + [torch.empty((H, W), device="cuda") for _ in range(2)]
            for p in pairs]
    try:
        for k, i in enumerate([0, 0, 0, 1, 0, 0, 1, 1, 1, 0]):     # eager, captured, replayed, refused, ...
            for b in sets:
                b[2].fill_(7.0)
                b[3].fill_(7.0)
            torch.cuda.synchronize()
            e.process_device(*[x.data_ptr() for x in sets[i]], W, H)
            torch.cuda.synchronize()
            assert same([x.cpu().numpy() for x in sets[i][2:]], refs[i]), k
            assert bool((sets[1 - i][2] == 7.0).all()), k
    finally:
        e.close()
        other.close()


def test_new_weights_wait_for_calls_in_flight():
    """elas_b200_set_proposal while pairs on a stream of their own are still
    running: those keep the weights that they were called with."""
    import torch

    import proposal_oracle as po

    W, H, D = 2880, 1988, 255
    L, R = eb.synth_pair(2, 390, width=W, height=H, disp_max=D, gt=False)[:2]
    first, second = eb.load_proposal(), po.init_params(2)
    e = eb.Elas(eb.params_config(D))
    try:
        refs = []
        for w in (first, second):
            e.set_proposal(w)
            refs.append(e.process(L, R))
        assert not same(*refs)
        st = torch.cuda.Stream()
        images = [torch.from_numpy(x).cuda() for x in (L, R)]
        outs = [[torch.empty((H, W), device="cuda") for _ in range(2)] for _ in range(8)]
        torch.cuda.synchronize()
        for k, o in enumerate(outs):            # new weights after every pair, none waited for
            e.set_proposal((first, second)[k % 2])
            e.process_device(*[x.data_ptr() for x in images + o], W, H, stream=st.cuda_stream)
        e.set_proposal(first)
        torch.cuda.synchronize()
        for k, o in enumerate(outs):
            assert same([x.cpu().numpy() for x in o], refs[k % 2]), k
    finally:
        e.close()
