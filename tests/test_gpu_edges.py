"""The kernels at the sizes where they could go wrong: edges of lanes, warps, blocks and slots,
remainders, the smallest and the largest of a range, each branch of a dispatch.  Against the CPU
oracle, or against another path of this package that the oracle pins."""
import sys

import numpy as np
import pytest
import torch

from oracle import oracle
from oracle.common import HostFsaVec, make_arcs
from pruned_util import decoding_graph
from util import close, random_dense, same_fsa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def k2():
    import k2_b200
    return k2_b200


# --------------------------------------------------------------------------- lattice scores
def layered_lattice(rng, widths, degree, scale, hub=None):
    """One FSA whose arcs go from a layer to the next; `degree` arcs into a state on average,
    `hub` of them into the first state of the middle layer."""
    first = np.concatenate([[0], np.cumsum(widths)])
    rows = []
    for l in range(1, len(widths)):
        for s in range(widths[l]):
            d = max(1, int(rng.poisson(degree)))
            if hub and s == 0 and l == len(widths) // 2:
                d = hub
            for src in rng.integers(0, widths[l - 1], size=d):
                label = -1 if l == len(widths) - 1 else int(rng.integers(0, 9))
                rows.append((first[l - 1] + src, first[l] + s, label, rng.normal() * scale))
    rows.sort(key=lambda r: r[0])
    r = np.array(rows, np.float64)
    rs2 = np.zeros(first[-1] + 1, np.int64)
    np.add.at(rs2, r[:, 0].astype(np.int64) + 1, 1)
    arcs = make_arcs(r[:, 0].astype(np.int32), r[:, 1].astype(np.int32),
                     r[:, 2].astype(np.int32), r[:, 3].astype(np.float32))
    host = HostFsaVec(np.array([0, first[-1]], np.int32), np.cumsum(rs2).astype(np.int32), arcs)
    return host, first


def with_layers(fsa, host, widths, first):
    arcs_per_layer = np.diff(host.row_splits2[first])
    fsa.arcs._levels = (torch.tensor([0, len(widths)], dtype=torch.int32, device=DEV),
                        torch.from_numpy(first.astype(np.int32)).to(DEV))
    fsa.arcs._layer_bounds = (1, len(widths), int(max(widths)), int(arcs_per_layer.max()))
    return fsa


@pytest.mark.parametrize("widths,degree,scale,hub", [
    ([1, 1], 1.0, 1.0, None),                        # one arc
    ([1, 31, 32, 33, 1], 1.2, 1.0, None),            # two arcs per lane, a warp and its edges
    ([1] + [4] * 40 + [1], 1.25, 1.0, None),         # ... in the log semiring, else three
    ([1] + [6] * 40 + [1], 1.25, 1.0, None),         # three
    ([1] + [60] * 70 + [1], 1.25, 1.0, None),        # ... the widest
    ([1] + [64] * 70 + [1], 1.25, 1.0, None),        # two
    ([1] + [40] * 70 + [1], 2.5, 1.0, None),         # three; several slots of 32 layers
    ([1, 70, 64, 65, 1], 5.0, 1.0, 33),              # four; a state over several lanes
    ([1, 30, 40, 50, 1], 12.0, 1.0, 300),            # eight; a state of more than 32 x 8 arcs
    ([1, 600, 700, 600, 1], 3.0, 60.0, None),        # values out of the shared exponent's range
    ([1, 1023, 1024, 1000, 1], 2.0, 1.0, 700),       # the widest that eight warps slice
    ([1, 1025, 1000, 1026, 1], 2.0, 1.0, 700),       # by four warps
    ([1, 500, 20000, 4097, 8, 1], 2.0, 1.0, None),   # wide: one to eight lanes per state
    ([1, 18000, 3, 18000, 1], 2.0, 1.0, 700),        # wide, with a state for the whole warp
    ([1, 4095, 4097, 8193, 513, 1024, 2, 1], 2.0, 1.0, 90),  # turns of 4096 and their edges
    ([1] + [5000, 12001, 10999, 11002] * 5 + [1], 1.5, 1.0, None),  # through L2 and not, in turn
    ([1] + [3] * 1100 + [1], 1.2, 1.0, None),        # paths traced in runs of 512 layers
    ([1] + [901] * 120 + [1], 1.1, 1.0, None),       # ... of 48 K states
    ([1] + [7001] * 9 + [1], 1.1, 1.0, None),        # ... too short to be staged
])
def test_lattice_scores_and_best_path(k2, widths, degree, scale, hub):
    from gpu_util import host_to_fsa
    rng = np.random.default_rng(len(widths))
    host, first = layered_lattice(rng, widths, degree, scale, hub)
    fsa = with_layers(host_to_fsa(host), host, widths, first)
    for log in (True, False):
        for get, want in ((fsa.get_forward_scores, oracle.forward_scores(host, log)),
                          (fsa.get_backward_scores, oracle.backward_scores(host, log))):
            got = get(use_double_scores=True, log_semiring=log).detach().cpu().numpy()
            assert close(got, want, rtol=1e-10, atol=1e-9)
    best = k2.shortest_path(fsa, use_double_scores=True)
    tot = fsa.get_tot_scores(log_semiring=False, use_double_scores=True)
    assert best.num_arcs == (len(widths) - 1 if torch.isfinite(tot).all() else 0)
    assert close(best.scores.double().sum().item(), tot[0].item(), rtol=1e-6, atol=1e-5)


def test_lattice_with_empty_layers_at_its_ends(k2):
    # the first state of a walk is not in the walk's first layer: it scores 0 all the same
    from gpu_util import host_to_fsa
    widths = [1] + [5] * 70 + [1]
    host, first = layered_lattice(np.random.default_rng(9), widths, 1.3, 1.0)
    for before, behind in ((0, 0), (1, 0), (0, 1), (3, 40)):
        splits = np.concatenate([np.zeros(before, np.int64), first, np.full(behind, first[-1])])
        fsa = with_layers(host_to_fsa(host), host, [0] * before + widths + [0] * behind, splits)
        for log in (True, False):
            for get, want in ((fsa.get_forward_scores, oracle.forward_scores(host, log)),
                              (fsa.get_backward_scores, oracle.backward_scores(host, log))):
                got = get(use_double_scores=True, log_semiring=log).detach().cpu().numpy()
                assert close(got, want, rtol=1e-10, atol=1e-9), (before, behind, log)


@pytest.mark.parametrize("copies", [2, 149, 297, 445])
@pytest.mark.parametrize("widths", [[1] + [400] * 40 + [1], [1] + [3, 2, 3] * 9 + [1]])
def test_best_paths_of_many_fsas(k2, copies, widths):
    # what a CTA traces at a time shrinks from 48 K states to 12 K with the number of FSAs (one has
    # 16 002 here, or 74, all of them in one run); copies of one FSA have the path of that FSA
    from gpu_util import host_to_fsa
    host, first = layered_lattice(np.random.default_rng(8), widths, 1.3, 1.0)
    na, ns = len(host.arcs), int(first[-1])
    every = np.arange(copies)[:, None]
    tiled = HostFsaVec((np.arange(copies + 1) * ns).astype(np.int32),
                       np.append((every * na + host.row_splits2[None, :-1]).reshape(-1),
                                 copies * na).astype(np.int32),
                       np.tile(host.arcs, (copies, 1)))
    fsa = with_layers(host_to_fsa(tiled), host, widths, first)
    splits = np.append((every * ns + first[None, :-1]).reshape(-1), copies * ns)
    fsa.arcs._levels = (torch.arange(copies + 1, dtype=torch.int32, device=DEV) * len(widths),
                        torch.from_numpy(splits.astype(np.int32)).to(DEV))
    _, entering = oracle.forward_scores(host, False, True, want_entering_arcs=True)
    want = oracle.shortest_path(host, entering)[1]
    best = k2.shortest_path(fsa, use_double_scores=True)._best_arc_map.cpu().numpy()
    assert len(want) == len(widths) - 1
    assert np.array_equal(best.reshape(copies, -1), every * na + want[None, :])


@pytest.mark.parametrize("widths", [
    [1, 4095, 4097, 8193, 513, 1],            # values from CTA to CTA
    [1, 12001, 300, 12001, 11000, 12500, 1],  # some through L2, with barriers of the cluster
])
def test_wide_layers_whose_waits_give_up_are_redone(k2, widths):
    # with a limit of 0 every wait of the wide chain gives up at its first layer: it ends, says so,
    # and the scores come from the kernel behind it
    from gpu_util import host_to_fsa
    from k2_b200 import _lib
    host, first = layered_lattice(np.random.default_rng(3), widths, 1.5, 1.0)
    for log in (True, False):
        fsa = with_layers(host_to_fsa(host), host, widths, first)
        want = (oracle.forward_scores(host, log), oracle.backward_scores(host, log))
        try:
            _lib.lib.k2b200_debug_set_copy_wait_limit(0)
            got = [get(use_double_scores=True, log_semiring=log).detach().cpu().numpy()
                   for get in (fsa.get_forward_scores, fsa.get_backward_scores)]
        finally:
            _lib.lib.k2b200_debug_set_copy_wait_limit(-1)
        for a, b in zip(got, want):
            assert close(a, b, rtol=1e-10, atol=1e-9)


# --------------------------------------------------------------------------- CTC loss
def ctc_inputs(rng, n, frames, classes, tokens, gaps):
    durs = np.sort(rng.integers(max(1, frames // 2), frames + 1, size=n))[::-1]
    durs[0] = frames
    x = torch.from_numpy(rng.normal(size=(n, frames + gaps, classes)).astype(np.float32) * 1.5)
    seg = np.stack([np.arange(n), np.full(n, gaps), durs], 1).astype(np.int32)
    symbols = [rng.integers(1, classes, size=int(min(rng.integers(1, tokens + 1), d // 3))).tolist()
               for d in durs]
    for s in symbols[1::2]:  # repeats
        s[1:2] = s[:1]
    symbols[-1] = []
    return x.to(DEV), torch.from_numpy(seg), symbols


@pytest.mark.parametrize("n,frames,classes,tokens,modified,gaps,lens_dtype,logits,delay", [
    (3, 1, 3, 1, False, 0, torch.int32, False, 0.0),       # one frame
    (4, 15, 29, 5, False, 1, torch.int64, False, 0.0),     # odd columns, rows of no sequence
    (3, 17, 501, 6, True, 0, torch.float32, True, 0.0),
    (2, 33, 1023, 11, False, 3, torch.float64, True, 0.0),
    (3, 40, 1500, 12, True, 0, torch.int32, False, 0.0),   # rows by state
    (2, 800, 40, 270, False, 0, torch.int64, False, 0.0),  # more than 512 states
    (3, 60, 30, 20, False, 2, torch.int32, False, 0.1),
    (3, 50, 1300, 16, True, 0, torch.int64, True, 0.2),
    (2, 600, 31, 190, False, 0, torch.int32, False, 0.2),  # the exact recursion
])
def test_ctc_loss_on_the_band_kernels(k2, n, frames, classes, tokens, modified, gaps, lens_dtype,
                                      logits, delay):
    module = sys.modules["k2_b200.ctc_loss"]
    rng = np.random.default_rng(frames + classes)
    x, seg, symbols = ctc_inputs(rng, n, frames, classes, tokens, gaps)
    if not logits:
        x = torch.log_softmax(x, -1)
    make = k2.DenseFsaVec.from_logits if logits else k2.DenseFsaVec
    lens = torch.tensor([max(1, len(s)) for s in symbols], dtype=lens_dtype, device=DEV)
    for reduction in ("sum", "mean"):
        got = []
        for fused in (True, False):
            module.FUSED_LOSS = fused
            try:
                graphs = k2.ctc_graph(symbols, modified=modified, device=DEV)
                leaf = x.clone().requires_grad_(True)
                loss = k2.ctc_loss(graphs, make(leaf, seg), output_beam=10.0, delay_penalty=delay,
                                   reduction=reduction, target_lengths=lens)
                loss.backward()
            finally:
                module.FUSED_LOSS = True
            got.append((loss.item(), leaf.grad.cpu().numpy()))
        # Totals in double, four of them added in float32: 4 x 2^-24.  The lattice adds at most 128
        # posteriors of a frame and label in float32 (128 x 2^-24); with a penalty it also rounds
        # the score of every arc.
        assert close(got[0][0], got[1][0], rtol=1e-4 if delay else 3e-7, atol=1e-6)
        assert np.abs(got[0][1] - got[1][1]).max() <= (1e-4 if delay else 1e-5)


@pytest.mark.parametrize("modified", [False, True])
@pytest.mark.parametrize("lengths", [[0], [1], [0, 3, 0], [31, 32, 33], [500, 0, 511, 512]])
def test_ctc_graph_on_the_device(k2, lengths, modified):
    from gpu_util import fsa_to_host
    rng = np.random.default_rng(len(lengths))
    symbols = [rng.integers(1, 3, size=k).tolist() for k in lengths]  # many repeats
    got = k2.ctc_graph(symbols, modified=modified, device=DEV)
    same_fsa(fsa_to_host(got), oracle.ctc_graphs(symbols, modified), f"{lengths}")
    cpu = k2.ctc_graph(symbols, modified=modified, device="cpu")
    assert torch.equal(got.aux_labels.cpu(), cpu.aux_labels)


def test_ctc_graph_of_symbols_that_are_not_integers(k2):
    """What the native conversion leaves to numpy: the kernels for symbols on the device."""
    got = k2.ctc_graph([[1.0, 2.0, 2.0], [3.5], []], device=DEV)
    want = k2.ctc_graph([[1, 2, 2], [3], []], device=DEV)
    for a, b in ((got.arcs.values(), want.arcs.values()), (got.aux_labels, want.aux_labels),
                 (got.arcs._row_splits1, want.arcs._row_splits1),
                 (got.arcs._row_splits2, want.arcs._row_splits2)):
        assert torch.equal(a, b)


# --------------------------------------------------------------------------- planned lanes
@pytest.mark.parametrize("phones", [40, 78, 80, 84, 105])  # around 768 and 1024 lanes
def test_lane_plans(k2, phones):
    from k2_b200 import synthetic as syn
    rs2, arcs = syn.den_graph(phones, phones)
    rng = np.random.default_rng(phones)
    lp = np.log(rng.dirichlet(np.ones(phones + 1) * 0.3, size=(2, 12))).astype(np.float32)
    w = syn.Workload("lfmmi", torch.from_numpy(lp), torch.tensor([[0, 0, 12], [1, 0, 9]],
                                                                dtype=torch.int32), 8.0,
                     graph_row_splits2=rs2, graph_arcs=arcs, num_symbols=None)
    graphs = syn.build_graphs(w, DEV)
    got = []
    for fused in (True, False):
        x = w.log_probs.to(DEV).requires_grad_(True)
        dense = k2.DenseFsaVec(x, w.supervision_segments)
        if fused:
            tot = k2.intersect_dense_tot_scores(graphs, dense, 8.0)
        else:
            tot = k2.intersect_dense(graphs, dense, 8.0).get_tot_scores(True, True)
        tot.sum().backward()
        got.append((tot.detach().cpu().numpy(), x.grad.cpu().numpy()))
    assert close(got[0][0], got[1][0], rtol=1e-6, atol=1e-5)
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-4


@pytest.mark.parametrize("classes", [613, 614, 1363, 1364, 2047, 4000])
def test_lane_plans_with_many_classes(k2, classes):
    """Rows of dense scores that leave shared memory fewer frames per CTA: 56 up to 614 columns of
    the score matrix, 32 up to 1364."""
    from k2_b200 import synthetic as syn
    rs2, arcs = syn.den_graph(20, 20)
    rng = np.random.default_rng(classes)
    lp = torch.log_softmax(torch.from_numpy(
        rng.normal(size=(2, 70, classes)).astype(np.float32)), -1).to(DEV)
    seg = torch.tensor([[0, 0, 70], [1, 0, 61]], dtype=torch.int32)
    graphs = syn.build_graphs(syn.Workload("lfmmi", lp.cpu(), seg, 8.0, graph_row_splits2=rs2,
                                           graph_arcs=arcs, num_symbols=None), DEV)
    got = []
    for fused in (True, False):
        x = lp.clone().requires_grad_(True)
        dense = k2.DenseFsaVec(x, seg)
        assert k2.autograd.dense_loss_supported(graphs, dense)
        if fused:
            tot = k2.intersect_dense_tot_scores(graphs, dense, 8.0)
        else:
            tot = k2.intersect_dense(graphs, dense, 8.0).get_tot_scores(True, True)
        tot.sum().backward()
        got.append((tot.detach().cpu().numpy(), x.grad.cpu().numpy()))
    assert close(got[0][0], got[1][0], rtol=1e-6, atol=1e-5)
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-4


@pytest.mark.parametrize("classes", [12796, 12800, 20000])
def test_lattice_of_many_classes(k2, classes):
    """Around the most columns of which four rows fit in the ring of the lane kernel."""
    from gpu_util import dense_from_scores, fsa_to_host, host_to_fsa, intersect_raw
    from k2_b200 import synthetic as syn
    rs2, arcs = syn.den_graph(8, 8)
    a = HostFsaVec(np.array([0, len(rs2) - 1], np.int32), rs2, arcs)
    scores, brs = random_dense(np.random.default_rng(classes), 1, 12, classes)
    want = oracle.intersect_dense(a, scores, brs, 6.0)
    fsa = host_to_fsa(a)
    assert fsa.arcs.max_degree() > 4
    lattice, ma, mb = intersect_raw(fsa, dense_from_scores(scores, brs), 6.0)
    same_fsa(fsa_to_host(lattice, ma, mb), want, f"{classes} classes")


@pytest.mark.parametrize("states,classes", [(40, 6016), (40, 6017), (40, 9000), (300, 7700)])
def test_lane_per_state_with_many_classes(k2, states, classes):
    """Graphs of at most four arcs per state that are no band graphs; rows so long that the kernels
    of the gradient take fewer of them than they have warps."""
    from gpu_util import host_to_fsa
    rng = np.random.default_rng(classes)
    rows = []
    for s in range(states - 1):
        for d in (0, 1, 2):
            if s + d < states:
                final = s + d == states - 1
                label = -1 if final else int(rng.integers(0, classes))
                rows.append((s, s + d, label, rng.normal()))
    r = np.array(rows)
    rs2 = np.zeros(states + 1, np.int64)
    np.add.at(rs2, r[:, 0].astype(np.int64) + 1, 1)
    graph = host_to_fsa(HostFsaVec(
        np.array([0, states], np.int32), np.cumsum(rs2).astype(np.int32),
        make_arcs(r[:, 0].astype(np.int32), r[:, 1].astype(np.int32), r[:, 2].astype(np.int32),
                  r[:, 3].astype(np.float32))))
    frames = states
    lp = torch.log_softmax(torch.from_numpy(
        rng.normal(size=(1, frames, classes)).astype(np.float32)), -1).to(DEV)
    seg = torch.tensor([[0, 0, frames]], dtype=torch.int32)
    got = []
    for fused in (True, False):
        x = lp.clone().requires_grad_(True)
        dense = k2.DenseFsaVec(x, seg)
        assert not k2.autograd.band_loss_supported(graph, dense)
        if fused:
            tot = k2.intersect_dense_tot_scores(graph, dense, 10.0)
        else:
            tot = k2.intersect_dense(graph, dense, 10.0).get_tot_scores(True, True)
        assert torch.isfinite(tot).all()
        tot.sum().backward()
        got.append((tot.detach().cpu().numpy(), x.grad.cpu().numpy()))
    assert close(got[0][0], got[1][0], rtol=1e-6, atol=1e-5)
    # (scores of a few hundred: the lattice rounds each arc's to float32)
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-4


# --------------------------------------------------------------------------- pruned search
@pytest.mark.parametrize("states,classes,hub,n,teams", [
    (50, 5, 0, 1, (0, 1, 2, 8)),       # fewer arcs than a warp has lanes
    (900, 20, 700, 2, (0, 1)),         # a state of more arcs than a byte counts
    (400, 9000, 0, 2, (0,)),           # rows of scores that stay in global memory
    (270000, 30, 0, 1, (0, 1)),        # states that share a bit of the set of new states
])
def test_pruned_search(k2, states, classes, hub, n, teams):
    from gpu_util import dense_from_scores, fsa_to_host, host_to_fsa
    from k2_b200.autograd import _intersect_dense_pruned_arcs
    rng = np.random.default_rng(states)
    g = decoding_graph(rng, states, classes, mean_degree=4.0)
    if hub:  # the arcs of the start state once more, with other labels
        s0 = g.row_splits2[1]
        label = rng.integers(1, classes, size=hub).astype(np.int32)
        dest = rng.integers(1, states // 2, size=hub).astype(np.int32)
        extra = make_arcs(np.zeros(hub, np.int32), dest, label,
                          rng.normal(size=hub).astype(np.float32))
        arcs = np.concatenate([g.arcs[:s0], extra, g.arcs[s0:]])
        rs2 = g.row_splits2.copy()
        rs2[1:] += hub
        g = HostFsaVec(g.row_splits1, rs2, arcs)
    scores, brs = random_dense(rng, n, 45, classes, scale=2.0, low_rows=False)
    params = (14.0, 6.0, 5, 700, False)
    want = oracle.intersect_dense_pruned(g, scores, brs, *params)
    a, dense = host_to_fsa(g), dense_from_scores(scores, brs)
    for team in teams:
        ragged, ma, mb = _intersect_dense_pruned_arcs(a.arcs, dense, *params, team)
        same_fsa(fsa_to_host(k2.Fsa(ragged, _check=False), ma, mb), want, f"{team} CTAs")


@pytest.mark.parametrize("lengths", [[0], [1, 0], [2, 31, 32], [130, 1, 0, 64]])
def test_incoming_arcs_of_band_graphs(k2, lengths):
    rng = np.random.default_rng(sum(lengths))
    symbols = [rng.integers(1, 3, size=k).tolist() for k in lengths]
    for modified in (False, True):
        arcs = k2.ctc_graph(symbols, modified=modified, device=DEV).arcs
        want = k2.ctc_graph(symbols, modified=modified, device=DEV).arcs
        want._band_graph = None  # the general index
        for got, ref in zip(arcs.incoming(), want.incoming()):
            assert torch.equal(got, ref), (lengths, modified)


# --------------------------------------------------------------------------- the loss as a node
def small_loss(k2, leaf, logits, reduction="sum", lens=None):
    seg = torch.tensor([[0, 0, 30], [1, 2, 20], [2, 0, 15]], dtype=torch.int32)
    graphs = k2.ctc_graph([[1, 2, 3, 3], [5, 6], [16]], device=DEV)
    make = k2.DenseFsaVec.from_logits if logits else k2.DenseFsaVec
    return k2.ctc_loss(graphs, make(leaf, seg), reduction=reduction, target_lengths=lens)


def small_input(logits):
    x = torch.from_numpy(np.random.default_rng(5).normal(size=(3, 30, 17)).astype(np.float32))
    return (x if logits else torch.log_softmax(x, -1)).to(DEV)


@pytest.mark.parametrize("logits", [False, True])
def test_forward_mode_is_refused(k2, logits):
    from torch.autograd import forward_ad
    x = small_input(logits)
    with forward_ad.dual_level():
        with pytest.raises(NotImplementedError, match="jvp"):
            small_loss(k2, forward_ad.make_dual(x, torch.ones_like(x)), logits)
    for transform in (torch.func.grad, torch.func.vmap):
        with pytest.raises(RuntimeError):
            transform(lambda y: small_loss(k2, y, logits))(x if transform is torch.func.grad
                                                           else x[None])


@pytest.mark.parametrize("logits", [False, True])
def test_gradient_of_the_target_lengths(k2, logits):
    """mean(-tot / length): the lengths may want a gradient, too."""
    x = small_input(logits)
    lens = torch.tensor([4.0, 2.0, 1.0], device=DEV, requires_grad=True)
    small_loss(k2, x.clone().requires_grad_(True), logits, "mean", lens).backward()
    each = small_loss(k2, x, logits, "none")
    want = (-each / (3 * lens.detach() ** 2)).cpu()
    assert torch.allclose(lens.grad.cpu(), want, rtol=1e-6)


@pytest.mark.parametrize("logits", [False, True])
def test_when_the_loss_can_be_differentiated(k2, logits):
    """Twice with retain_graph and the same bits both times, else once; not when the target lengths
    changed in between."""
    x = small_input(logits)
    for reduction in ("sum", "mean"):
        leaf = x.clone().requires_grad_(True)
        lens = torch.tensor([4, 2, 1], device=DEV)
        loss = small_loss(k2, leaf, logits, reduction, lens)
        first, = torch.autograd.grad(loss, leaf, retain_graph=True)
        again, = torch.autograd.grad(loss, leaf, retain_graph=True)
        assert torch.equal(first, again) and first.abs().max() > 0
        if reduction == "mean":
            lens.mul_(2)
            with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                torch.autograd.grad(loss, leaf, retain_graph=True)
            loss = small_loss(k2, leaf, logits, reduction, lens)
        loss.backward()
        assert torch.equal(leaf.grad, first if reduction == "sum" else first / 2)
        with pytest.raises(RuntimeError, match="retain_graph"):
            loss.backward()


@pytest.mark.parametrize("upstream", [1.0, -2.0, 0.0, float("inf"), float("nan")])
def test_gradients_that_are_not_finite(k2, upstream):
    """Against the lattice: an upstream gradient of infinity or NaN (a target length of 0 makes one)
    reaches the elements that some path uses, no others; log-probs of NaN have a gradient of NaN
    through the softmax, on every row of an utterance without a path too."""
    module = sys.modules["k2_b200.ctc_loss"]
    for logits in (False, True):
        x = small_input(logits)
        if logits:
            x[1, 6, 3] = float("nan")    # a row of NaN
            x[2] = -float("inf")         # an utterance without a path
        got = []
        for fused in (True, False):
            module.FUSED_LOSS = fused
            try:
                leaf = x.clone().requires_grad_(True)
                small_loss(k2, leaf, logits).backward(torch.tensor(upstream, device=DEV))
            finally:
                module.FUSED_LOSS = True
            got.append(leaf.grad.cpu())
        # (posteriors to 1e-6, twice for the upstream gradient of -2)
        assert torch.allclose(got[0], got[1], rtol=0, atol=2e-6, equal_nan=True)
        assert torch.equal(got[0].isinf(), got[1].isinf())


def test_pruned_search_passes_by_scores_that_are_not_numbers(k2):
    """A NaN among the scores costs the arcs that read it, not the utterance.  (On graphs in which
    the arcs into a state have one label, so that a state whose arcs are NaN does not come up.)"""
    from gpu_util import dense_from_scores, fsa_to_host, host_to_fsa
    from k2_b200.autograd import _intersect_dense_pruned_arcs
    rng = np.random.default_rng(17)
    symbols = [rng.integers(1, 9, size=7).tolist() for _ in range(4)]
    graphs = oracle.ctc_graphs(symbols, False)
    scores, brs = random_dense(rng, 4, 60, 9, low_rows=False)
    holes = rng.random(scores.shape) < 0.03
    holes[:, 0] = holes[:, 1] = False
    holes[brs[1:] - 1] = False
    scores[holes] = np.nan
    params = (20.0, 8.0, 0, 10000, False)
    want = oracle.intersect_dense_pruned(graphs, scores, brs, *params)
    assert all(np.diff(want.row_splits2[want.row_splits1])[:3] > 100)  # (the last has 3 frames)
    for team in (0, 1, 4):
        ragged, ma, mb = _intersect_dense_pruned_arcs(
            host_to_fsa(graphs).arcs, dense_from_scores(scores, brs), *params, team)
        same_fsa(fsa_to_host(k2.Fsa(ragged, _check=False), ma, mb), want, f"{team} CTAs")


@pytest.mark.parametrize("n,frames,classes", [
    (1, 1, 1), (1, 1, 2), (1, 1, 5), (1, 2, 1), (2, 3, 5), (1, 17, 7), (3, 33, 29), (2, 16, 500),
])
def test_log_probs_of_any_alignment(k2, n, frames, classes):
    """The same bits wherever the log-probs start, with NaN in front of them and behind."""
    rng = np.random.default_rng(frames)
    x = torch.log_softmax(torch.from_numpy(
        rng.normal(size=(n, frames, classes)).astype(np.float32)), -1).to(DEV)
    seg = torch.tensor([[i, 0, frames] for i in range(n)], dtype=torch.int32)
    symbols = [[1] if classes > 1 else [] for _ in range(n)]
    got = []
    for offset in range(5):
        buf = torch.full((x.numel() + 12,), float("nan"), device=DEV)
        leaf = buf[offset:offset + x.numel()].view(x.shape)
        leaf.copy_(x)
        leaf.requires_grad_(True)
        loss = k2.ctc_loss(k2.ctc_graph(symbols, device=DEV), k2.DenseFsaVec(leaf, seg))
        loss.backward()
        got.append((loss.detach(), leaf.grad))
    assert torch.isfinite(got[0][0]) and torch.isfinite(got[0][1]).all()
    for loss, grad in got[1:]:
        assert torch.equal(loss, got[0][0]) and torch.equal(grad, got[0][1])


# --------------------------------------------------------------------------- workspaces
def test_one_pool_of_workspaces(k2):
    """Large workspaces come back to the next call on their stream, whichever path makes it; at most
    three are kept, and given back when asked."""
    from k2_b200 import _lib
    k2._lib.release_workspaces()
    torch.cuda.empty_cache()
    before = torch.cuda.memory_allocated()
    mb = 1 << 20
    first = _lib.workspace(100 * mb, DEV)
    at = first.tensor.data_ptr()
    assert first.tensor.numel() >= 100 * mb and first.tensor.device == torch.device(DEV)
    del first
    assert _lib.workspace(90 * mb, DEV).tensor.data_ptr() == at     # as large, or half as large
    with torch.cuda.stream(torch.cuda.Stream()):
        other = _lib.workspace(90 * mb, DEV)                        # another stream, another one
    assert other.tensor.data_ptr() != at
    del other
    k2._lib.release_workspaces()
    several = [_lib.workspace(n * 40 * mb, DEV) for n in range(1, 6)]
    del several
    kept = torch.cuda.memory_allocated() - before
    assert (3 + 4 + 5) * 40 * mb <= kept <= 1.2 * (3 + 4 + 5) * 40 * mb
    small = _lib.workspace(mb, DEV)                                 # not pooled
    del small
    # the general kernels and the band kernels of one batch size use one workspace after another
    k2._lib.release_workspaces()
    x = torch.log_softmax(torch.randn(16, 400, 60, device=DEV), -1)
    seg = torch.tensor([[i, 0, 400] for i in range(16)], dtype=torch.int32)
    graphs = k2.ctc_graph([[1 + i % 50 for i in range(100)]] * 16, device=DEV)
    for band in (True, False, True, False):
        k2.intersect_dense_tot_scores(graphs, k2.DenseFsaVec(x, seg), 10.0, band=band)
    torch.cuda.synchronize()
    del x, graphs
    k2._lib.release_workspaces()
    assert torch.cuda.memory_allocated() <= before + mb


@pytest.mark.parametrize("band", [True, False])
def test_captured_calls_keep_off_the_pool(k2, band):
    """A loss and its gradient as a CUDA graph: replays give the bits of eager calls whatever became
    of the pool since, and change nothing that other calls hold."""
    k2._lib.release_workspaces()
    n, frames, classes = 16, 400, 60
    seg = torch.tensor([[i, 0, frames] for i in range(n)], dtype=torch.int32)
    graphs = k2.ctc_graph([[1 + (3 * i + j) % 50 for i in range(100)] for j in range(n)], device=DEV)
    gen = torch.Generator(DEV).manual_seed(1)
    draw = lambda: torch.log_softmax(  # noqa: E731
        torch.randn(n, frames, classes, device=DEV, generator=gen), -1)

    def step(x):
        tot = k2.intersect_dense_tot_scores(graphs, k2.DenseFsaVec(x, seg), 10.0, band=band)
        return tot, torch.autograd.grad(tot.sum(), x)[0]

    static = draw().requires_grad_(True)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(2):
            step(static)
    torch.cuda.synchronize()
    captured = torch.cuda.CUDAGraph()
    with torch.cuda.graph(captured, stream=stream):
        got = step(static)
    k2._lib.release_workspaces()
    held = torch.full((1 << 28,), 3.0, device=DEV)  # where the warm-up's workspace was, among others
    for _ in range(3):
        x = draw()
        with torch.no_grad():
            static.copy_(x)
        captured.replay()
        want = step(x.requires_grad_(True))
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert bool((held == 3.0).all())


# --------------------------------------------------------------------------- streaming
def test_chunks_give_the_best_path_of_the_whole(k2):
    """Streams of 48 frames in chunks of 16 with beams that prune next to nothing: the best path of
    the last lattice has the score of the best path of the whole utterance."""
    from gpu_util import host_to_fsa
    rng = np.random.default_rng(23)
    graph = host_to_fsa(decoding_graph(rng, 400, 12, mean_degree=3.0))
    lp = torch.log_softmax(torch.from_numpy(
        rng.normal(size=(3, 48, 12)).astype(np.float32) * 2.0), -1).to(DEV)
    beams = (60.0, 50.0, 0, 10000)
    decoder = k2.OnlineDenseIntersecter(graph, 3, *beams)
    states = [None] * 3
    seg = torch.tensor([[i, 0, 16] for i in range(3)], dtype=torch.int32)
    for c in range(3):
        chunk = lp[:, 16 * c:16 * (c + 1)].contiguous()
        lattice, states = decoder.decode(k2.DenseFsaVec(chunk, seg), states)
    whole = k2.intersect_dense_pruned(
        graph, k2.DenseFsaVec(lp, torch.tensor([[i, 0, 48] for i in range(3)], dtype=torch.int32)),
        *beams)
    got = k2.shortest_path(lattice, use_double_scores=True)
    want = k2.shortest_path(whole, use_double_scores=True)
    assert torch.equal(got.arcs._row_splits2, want.arcs._row_splits2)
    assert torch.equal(got.labels, want.labels)
    # (arc scores are float32 sums of the same two numbers)
    assert torch.equal(got.scores, want.scores)


def test_backward_after_the_inputs_are_gone(k2):
    """A loss keeps the host arrays that its backward reads: the DenseFsaVec and the map are dropped
    and their memory is written over in between."""
    from k2_b200 import synthetic as syn
    rs2, arcs = syn.den_graph(20, 20)
    seg = torch.tensor([[i, 0, 60 - i] for i in range(16)], dtype=torch.int32)
    lp = torch.log_softmax(torch.randn(16, 60, 21, device=DEV), -1)
    graphs = {"den": syn.build_graphs(syn.Workload("x", lp.cpu(), seg, 8.0, graph_row_splits2=rs2,
                                                   graph_arcs=arcs, num_symbols=None), DEV),
              "ctc": k2.ctc_graph([[1, 2, 3]] * 16, device=DEV)}
    for name, graph in graphs.items():
        for amap in (None, list(range(16))):
            for band in (True, False):
                grads = []
                for drop in (False, True):
                    x = lp.clone().requires_grad_(True)
                    dense = k2.DenseFsaVec(x, seg)
                    m = None if amap is None else torch.tensor(amap, dtype=torch.int32)
                    tot = k2.intersect_dense_tot_scores(graph, dense, 8.0, a_to_b_map=m, band=band)
                    if drop:
                        del dense, m
                        over = [np.full(n, -1, np.int32) for n in (16, 17) for _ in range(200)]
                    tot.sum().backward()
                    grads.append(x.grad)
                del over
                assert torch.equal(grads[0], grads[1]), (name, amap is None, band)


def test_score_matrix_made_inside_a_loss(k2):
    """The matrix of a DenseFsaVec is made on first use.  Where that is inside a loss (which takes the
    gradient past it) or under no_grad, a lattice made from the same DenseFsaVec has its gradient;
    one made under no_grad has none."""
    from k2_b200 import synthetic as syn
    rs2, arcs = syn.den_graph(10, 10)
    seg = torch.tensor([[0, 0, 20], [1, 0, 18]], dtype=torch.int32)
    lp = torch.log_softmax(torch.randn(2, 20, 11, device=DEV), -1)
    graph = syn.build_graphs(syn.Workload("x", lp.cpu(), seg, 8.0, graph_row_splits2=rs2,
                                          graph_arcs=arcs, num_symbols=None), DEV)
    grads = []
    for first_use in ("lattice", "loss", "no_grad"):
        x = lp.clone().requires_grad_(True)
        dense = k2.DenseFsaVec(x, seg)
        if first_use == "loss":
            k2.intersect_dense_tot_scores(graph, dense, 8.0)
        elif first_use == "no_grad":
            with torch.no_grad():
                dense.scores
        k2.intersect_dense(graph, dense, 8.0).get_tot_scores(True, True).sum().backward()
        grads.append(x.grad)
    for grad in grads[1:]:  # (posteriors, added in any order)
        assert torch.allclose(grad, grads[0], rtol=0, atol=1e-5) and grad.abs().max() > 0.1
    with torch.no_grad():
        dense = k2.DenseFsaVec(lp.clone().requires_grad_(True), seg)
    assert not dense.scores.requires_grad
