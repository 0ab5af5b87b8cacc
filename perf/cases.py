"""The work that a user has this framework do, as cases that can be timed and compared.

Four kinds of call, each through the public entry points, over the range of sizes of the
configurations in `k2_b200/synthetic.py` and of the callers around them:

  ctc     a training step: graphs from the transcripts of the batch, `DenseFsaVec`,
          `ctc_loss`, backward to the network output (log-probs or logits)
  align   forced alignment: graphs from the transcripts, `intersect_dense`, `shortest_path`
  lfmmi   LF-MMI: the denominator graph (and numerator graphs) against the network output,
          with or without the lattice, total scores and backward
  decode  `get_lattice` on a decoding graph shared by the batch, best path, output symbols
  online  the same chunk by chunk with `OnlineDenseIntersecter`

`prepare` makes what a program holds before the call: network outputs on the GPU and the
transcripts as Python lists (a batch brings new transcripts, so their graphs are built
inside the pass), or the graphs that a program keeps over all batches (denominator and
decoding graphs; numerator graphs come from a lexicon outside this framework)."""
import itertools
import math

import numpy as np
import torch

import k2_b200 as k2
from k2_b200 import synthetic

#: search beam, output beam, min / max active states of the decoding benchmark
DECODE = dict(search_beam=20.0, output_beam=8.0, min_active=30, max_active=10000)


def _ctc(name, kind="ctc", **kw):
    """frames: longest utterance; short: the shortest one as a share of it; tokens: longest
    transcript, the shortest has 2/5 of it; sigma: spread of the logits; peak: added to the
    logit of a reference alignment (0: flat posteriors of an untrained network, 9: a trained
    one)."""
    case = dict(name=name, kind=kind, utterances=8, frames=200, short=1.0, classes=500,
                tokens=50, sigma=1.0, peak=0.0, modified=False, logits=False,
                delay_penalty=0.0, reduction="sum", double=True, beam=10.0)
    if kind == "align":
        for key in ("logits", "delay_penalty", "reduction"):
            del case[key]
    return dict(case, **kw)


def _lfmmi(name, **kw):
    return dict(dict(name=name, kind="lfmmi", utterances=16, frames=500, phones=71,
                     numerators=False, lattice=False, beam=8.0), **kw)


def _decode(name, **kw):
    return dict(dict(name=name, kind="decode", utterances=32, frames=500, classes=500,
                     states=200000, **DECODE), **kw)


def listed():
    return [
        # one short utterance: adaptation on a single sentence, a unit of a small evaluation
        _ctc("ctc_one", utterances=1, frames=80, tokens=12, peak=9.0),
        # the small benchmark configuration
        _ctc("ctc_small"),
        # the headline configuration: a full batch of long, ragged utterances
        _ctc("ctc_large", utterances=64, frames=1000, short=0.6, tokens=250, sigma=1.5),
        # modified topology and a large vocabulary
        _ctc("ctc_modified", utterances=32, frames=500, classes=5000, tokens=150, modified=True),
        # characters: few classes, an odd number of them, transcripts of hundreds of tokens
        _ctc("ctc_chars", utterances=16, frames=1500, short=0.5, classes=29, tokens=400,
             sigma=1.5, peak=6.0),
        # straight from the logits of a network with 500 pieces and a blank
        _ctc("ctc_logits", utterances=32, frames=600, short=0.4, classes=501, tokens=120,
             sigma=1.5, peak=9.0, logits=True),
        # forced alignment of a corpus with a trained network
        _ctc("align", kind="align", utterances=32, frames=800, short=0.4, tokens=200, sigma=1.5,
             peak=9.0),
        # LF-MMI as the reference's recipes do it: numerator and denominator graph of every
        # utterance in one intersection, total scores of its lattice
        _lfmmi("lfmmi_lattice", frames=300, numerators=True, lattice=True),
        # the denominator benchmark configuration
        _lfmmi("lfmmi_den", utterances=128),
        # one utterance on a small graph, as a recogniser without batching does
        _decode("decode_one", utterances=1, frames=150, states=20000),
        # the decoding benchmark configuration
        _decode("decode_large"),
        # streaming: a few streams, chunk by chunk
        dict(name="online", kind="online", utterances=4, frames=96, chunk=16, classes=500,
             states=20000, **DECODE),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ctc", "ctc", "ctc", "align", "lfmmi", "decode", "online"])
    if kind in ("ctc", "align"):
        case = _ctc("", kind=kind)
        frames = _log_int(rng, 40, 1500)
        case.update(frames=frames, utterances=_log_int(rng, 1, 64), short=round(rng.uniform(0.3, 1), 2),
                    classes=_log_int(rng, 29, 5000), tokens=max(2, int(frames * rng.uniform(0.06, 0.27))),
                    sigma=rng.choice([1.0, 1.5, 2.0]), peak=rng.choice([0.0, 6.0, 9.0]),
                    modified=rng.random() < 0.3, double=rng.random() < 0.7)
        # at most the log-probs of the largest listed case
        case["utterances"] = max(1, min(case["utterances"], 80000000 // (frames * case["classes"])))
        if case["kind"] == "ctc":
            case.update(logits=rng.random() < 0.3, reduction=rng.choice(["sum", "sum", "mean"]),
                        delay_penalty=0.1 if rng.random() < 0.2 else 0.0)
    elif kind == "lfmmi":
        case = _lfmmi("", frames=_log_int(rng, 50, 600), phones=rng.randint(35, 100),
                      numerators=rng.random() < 0.6, lattice=rng.random() < 0.4)
        case["utterances"] = _log_int(rng, 2, 24 if case["lattice"] else 128)
    else:
        case = _decode("", utterances=_log_int(rng, 1, 32 if kind == "decode" else 8),
                       frames=_log_int(rng, 50, 500), states=_log_int(rng, 2000, 200000),
                       classes=_log_int(rng, 100, 1000), search_beam=rng.choice([12.0, 16.0, 20.0]),
                       output_beam=rng.choice([4.0, 6.0, 8.0]),
                       max_active=_log_int(rng, 1000, 10000))
        if kind == "online":
            chunk = rng.randint(8, 32)
            case.update(kind="online", chunk=chunk, frames=chunk * rng.randint(2, 6),
                        states=_log_int(rng, 2000, 50000))
    del case["name"]
    return case


# --------------------------------------------------------------------------- inputs
def _logits(case, classes, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    shape = (case["utterances"], case["frames"], classes)
    return torch.randn(shape, generator=gen, device="cuda"), gen


def _segments(durations):
    """[utterance, first frame, frames], longest first as the intersection wants them."""
    order = np.argsort(-durations, kind="stable")
    return torch.from_numpy(np.stack([order, np.zeros_like(order), durations[order]],
                                     1).astype(np.int32))


def _spread(longest, short, n):
    """Lengths of n utterances, evenly between the longest and a share of it."""
    return np.maximum(2, np.linspace(longest, short * longest, n).astype(np.int64))


def _prepare_ctc(case, seed):
    rng = np.random.default_rng(seed)
    n, t, c = case["utterances"], case["frames"], case["classes"]
    dur = rng.permutation(_spread(t, case["short"], n))
    top = np.minimum(case["tokens"], dur // 3)
    lens = np.maximum(1, rng.integers(2 * top // 5, top + 1))
    symbols = [rng.integers(1, c, size=k) for k in lens]
    x, _ = _logits(case, c, seed)
    x *= case["sigma"]
    if case["peak"]:
        # every token is held for a part of its share of the frames, the rest is blank
        at = np.zeros((n, t), np.int64)
        for i in range(n):
            share = np.arange(dur[i]) * lens[i] / dur[i]
            at[i, :dur[i]] = np.where(share % 1.0 < 0.5, symbols[i][share.astype(np.int64)], 0)
        x.scatter_add_(2, torch.from_numpy(at).cuda()[:, :, None],
                       torch.full((n, t, 1), case["peak"], device="cuda"))
    seg = _segments(dur)
    order = seg[:, 0].tolist()
    state = dict(case=case, segments=seg, symbols=[symbols[i].tolist() for i in order],
                 x=x if case.get("logits") else torch.log_softmax(x, -1))
    if case.get("reduction") == "mean":
        state["target_lengths"] = torch.from_numpy(lens[order]).cuda()
    return state


def _prepare_lfmmi(case, seed):
    rng = np.random.default_rng(seed)
    n, t, p = case["utterances"], case["frames"], case["phones"]
    x, _ = _logits(case, p + 1, seed)
    rs2, arcs = synthetic.den_graph(seed, p)
    seg = _segments(np.full(n, t))
    lens = rng.integers(t // 12, t // 5 + 1, size=n)
    w = synthetic.Workload("lfmmi", x, seg, case["beam"], graph_row_splits2=rs2, graph_arcs=arcs,
                           num_symbols=[rng.integers(1, p + 1, size=k).tolist() for k in lens])
    state = dict(case=case, segments=seg, x=torch.log_softmax(x, -1))
    if case["numerators"]:
        splits1, splits2, arcs, a_to_b = synthetic.num_den_graphs(w)
        state["graphs"] = k2.Fsa(k2.RaggedArc(torch.from_numpy(arcs).cuda(),
                                              torch.from_numpy(splits1).cuda(),
                                              torch.from_numpy(splits2).cuda()))
        state["a_to_b_map"] = torch.from_numpy(a_to_b)
    else:
        state["graphs"] = synthetic.build_graphs(w, "cuda")
    return state


def _prepare_decode(case, seed):
    rng = np.random.default_rng(seed)
    x, _ = _logits(case, case["classes"], seed)
    rs2, arcs = synthetic.decoding_graph(seed, case["states"], case["classes"])
    # one arc in eight puts out a word
    words = rng.integers(1, 50000, size=len(arcs), dtype=np.int32)
    words[rng.random(len(arcs)) > 0.125] = 0
    words[arcs[:, 2] == -1] = -1
    graph = k2.Fsa(k2.RaggedArc(torch.from_numpy(arcs).cuda(),
                                torch.tensor([0, len(rs2) - 1], dtype=torch.int32).cuda(),
                                torch.from_numpy(rs2).cuda()),
                   aux_labels=torch.from_numpy(words).cuda())
    x = torch.log_softmax(2.0 * x, -1)
    state = dict(case=case, graph=graph)
    if case["kind"] == "online":
        n, chunk = case["utterances"], case["chunk"]
        state["chunks"] = [x[:, k:k + chunk].contiguous() for k in range(0, case["frames"], chunk)]
        state["segments"] = torch.tensor([[i, 0, chunk] for i in range(n)], dtype=torch.int32)
    else:
        state["x"] = x
        state["lengths"] = torch.from_numpy(_spread(case["frames"], 0.6, case["utterances"]))
    return state


def prepare(case, seed):
    if case["kind"] in ("ctc", "align"):
        return _prepare_ctc(case, seed)
    if case["kind"] == "lfmmi":
        return _prepare_lfmmi(case, seed)
    return _prepare_decode(case, seed)


# --------------------------------------------------------------------------- passes
def _run_ctc(s):
    case = s["case"]
    graphs = k2.ctc_graph(s["symbols"], modified=case["modified"], device=s["x"].device)
    x = s["x"].detach().requires_grad_(True)
    make = k2.DenseFsaVec.from_logits if case["logits"] else k2.DenseFsaVec
    loss = k2.ctc_loss(graphs, make(x, s["segments"]), output_beam=case["beam"],
                       delay_penalty=case["delay_penalty"], reduction=case["reduction"],
                       use_double_scores=case["double"], target_lengths=s.get("target_lengths"))
    loss.backward()
    return {"loss": loss.detach(), "grad": x.grad}


def _run_align(s):
    case = s["case"]
    graphs = k2.ctc_graph(s["symbols"], modified=case["modified"], device=s["x"].device)
    lattice = k2.intersect_dense(graphs, k2.DenseFsaVec(s["x"], s["segments"]), case["beam"])
    best = k2.shortest_path(lattice, use_double_scores=case["double"])
    return {"labels": best.labels, "aux_labels": best.aux_labels, "scores": best.scores,
            "states": best.arcs.row_splits(1)}


def _run_lfmmi(s):
    case, a_to_b = s["case"], s.get("a_to_b_map")
    x = s["x"].detach().requires_grad_(True)
    dense = k2.DenseFsaVec(x, s["segments"])
    if case["lattice"]:
        lattice = k2.intersect_dense(s["graphs"], dense, case["beam"], a_to_b_map=a_to_b)
        tot = lattice.get_tot_scores(log_semiring=True, use_double_scores=True)
    else:
        tot = k2.intersect_dense_tot_scores(s["graphs"], dense, case["beam"], a_to_b_map=a_to_b)
    loss = -(tot[0::2] - tot[1::2]).sum() if case["numerators"] else tot.sum()
    loss.backward()
    return {"tot_scores": tot.detach(), "grad": x.grad}


def _paths(lattice):
    """Words and alignment of the best path, total score and size of the lattice."""
    best = k2.one_best_decoding(lattice)
    words = k2.get_aux_labels(best)
    tot = lattice.get_tot_scores(log_semiring=True, use_double_scores=True)
    flat = np.zeros(best.num_arcs, np.int64)  # as many as there are frames, the rest 0
    every = list(itertools.chain.from_iterable(words))
    flat[:len(every)] = every
    return {"words": flat, "lengths": np.array([len(w) for w in words]), "labels": best.labels,
            "scores": best.scores, "tot_scores": tot, "lattice_arcs": lattice.num_arcs,
            "lattice_states": lattice.arcs.row_splits(1)}


def _run_decode(s):
    case = s["case"]
    return _paths(k2.get_lattice(s["x"], s["lengths"], s["graph"],
                                 search_beam=case["search_beam"], output_beam=case["output_beam"],
                                 min_active_states=case["min_active"],
                                 max_active_states=case["max_active"]))


def _run_online(s):
    case, n = s["case"], s["case"]["utterances"]
    decoder = k2.OnlineDenseIntersecter(s["graph"], n, case["search_beam"], case["output_beam"],
                                        case["min_active"], case["max_active"])
    states = [None] * n
    partial = []  # results are shown after every chunk
    for x in s["chunks"]:
        lattice, states = decoder.decode(k2.DenseFsaVec(x, s["segments"]), states)
        partial.append(_paths(lattice))
    return partial


_RUN = dict(ctc=_run_ctc, align=_run_align, lfmmi=_run_lfmmi, decode=_run_decode,
            online=_run_online)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# --------------------------------------------------------------------------- what a pass needs
def work(case):
    """Network output read once, its gradient (or the lattice and the best paths) written
    once, the graph arcs read once; an addition and a maximum per arc and frame in either
    direction of the exact intersections, per expanded arc of the pruned ones."""
    n, t = case["utterances"], case["frames"]
    if case["kind"] in ("ctc", "align"):
        rows = n * t * (1 + case["short"]) / 2
        states = 2 * 0.7 * min(case["tokens"], t / 3) + 2
        out = 4 * n * t * case["classes"] if case["kind"] == "ctc" else 16 * rows
        return {"bytes": 4 * rows * case["classes"] + out + 4 * n * states,
                "flops": 4 * 2.5 * states * rows}
    if case["kind"] == "lfmmi":
        arcs = (2 * case["phones"] + 1) * 32
        return {"bytes": 2 * 4 * n * t * (case["phones"] + 1) + 16 * arcs,
                "flops": 4 * arcs * n * t}
    # a lattice of beam 8 has about 260 arcs and as many states per frame on these graphs
    rows = n * t * (0.8 if case["kind"] == "decode" else 1.0)
    kept = 260 * min(1.0, case["output_beam"] / 8) * rows
    return {"bytes": 4 * rows * case["classes"] + 20 * kept + 16 * 6 * case["states"],
            "flops": 3 * 6 * min(case["max_active"], case["states"]) * rows}


def tolerance(case):
    """Totals in double and gradients as 32-bit floats; lattices, alignments and words are
    decided by 32-bit additions in a fixed order and come out the same."""
    return {"rel": 1e-5}
