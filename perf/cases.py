"""The work that users of this package have it do, as measurable cases.

A protein-sequencing lab classifies the reads of a run (`classify hmm|nn|
hybrid`, or the learned proposal in front of the HMM), fits the error model
to control peptides (`fit`, with bootstrap rounds), trains the proposal
network, and simulates dye-track training sets (`simulate dt`).  Each case
goes through the Python front of the C ABI (whatprot_gb300.capi) as such a
program does.  Reads come from a seeded simulator of the same generative
model (dud, detach, Edman failure, bleaching; normal intensities), written
here in torch so that inputs do not depend on the package.

What the package computes in FP32 and only adds up over reads in FP64 (the
expected counts of a fit) is returned as float32: that is the precision that
the values carry.  Classification scores are returned as they are given.
"""
import functools
import math
import sys

import numpy as np
import torch

from whatprot_gb300 import capi
from whatprot_gb300.model import ChannelModel, DyeSeqSet, SequencingModel

DEV = "cuda"
CUTOFF = 5.0
UNPRUNED = sys.float_info.max


def listed():
    return [
        # A single read as it comes off the instrument, on the small assay
        # (2 channels, 8 timesteps, 100 dye-seqs): latency.
        {"name": "classify_one_read", "kind": "classify", "call": "host", "reads": 1, "peptides": 100, "channels": 2,
         "timesteps": 8, "min_len": 6, "max_len": 12, "most": 15, "pruned": True, "block": 0.0, "interactions": False},
        # A whole run of reads already on the device against a peptide set
        # (the benchmark's batch): throughput.
        {"name": "classify_run", "kind": "classify", "call": "device", "reads": 100000, "peptides": 1000,
         "channels": 3, "timesteps": 16, "min_len": 8, "max_len": 30, "most": 5, "pruned": True, "block": 0.0,
         "interactions": False},
        # A field of view from host memory with a model that has blocked
        # N-termini, at sizes that are multiples of nothing.
        {"name": "classify_blocked", "kind": "classify", "call": "host", "reads": 3001, "peptides": 333,
         "channels": 2, "timesteps": 13, "min_len": 5, "max_len": 22, "most": 7, "pruned": True, "block": 0.03,
         "interactions": False},
        # The command line's default: no pruning cutoff given, every state of
        # every pair is computed.
        {"name": "classify_unpruned", "kind": "classify", "call": "host", "reads": 400, "peptides": 200,
         "channels": 3, "timesteps": 16, "min_len": 8, "max_len": 30, "most": 5, "pruned": False, "block": 0.0,
         "interactions": False},
        # `classify nn` on a mid-sized training set, the best ids per read.
        {"name": "nn_kdtree", "kind": "nn", "reads": 2000, "peptides": 1000, "channels": 2, "timesteps": 12,
         "min_len": 6, "max_len": 20, "most": 5, "per_peptide": 100, "k": 1000, "h": 50, "selection": "kdtree"},
        # `classify hybrid` at the size of its configuration (20,000 dye-seqs,
        # 2,000,000 simulated dye-tracks, k = 10,000, H = 1,000), the
        # reference's k-hit set.
        {"name": "hybrid_kdtree", "kind": "hybrid", "reads": 4000, "peptides": 20000, "channels": 3, "timesteps": 16,
         "min_len": 8, "max_len": 30, "most": 5, "per_peptide": 100, "k": 10000, "h": 1000, "selection": "kdtree"},
        # The same classifier with the distance-ordered k-hit set, a smaller
        # peptide set and a ragged batch.
        {"name": "hybrid_prefix", "kind": "hybrid", "reads": 10007, "peptides": 5000, "channels": 3, "timesteps": 12,
         "min_len": 8, "max_len": 30, "most": 5, "per_peptide": 60, "k": 3000, "h": 300, "selection": "prefix"},
        # The learned proposal in front of the HMM at its configured size
        # (48 -> 1024 -> 1024 -> 20,000 logits, the top 200 rescored).
        {"name": "learned_hybrid", "kind": "learned", "reads": 20000, "peptides": 20000, "channels": 3,
         "timesteps": 16, "min_len": 8, "max_len": 30, "most": 5, "hidden": 1024, "h": 200},
        # Training that network: steps of 4,096 freshly simulated reads, then
        # its weights read back to be saved.
        {"name": "proposal_train", "kind": "train", "steps": 64, "batch": 4096, "peptides": 20000, "channels": 3,
         "timesteps": 16, "min_len": 8, "max_len": 30, "most": 5, "hidden": 1024},
        # One Baum-Welch E-step of a fit of the whole model on a control
        # peptide (20 positions, 4/3/3 dyes), rates and emission statistics.
        {"name": "fit_estep", "kind": "fit", "reads": 50000, "channels": 3, "timesteps": 16, "length": 20,
         "dyes": "433", "emission": False, "block": 0.0},
        # The E-steps of 20 bootstrap rounds of a fit on a small sample.
        {"name": "fit_bootstrap", "kind": "bootstrap", "rounds": 20, "reads": 701, "channels": 2, "timesteps": 10,
         "length": 12, "dyes": "32", "block": 0.0},
        # `simulate dt`: the hybrid's training set generated, deduplicated
        # and downloaded.
        {"name": "simulate_dye_tracks", "kind": "tracks", "peptides": 20000, "channels": 3, "timesteps": 16,
         "min_len": 8, "max_len": 30, "most": 5, "per_peptide": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["classify", "classify", "classify", "nn", "hybrid", "hybrid", "learned", "train", "fit", "fit",
                       "bootstrap", "tracks"])
    C = rng.choice([1, 2, 3, 3, 4])
    T = rng.randint(6, 16)
    case = {"kind": kind, "channels": C, "timesteps": T}
    if kind in ("fit", "bootstrap"):
        dyes = [rng.randint(1, 4) for _ in range(min(C, 3))]
        case["channels"] = len(dyes)
        case["dyes"] = "".join(str(d) for d in dyes)
        case["length"] = sum(dyes) + rng.randint(1, 10)
        case["block"] = rng.choice([0.0, 0.0, 0.02])
        if kind == "fit":
            case["reads"] = _log(rng, 300, 50000)
            case["emission"] = rng.random() < 0.5
        else:
            case["rounds"] = rng.randint(5, 40)
            case["reads"] = _log(rng, 100, 3000)
        return case
    lo = rng.randint(5, 10)
    case["min_len"], case["max_len"], case["most"] = lo, lo + rng.randint(3, 22), rng.randint(3, 5)
    if kind == "classify":
        case["pruned"] = rng.random() < 0.8
        case["call"] = rng.choice(["host", "device"])
        case["block"] = rng.choice([0.0, 0.0, 0.02, 0.05])
        case["interactions"] = rng.random() < 0.2
        case["peptides"] = _log(rng, 20, 1500 if case["pruned"] else 150)
        most = 30_000_000 if case["pruned"] else 60_000
        case["reads"] = _log(rng, 1, max(2, min(100000, most // case["peptides"])))
    elif kind in ("nn", "hybrid"):
        case["peptides"] = _log(rng, 200, 5000)
        case["per_peptide"] = rng.randint(20, 100)
        case["k"] = _log(rng, 50, max(60, min(10000, case["peptides"] * case["per_peptide"] // 40)))
        case["h"] = _log(rng, 1, min(1000, case["peptides"] // 2))
        case["reads"] = _log(rng, 1, 10000)
        case["selection"] = rng.choice(["kdtree", "kdtree", "prefix"])
    elif kind == "learned":
        case["peptides"] = _log(rng, 500, 20000)
        case["hidden"] = rng.choice([256, 512, 1024])
        case["h"] = _log(rng, 10, min(500, case["peptides"] // 3))
        case["reads"] = _log(rng, 1, 20000)
    elif kind == "train":
        case["peptides"] = _log(rng, 200, 20000)
        case["hidden"] = rng.choice([256, 512, 1024])
        case["batch"] = 64 * rng.randint(4, 64)
        case["steps"] = rng.randint(4, 64)
    else:
        case["peptides"] = _log(rng, 100, 20000)
        case["per_peptide"] = rng.randint(10, 100)
    return case


# ------------------------------------------------------------------ inputs


def _model(case):
    """The error model of the benchmark configurations, with the options that
    the case asks for."""
    C, b = case["channels"], case.get("block", 0.0)
    sm = SequencingModel(0.06, 0.05, 0.0, 0.0, b, b / 2, [])
    inter = [0.97 if case.get("interactions") else 1.0] * C
    for _ in range(C):
        sm.channel_models.append(ChannelModel(0.05, 0.07, 0.00667, 1.0, 0.16, list(inter), [1.0] * C))
    return sm


@functools.lru_cache(maxsize=8)
def _peptides(num, C, lo, hi, most):
    """num dye-seqs of lo .. hi positions as a -1 padded matrix [num, hi] and their
    lengths: each position carries a given channel's dye with probability 0.1,
    at most `most` per channel and at least one dye.  (A peptide set is the
    lab's database: it does not change from run to run.)"""
    rng = np.random.default_rng(1234 + 7 * num + C)
    rows, lens = [], []
    have = 0
    while have < num:
        n = 2 * num + 64
        L = rng.integers(lo, hi + 1, n)
        u = rng.random((n, hi))
        s = np.floor(u * 10).astype(np.int16)
        s[(s >= C) | (np.arange(hi)[None, :] >= L[:, None])] = -1
        per = np.stack([(s == c).sum(1) for c in range(C)], 1)
        ok = (per.max(1) <= most) & (per.sum(1) >= 1)
        s = s[ok]
        rows.append(s)
        lens.append(hi - np.argmax(s[:, ::-1] >= 0, axis=1))  # trailing unlabeled positions are trimmed
        have += len(s)
    return np.concatenate(rows)[:num], np.concatenate(lens)[:num].astype(np.int64)


def _peptide_set(case):
    mat, lens = _peptides(case["peptides"], case["channels"], case["min_len"], case["max_len"], case["most"])
    n = len(lens)
    return DyeSeqSet(case["channels"], [mat[i, :lens[i]] for i in range(n)], np.arange(n, dtype=np.int32),
                     np.ones(n, np.int32)), mat, lens


def _fit_peptide(case):
    """A control peptide: `length` positions, the given number of dyes of
    each channel at seeded places."""
    rng = np.random.default_rng(4)
    seq = np.full(case["length"], -1, np.int16)
    pos = rng.permutation(case["length"])
    at = 0
    for c, d in enumerate(case["dyes"]):
        seq[pos[at:at + int(d)]] = c
        at += int(d)
    return seq


def _reads(sm, mat, T, num, seed):
    """num reads [num, T, C] (float64, on the device) of peptides drawn from
    the rows of mat, and the rows drawn: duds, blocking, and per timestep
    detachment, Edman failure and bleaching; reads without a dye at the first
    timestep are not seen by the instrument."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2 + 1)
    C, L = sm.num_channels, mat.shape[1]
    M = torch.from_numpy(np.ascontiguousarray(mat)).to(DEV).long()
    kept, kept_rows, have = [], [], 0
    while have < num:
        n = int(1.3 * (num - have)) + 64
        rows = torch.randint(len(M), (n,), generator=g, device=DEV)
        s = M[rows]
        s = torch.where(torch.rand(s.shape, generator=g, device=DEV) < sm.channel_models[0].p_dud, -1, s)
        pos = torch.arange(L, device=DEV)[None, :]
        e = torch.zeros(n, dtype=torch.long, device=DEV)
        blocked = torch.rand(n, generator=g, device=DEV) < sm.p_initial_block
        tracks = torch.zeros(n, T, C, dtype=torch.float64, device=DEV)
        for t in range(T):
            for c in range(C):
                tracks[:, t, c] = ((s == c) & (pos >= e[:, None])).sum(1)
            u = torch.rand(3, n, generator=g, device=DEV)
            blocked |= u[0] < sm.p_cyclic_block
            e = torch.where(u[1] < sm.p_detach_at(t), L, e)
            e = torch.where(blocked | (u[2] < sm.p_edman_failure), e, e + 1)
            s = torch.where(torch.rand(s.shape, generator=g, device=DEV) < sm.channel_models[0].p_bleach, -1, s)
        seen = tracks[:, 0].sum(1) > 0
        kept.append(tracks[seen])
        kept_rows.append(rows[seen])
        have += int(seen.sum())
    tracks, rows = torch.cat(kept)[:num], torch.cat(kept_rows)[:num]
    mu = _adjusted_mu(sm, tracks)
    cm = sm.channel_models[0]
    sig = torch.sqrt(cm.bg_sig ** 2 + mu * cm.sig ** 2)
    return mu + sig * torch.randn(mu.shape, generator=g, device=DEV, dtype=torch.float64), rows


def _adjusted_mu(sm, n):
    """Mean intensity of dye counts n [..., C]: mu n, times the channel's
    interaction factors for the other dyes present."""
    out = []
    for c, cm in enumerate(sm.channel_models):
        mu = cm.mu * n[..., c]
        for o in range(n.shape[-1]):
            if cm.interactions[o] != 1.0:
                k = (n[..., o] - 1).clamp(min=0) if o == c else n[..., o]
                mu = mu * cm.interactions[o] ** k
        out.append(mu)
    return torch.stack(out, -1)


def _context(case, ds):
    ctx = capi.Context(0)
    ctx.upload_model(_model(case), case["timesteps"])
    if ds is not None:
        ctx.upload_peptides(ds)
    return ctx


def _on_device(state, reads):
    state["d_rads"] = reads.contiguous()
    n = len(reads)
    state["d_id"] = torch.empty(n, dtype=torch.int32, device=DEV)
    state["d_score"] = torch.empty(n, dtype=torch.float64, device=DEV)
    state["d_total"] = torch.empty(n, dtype=torch.float64, device=DEV)


def _proposal_weights(case, mat, hidden):
    """Weights with which the network proposes sensibly without training:
    random features, and as each peptide's output row the features of its
    mean read (a nearest-mean classifier)."""
    C, T, P = case["channels"], case["timesteps"], len(mat)
    g = torch.Generator(device=DEV)
    g.manual_seed(99)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    W1 = normal(hidden, 64) * 0.25
    W1[:, T * C:] = 0
    b1, b2 = normal(hidden) * 0.5, normal(hidden) * 0.5
    W2 = normal(hidden, hidden) * (1.5 / math.sqrt(hidden))
    M = torch.from_numpy(np.ascontiguousarray(mat)).to(DEV)
    pos = torch.arange(M.shape[1], device=DEV)[None, :]
    mean = torch.zeros(P, 64, device=DEV)
    for t in range(T):
        for c in range(C):
            here = ((M == c) & (pos >= int(0.94 * t + 0.5))).sum(1)
            mean[:, t * C + c] = here * 0.93 * 0.95 ** t * 0.95 ** t
    gelu = torch.nn.functional.gelu
    feats = gelu(gelu(mean @ W1.T + b1) @ W2.T + b2)
    feats = feats - feats.mean(0)
    scale = 40.0 / feats.square().sum(1).mean()
    Ppad = (P + 63) // 64 * 64
    W3, b3 = torch.zeros(Ppad, hidden, device=DEV), torch.zeros(Ppad, device=DEV)
    W3[:P] = feats * scale
    b3[:P] = -0.5 * scale * feats.square().sum(1)
    return [x.cpu().numpy() for x in (W1, b1, W2, b2, W3, b3)]


def prepare(case, seed):
    kind, T = case["kind"], case["timesteps"]
    state = {"case": case}
    sm = _model(case)
    if kind in ("fit", "bootstrap"):
        seq = _fit_peptide(case)
        reads, _ = _reads(sm, seq[None, :], T, case["reads"], seed)
        ctx = _context(case, None)
        ctx.fit_begin(seq, reads.cpu().numpy())
        if kind == "fit":
            ctx.fit_set_emission(case["emission"])
        else:
            rng = np.random.default_rng(seed)
            state["idx"] = rng.integers(0, case["reads"], (case["rounds"], case["reads"])).astype(np.int32)
            state["models"] = [_round_model(case, i) for i in range(case["rounds"])]
        state["ctx"] = ctx
        return state
    ds, mat, _ = _peptide_set(case)
    ctx = state["ctx"] = _context(case, ds)
    if kind == "tracks":
        state["seed"] = int(seed) + 1
        n = case["peptides"] * case["per_peptide"]
        state["buffers"] = buf = capi.DyeTrackBuffers(n, n, T, case["channels"])
        for x in (buf.counts, buf.off, buf.sid, buf.scnt, buf.shit):
            x.fill(0)
        return state
    if kind == "train":
        state["net"] = capi.ProposalNet(ctx, hidden=case["hidden"], seed=11)
        state["seed"] = int(seed) + 1
        return state
    reads, _ = _reads(sm, mat, T, case["reads"], seed)
    if kind in ("nn", "hybrid"):
        ctx.simulate_dye_track_set(case["per_peptide"], seed=4321, to_nn=True, download=False)
        ctx.set_nn_selection(case["selection"])
        if kind == "nn":
            state["rads"] = reads.cpu().numpy()
        else:
            _on_device(state, reads)
    elif kind == "learned":
        net = state["net"] = capi.ProposalNet(ctx, hidden=case["hidden"], seed=11)
        for i, w in enumerate(_proposal_weights(case, mat, case["hidden"])):
            net.set(i, w)
        _on_device(state, reads)
    elif case["call"] == "host":
        state["rads"] = reads.cpu().numpy()
    else:
        _on_device(state, reads)
    torch.cuda.synchronize()
    return state


def _round_model(case, i):
    """Where round i of a bootstrap stands after some iterations: a model
    near the others'."""
    sm = _model(case)
    rng = np.random.default_rng(100 + i)
    sm.p_edman_failure *= rng.uniform(0.8, 1.2)
    sm.p_detach *= rng.uniform(0.8, 1.2)
    for cm in sm.channel_models:
        cm.p_bleach *= rng.uniform(0.8, 1.2)
        cm.p_dud *= rng.uniform(0.8, 1.2)
    return sm


# --------------------------------------------------------------------- run


def _sums(case, s, sum_logp, num_zero):
    d = s.as_dict(case["timesteps"], case["channels"])
    out = {k: np.asarray(v, np.float32) for k, v in d.items()}
    out["sum_logp"] = np.float32(sum_logp)
    out["num_zero"] = int(num_zero)
    return out


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "classify":
        cutoff = CUTOFF if case["pruned"] else UNPRUNED
        if case["call"] == "host":
            ids, score, total, log_score = ctx.classify(state["rads"], cutoff)
            return {"id": ids, "score": score, "total": total, "log_score": log_score}
        ctx.classify_device(state["d_rads"].data_ptr(), case["reads"], cutoff, state["d_id"].data_ptr(),
                            state["d_score"].data_ptr(), state["d_total"].data_ptr())
        return {"id": state["d_id"], "score": state["d_score"], "total": state["d_total"]}
    if kind == "nn":
        n, ids, scores, total = ctx.nn_classify(state["rads"], case["k"], 0.5, case["h"])
        return {"n": n, "ids": ids, "scores": scores, "total": total}
    if kind == "hybrid":
        ctx.hybrid_classify_device(state["d_rads"].data_ptr(), case["reads"], case["k"], 0.5, case["h"], CUTOFF,
                                   state["d_id"].data_ptr(), state["d_score"].data_ptr(), state["d_total"].data_ptr())
        return {"id": state["d_id"], "score": state["d_score"], "total": state["d_total"]}
    if kind == "learned":
        state["net"].hybrid_classify_device(state["d_rads"].data_ptr(), case["reads"], case["h"], CUTOFF,
                                            state["d_id"].data_ptr(), state["d_score"].data_ptr(),
                                            state["d_total"].data_ptr())
        return {"id": state["d_id"], "score": state["d_score"], "total": state["d_total"]}
    if kind == "train":
        net = state["net"]
        loss = net.train(case["steps"] * case["batch"], batch=case["batch"], lr=1e-3, seed=state["seed"])
        return {"loss": np.float32(loss), "weights": [net.get(i) for i in range(6)]}
    if kind == "fit":
        s, sum_logp, num_zero = ctx.fit_estep()
        out = _sums(case, s, sum_logp, num_zero)
        if case["emission"]:
            for k, v in zip(("w", "x", "xx"), ctx.fit_emission_sums().arrays(case["channels"])):
                out["emission_" + k] = v.astype(np.float32)
        return out
    if kind == "bootstrap":
        sums, sum_logp, num_zero = ctx.fit_estep_batch(state["models"], state["idx"])
        each = [_sums(case, s, a, b) for s, a, b in zip(sums, sum_logp, num_zero)]
        return {k: np.stack([np.asarray(d[k]) for d in each]) for k in each[0]}
    dts = ctx.simulate_dye_track_set(case["per_peptide"], seed=state["seed"], into=state["buffers"])
    # how many distinct tracks there are depends on the seed: the buffers
    # whole, zero beyond the set's end
    buf = state["buffers"]
    return {"num_tracks": len(dts.tracks), "num_sources": len(dts.src_id), "tracks": buf.counts, "src_off": buf.off,
            "src_id": buf.sid, "src_count": buf.scnt, "src_hits": buf.shit}


# -------------------------------------------------------------------- work


def _mean_states(case):
    """States per Edman slice of a mean dye-seq: the box of its dye counts."""
    mat, _ = _peptides(case["peptides"], case["channels"], case["min_len"], case["max_len"], case["most"])
    per = np.stack([(mat == c).sum(1) for c in range(case["channels"])], 1)
    return float(np.prod(per + 1, axis=1).mean())


def work(case):
    kind, C, T = case["kind"], case["channels"], case["timesteps"]
    row = 8 * T * C
    if kind == "classify":
        pairs = case["reads"] * case["peptides"]
        # per visited state and timestep: Edman, detachment and emission, and
        # one multiply-add of the bleaching per channel; pruning leaves about a
        # third of the pairs, with a state or two per Edman slice
        states, share = (_mean_states(case), 1.0) if not case["pruned"] else (2.0, 0.33)
        flops = pairs * share * states * T * (T + 1) / 2 * (9 + 2 * C)
        return {"bytes": case["reads"] * (row + 20), "flops": flops}
    if kind in ("nn", "hybrid"):
        # a distance to every distinct dye-track (about half of those drawn)
        n = 0.5 * case["peptides"] * case["per_peptide"]
        flops = 2.0 * case["reads"] * n * T * C
        if kind == "hybrid":
            flops += case["reads"] * case["h"] * 0.9 * 2 * T * (T + 1) / 2 * (9 + 2 * C)
        out = 12 * case["h"] + 12 if kind == "nn" else 20
        return {"bytes": n * (T * C + 12) + case["reads"] * (row + out), "flops": flops}
    if kind in ("learned", "train"):
        H, P = case["hidden"], case["peptides"]
        weights = 64 * H + H * H + H * P
        if kind == "learned":
            flops = 2.0 * case["reads"] * weights + case["reads"] * case["h"] * 0.9 * 2 * T * (T + 1) / 2 * (9 + 2 * C)
            return {"bytes": 2 * weights + case["reads"] * (row + 20), "flops": flops}
        n = case["steps"] * case["batch"]
        return {"bytes": case["steps"] * 28.0 * weights + 4.0 * weights, "flops": 6.0 * n * weights}
    if kind in ("fit", "bootstrap"):
        S = float(np.prod([int(d) + 1 for d in case["dyes"]])) * (2 if case["block"] else 1)
        n = case["reads"] * case.get("rounds", 1)
        # forward, backward and the expected counts
        return {"bytes": n * row, "flops": 3.0 * n * S * T * (T + 1) / 2 * (9 + 4 * C)}
    n = case["peptides"] * case["per_peptide"]
    # half of the drawn tracks are distinct, and each has a few sources
    return {"bytes": n * (0.5 * 2 * T * C + 0.5 * 4 + 0.8 * 12), "flops": n * T * (4 + case["max_len"] * 0.3)}


# ------------------------------------------------------------------- exact


def _emission(sm, reads, dmax, cutoff):
    """Per read, timestep and channel the density of the intensity given 0 ..
    dmax live dyes, [R, T, C, dmax + 1], zero outside the pruning window (no
    interactions), and that window's lower ends."""
    cm = sm.channel_models[0]
    n = torch.arange(dmax + 1, dtype=torch.float64, device=DEV)
    mu = cm.mu * n
    sig = torch.sqrt(cm.bg_sig ** 2 + mu * cm.sig ** 2)
    x = reads[..., None]
    pr = torch.exp(-(x - mu) ** 2 / (2 * sig ** 2)) / (sig * math.sqrt(2 * math.pi))
    if cutoff == UNPRUNED:
        return pr
    above = mu + cutoff * sig > x
    lo = torch.where(above.any(-1), above.int().argmax(-1), dmax + 1)
    beyond = (mu - cutoff * sig > x) & (n >= lo[..., None])
    hi = torch.where(beyond.any(-1), beyond.int().argmax(-1), dmax + 1)
    inside = (n >= lo[..., None]) & (n < hi[..., None])
    return pr * inside


def _binomial(q, s, n):
    """Lower triangular [n + 1, n + 1]: from -> to, each dye lost with
    probability q (s = 1 - q, kept apart so that both can be differentiated)."""
    rows = []
    for i in range(n + 1):
        rows.append(torch.stack([math.comb(i, j) * q ** (i - j) * s ** j if j <= i else torch.zeros_like(q)
                                 for j in range(n + 1)]))
    return torch.stack(rows)


def _forward(sm, seq, T, pr, rate):
    """log P [R] of one dye-seq in 64 bits: state [R, Edman cuts, dye counts
    ...] for free and blocked N-termini, and the detached mass.  `rate` holds
    the probabilities of every event and of its absence.  pr: [R, T, C, n]."""
    C, R = sm.num_channels, len(pr)
    D = [int((seq == c).sum()) for c in range(C)]
    shape = [d + 1 for d in D]
    left = np.zeros((T + 1, C), int)  # dyes at positions >= t
    for t in range(T + 1):
        for c in range(C):
            left[t, c] = int((seq[t:] == c).sum())
    nonzero = torch.ones(shape, dtype=torch.bool, device=DEV)
    nonzero.view(-1)[0] = False
    blocks = sm.p_initial_block > 0 or sm.p_cyclic_block > 0

    def along(x, M, c):  # x over counts of channel c times M [from, to]
        return torch.movedim(torch.tensordot(torch.movedim(x, 2 + c, -1), M, dims=([-1], [0])), -1, 2 + c)

    def weight(t):
        w = pr[:, t, 0, :shape[0]]
        for c in range(1, C):
            w = w[..., None] * pr[:, t, c, :shape[c]].reshape([R] + [1] * c + [shape[c]])
        return w[:, None]

    start = torch.zeros([R, 1] + shape, dtype=torch.float64, device=DEV)
    start.view(R, -1)[:, -1] = 1.0
    a = start * rate["no_init_block"]
    b = start * rate["init_block"] if blocks else None
    for c in range(C):
        M = _binomial(rate["dud"][c], rate["no_dud"][c], D[c])
        a = along(a, M, c)
        b = along(b, M, c) if blocks else None
    det = torch.zeros(R, dtype=torch.float64, device=DEV)
    log_p = torch.zeros(R, dtype=torch.float64, device=DEV)
    for t in range(T):
        if t > 0:
            if blocks:
                b = b + a * rate["cyc_block"]
            a = a * rate["no_cyc_block"]
            both = a.sum(1) + b.sum(1) if blocks else a.sum(1)
            dims = list(range(1, both.dim()))
            some = both * nonzero
            det = (det + some.sum(dims) * rate["detach"][t - 1] +
                   (both * ~nonzero).sum(dims) * sm.p_detach_at(t - 1))
            keep = torch.where(nonzero, rate["no_detach"][t - 1], 1 - sm.p_detach_at(t - 1))
            a = a * keep
            b = b * keep if blocks else None
            for c in range(C):
                M = _binomial(rate["bleach"][c], rate["no_bleach"][c], D[c])
                a = along(a, M, c)
                b = along(b, M, c) if blocks else None
            fail = torch.where(nonzero, rate["edman_fail"], sm.p_edman_failure)
            good = torch.where(nonzero, rate["edman"], 1 - sm.p_edman_failure)
            slices = [a[:, e] * fail for e in range(t)] + [torch.zeros_like(a[:, 0])]
            for e in range(t):
                moved = a[:, e] * good
                c = int(seq[e]) if e < len(seq) else -1
                if c < 0:
                    slices[e + 1] = slices[e + 1] + moved
                    continue
                n = torch.arange(shape[c], dtype=torch.float64, device=DEV).reshape([-1] + [1] * (C - 1 - c))
                ratio = (n / left[e, c]).clamp(max=1.0)
                slices[e + 1] = slices[e + 1] + moved * (1 - ratio)
                down = torch.narrow(moved * ratio, 1 + c, 1, shape[c] - 1)
                pad = [0, 0] * (C - 1 - c) + [0, 1]
                slices[e + 1] = slices[e + 1] + torch.nn.functional.pad(down, pad)
            a = torch.stack(slices, 1)
            if blocks:
                b = torch.cat([b, torch.zeros_like(b[:, :1])], 1)
        w = weight(t)
        a = a * w
        b = b * w if blocks else None
        det = det * w.reshape(R, -1)[:, 0]
        total = a.flatten(1).sum(1) + det + (b.flatten(1).sum(1) if blocks else 0)
        with torch.no_grad():
            scale = torch.where(total > 0, total.detach(), 1.0)
        log_p = log_p + torch.log(scale)
        inv = 1 / scale
        a = a * inv.reshape([R] + [1] * (a.dim() - 1))
        b = b * inv.reshape([R] + [1] * (b.dim() - 1)) if blocks else None
        det = det * inv
    total = a.flatten(1).sum(1) + det + (b.flatten(1).sum(1) if blocks else 0)
    return log_p + torch.log(total)


def _rates(sm, T, grad):
    def v(x):
        return torch.tensor(x, dtype=torch.float64, device=DEV, requires_grad=grad)

    p = {"edman_fail": sm.p_edman_failure, "init_block": sm.p_initial_block, "cyc_block": sm.p_cyclic_block}
    r = {k: v(x) for k, x in p.items()}
    r.update({"edman": v(1 - sm.p_edman_failure), "no_init_block": v(1 - sm.p_initial_block),
              "no_cyc_block": v(1 - sm.p_cyclic_block)})
    r["detach"] = [v(sm.p_detach_at(t)) for t in range(T - 1)]
    r["no_detach"] = [v(1 - sm.p_detach_at(t)) for t in range(T - 1)]
    for name in ("bleach", "dud"):
        q = [getattr(cm, "p_" + name) for cm in sm.channel_models]
        r[name], r["no_" + name] = [v(x) for x in q], [v(1 - x) for x in q]
    return r


def _expected_counts(sm, case, seq, reads, chosen=None):
    """The E-step's expected counts in 64 bits: the expected number of times
    an event with probability p happens is p times the derivative of the
    log-likelihood in p, event and absence taken as independent factors."""
    T, C = case["timesteps"], case["channels"]
    dmax = max(int(d) for d in case["dyes"])
    weight = (torch.ones(len(reads), dtype=torch.float64, device=DEV) if chosen is None
              else torch.bincount(chosen, minlength=len(reads)).double())
    out = {}

    def add(k, x):
        out[k] = out[k] + x if k in out else x

    for r0 in range(0, len(reads), 4096):
        part, w = reads[r0:r0 + 4096], weight[r0:r0 + 4096]
        rate = _rates(sm, T, True)
        pr = _emission(sm, part, dmax, UNPRUNED).requires_grad_(bool(case.get("emission")))
        log_p = _forward(sm, seq, T, pr, rate)
        ll = (log_p * w).sum()
        ll.backward()

        def n(x):
            return float(x.detach() * x.grad) if x.grad is not None else 0.0

        def pair(name, ev, no):
            add(name + "_num", np.array([n(x) for x in ev]))
            add(name + "_den", np.array([n(x) + n(y) for x, y in zip(ev, no)]))

        pair("edman", [rate["edman_fail"]], [rate["edman"]])
        pair("init_block", [rate["init_block"]], [rate["no_init_block"]])
        pair("cyc_block", [rate["cyc_block"]], [rate["no_cyc_block"]])
        pair("bleach", rate["bleach"], rate["no_bleach"])
        pair("dud", rate["dud"], rate["no_dud"])
        add("detach_x", np.array([n(x) for x in rate["detach"]]))
        add("detach_n", np.array([n(x) + n(y) for x, y in zip(rate["detach"], rate["no_detach"])]))
        add("sum_logp", float(ll.detach()))
        if case.get("emission"):
            g = pr.detach() * pr.grad
            for k, x in (("w", torch.ones_like(part)), ("x", part), ("xx", part * part)):
                full = np.zeros((C, capi.WP_EMIS_N))
                full[:, :dmax + 1] = (g * x[..., None]).sum((0, 1)).cpu().numpy()
                add("emission_" + k, full)
    for k in ("edman", "init_block", "cyc_block"):
        for e in ("_num", "_den"):
            out[k + e] = float(out[k + e][0])
    out["num_zero"] = None
    return {k: v if v is None else np.asarray(v, np.float64) for k, v in out.items()}


def exact(case, seed):
    kind, T = case["kind"], case["timesteps"]
    sm = _model(case)
    if kind in ("fit", "bootstrap"):
        seq = _fit_peptide(case)
        reads, _ = _reads(sm, seq[None, :], T, case["reads"], seed)
        if kind == "fit":
            return _expected_counts(sm, case, seq, reads)
        rng = np.random.default_rng(seed)
        idx = rng.integers(0, case["reads"], (case["rounds"], case["reads"])).astype(np.int32)
        each = [_expected_counts(_round_model(case, i), case, seq, reads, torch.from_numpy(idx[i]).long().to(DEV))
                for i in range(case["rounds"])]
        return {k: None if each[0][k] is None else np.stack([d[k] for d in each]) for k in each[0]}
    # which dye-tracks the k hits are, and which peptides a bf16 network
    # proposes, is not a matter of 64 bits; a training run draws its own reads
    if kind != "classify" or case["interactions"] or case["reads"] * case["peptides"] > 4_000_000:
        return None
    _, mat, _ = _peptide_set(case)
    reads, _ = _reads(sm, mat, T, case["reads"], seed)
    rate = _rates(sm, T, False)
    dmax = int(max((mat == c).sum(1).max() for c in range(case["channels"])))
    cutoff = CUTOFF if case["pruned"] else UNPRUNED
    best = torch.full((len(reads),), -math.inf, dtype=torch.float64, device=DEV)
    total = torch.zeros(len(reads), dtype=torch.float64, device=DEV)
    with torch.no_grad():
        pr = _emission(sm, reads, dmax, cutoff)
        for row in mat:
            log_p = _forward(sm, row, T, pr, rate)
            best = torch.maximum(best, log_p)
            total += torch.exp(log_p)
    out = {"id": None, "score": torch.exp(best), "total": total}
    if case["call"] == "host":
        out["log_score"] = best
    # a read that no peptide explains: score 0 of 1
    nothing = total == 0
    out["total"] = torch.where(nothing, 1.0, total)
    return out
