"""The calls that a user of this framework makes, as measurable cases.

A case is a plain dict: the kind of call, the sizes of the reference and the query, and the options.
The sizes are those of the framework's own workloads (cusingler_b200/synth.py: small, mid, stress and
full) or lie between them.  The cells follow the same model as synth.py (negative-binomial counts with
marker blocks per label and a mean-dependent dropout, stored as log2(1 + x)), generated on the GPU.

  listed()             the cases, one for each way the framework is called
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the caller has in hand before the call (inputs, trained reference)
  run(state)           one call through the public entry points, and its outputs
  work(case)           the bytes and operations that one call cannot do without
  exact(case, seed)    the outputs that are computed numbers, in 64 bits, by plain torch
"""

from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from cusingler_b200 import abi, synth

QUANTILE, THRE = 0.8, 0.05

# label blocks as in synth.WORKLOADS: marker genes per label (least, most), factor (least, most)
BLOCK_SMALL = (60, 60, 4.0, 4.0)
BLOCK = (40, 80, 3.0, 5.0)
PRIVATE = (8, 15, 1.5)  # families: genes of a label's own (least, most), factor
CHUNK_CELLS = 1 << 27   # cells x genes drawn at once
MARKERS_PER_LABEL = 36  # score-step marker genes per label on these data, about


def _case(name, kind, n_ref, n_qry, n_genes, n_labels, density, family=0, host=False, batches=1):
    c = dict(kind=kind, n_ref=n_ref, n_qry=n_qry, n_genes=n_genes, n_labels=n_labels, density=density,
             family=family, host=host, batches=batches)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one cell from a notebook or a service: latency and launches count (host arrays, small reference)
        _case("small_one_cell", "annotate", 1900, 1, 15000, 13, 0.10, host=True),
        # the small workload in one call: an experiment of a few hundred cells against a published atlas
        _case("small_annotate", "annotate", 1900, 800, 15000, 13, 0.10, host=True),
        # the same through the drop-in module, which trains and annotates in each call
        _case("small_run", "run", 1900, 800, 15000, 13, 0.10, host=True),
        # the mid workload, plain form, query already on the GPU: the reference's own pipeline
        _case("mid_annotate", "annotate", 20000, 100000, 25000, 30, 0.06),
        # the mid workload, learned form: the proposal network decides, hard cells are fine-tuned
        _case("mid_learned", "learned", 20000, 100000, 25000, 30, 0.06),
        # first labels and label scores alone, a ragged batch (the input of the network's training too)
        _case("mid_score", "score", 20000, 12345, 25000, 30, 0.06),
        # the reference's FP32 operation order, used to compare labels with the reference's own
        _case("mid_fp32ref", "fp32ref", 20000, 1000, 25000, 30, 0.06),
        # families of near-identical labels, many fine-tune rounds (stress workload, fewer cells)
        _case("stress_annotate", "annotate", 30000, 16000, 25000, 60, 0.06, family=5),
        # host batches streamed against a large reference with 120 labels (full workload, fewer cells)
        _case("full_stream", "stream", 40000, 16384, 30000, 120, 0.05, family=6, host=True, batches=3),
        # marker training and ranking of the mid reference, once per reference and gene list
        _case("mid_train", "train", 20000, 0, 25000, 30, 0.06, host=True),
        # one epoch of the proposal network's training on labelled cells (forward, backward, AdamW)
        _case("mlp_train", "mlp_train", 0, 20000, 0, 30, 0.0, host=True),
        # label selection on score rows that another framework holds on the GPU
        _case("mid_select", "select", 20000, 8000, 0, 30, 0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["annotate", "annotate", "annotate", "learned", "score", "score", "fp32ref", "stream", "run",
                       "train", "mlp_train", "select"])
    n_genes = _log_int(rng, 4000, 30000)
    n_labels = rng.randint(5, 45)
    family = rng.choice([0, 0, 5])
    if family:
        n_labels = 5 * rng.randint(2, 10)
    n_ref = _log_int(rng, 1000, 30000)
    density = round(rng.uniform(0.05, 0.1), 3)
    host = rng.random() < 0.4
    # the largest listed cases score 2e9 pairs of cells, or 5e8 where families are fine-tuned
    most = 5e8 if family else 1.5e9
    n_qry = _log_int(rng, 1, max(2, min(80000, most / n_ref)))
    if kind == "learned":
        n_qry = max(n_qry, 500)
    if kind == "fp32ref":
        n_qry = min(n_qry, max(1, int(2e7 / n_ref)), 1500)
    if kind == "stream":
        return _case("", kind, n_ref, max(2, n_qry // 3), n_genes, n_labels, density, family, True, rng.randint(2, 4))
    if kind == "run":
        return _case("", kind, min(n_ref, 6000), min(n_qry, 6000), n_genes, n_labels, density, family, True)
    if kind == "train":
        return _case("", kind, min(n_ref, 20000), 0, min(n_genes, 25000), n_labels, density, family, True)
    if kind == "mlp_train":
        return _case("", kind, 0, _log_int(rng, 2000, 20000), 0, n_labels, 0.0, 0, True)
    if kind == "select":
        return _case("", kind, n_ref, _log_int(rng, 10, 8000), 0, n_labels, 0.0)
    return _case("", kind, n_ref, n_qry, n_genes, n_labels, density, family, host)


# ---- synthetic cells, on the GPU ----------------------------------------------------------------


@dataclasses.dataclass
class Csr:
    n_rows: int
    n_cols: int
    data: torch.Tensor     # float32
    indices: torch.Tensor  # int32
    indptr: torch.Tensor   # int32
    labels: torch.Tensor   # int64, the cells' true labels


@dataclasses.dataclass
class HostCsr:
    n_rows: int
    n_cols: int
    data: np.ndarray
    indices: np.ndarray
    indptr: np.ndarray


def _world(case, seed):
    """Gene means per label (L x W), label proportions and the dropout's midpoint."""
    rng = np.random.default_rng([seed, 7919])
    W, L, fam = case["n_genes"], case["n_labels"], case["family"]
    block = BLOCK_SMALL if case["n_ref"] < 3000 else BLOCK
    props = np.maximum(rng.dirichlet(np.ones(L)), 0.25 / L)
    mean = np.exp(rng.uniform(np.log(0.5), np.log(20.0), size=W))[None, :].repeat(L, 0)
    perm, pos = rng.permutation(W), 0
    for first in range(0, L, fam or 1):
        m = int(rng.integers(block[0], block[1] + 1))
        mean[first:first + (fam or 1), perm[pos:pos + m]] *= rng.uniform(block[2], block[3])
        pos += m
        for lab in range(first, first + fam):
            m = int(rng.integers(PRIVATE[0], PRIVATE[1] + 1))
            mean[lab, perm[pos:pos + m]] *= PRIVATE[2]
            pos += m
    mean = torch.from_numpy(mean).cuda()
    props = torch.from_numpy(props / props.sum()).cuda()
    r = 1.0 / synth.DISPERSION
    positive = 1.0 - (r / (r + mean)) ** r
    lo, hi = -10.0, 15.0
    for _ in range(40):  # the midpoint at which the stored fraction is the wanted density
        mid = 0.5 * (lo + hi)
        stored = (props[:, None] * torch.sigmoid(synth.DROPOUT_SLOPE * (mean.log() - mid)) * positive).sum(0).mean()
        lo, hi = (mid, hi) if float(stored) > case["density"] else (lo, mid)
    detect = torch.sigmoid(synth.DROPOUT_SLOPE * (mean.log() - 0.5 * (lo + hi)))
    return mean.float(), detect.float(), props.float()


def _cells(world, n, seed, every_label=False):
    """n cells of a world, as a CSR on the GPU; every_label: the first cells cover each label once."""
    mean, detect, props = world
    L, W = mean.shape
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    labels = torch.multinomial(props, n, replacement=True, generator=g)
    if every_label:
        labels[:L] = torch.arange(L, device="cuda")
    shape, data, indices, counts = 1.0 / synth.DISPERSION, [], [], []
    step = max(1, CHUNK_CELLS // W)
    for a in range(0, n, step):
        lab = labels[a:a + step]
        row, col = (torch.rand((len(lab), W), device="cuda", generator=g) < detect[lab]).nonzero(as_tuple=True)
        m = mean[lab[row], col]
        x = torch.poisson(torch._standard_gamma(torch.full_like(m, shape), generator=g) * (m / shape), generator=g)
        keep = x > 0
        data.append(torch.log2(1.0 + x[keep]))
        indices.append(col[keep].int())
        counts.append(torch.bincount(row[keep], minlength=len(lab)))
    indptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    indptr[1:] = torch.cumsum(torch.cat(counts), 0)
    return Csr(n, W, torch.cat(data), torch.cat(indices), indptr, labels)


def _host(c, pinned=False):
    """The CSR as host arrays, page-locked for streaming."""
    def one(t):
        return torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned).copy_(t).numpy()
    return HostCsr(c.n_rows, c.n_cols, one(c.data), one(c.indices), one(c.indptr))


def _dataset(case, seed):
    world = _world(case, seed)
    ref = _cells(world, case["n_ref"], 3 * seed + 1, every_label=True)
    qry = [_cells(world, case["n_qry"], 3 * seed + 2 + (1 << 40) * b) for b in range(case["batches"])] \
        if case["n_qry"] else []
    return world, ref, qry


def _mlp_rows(case, seed):
    """Label scores as the score step gives them, and the labels to learn (mostly the best score)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, L = case["n_qry"], case["n_labels"]
    scores = 0.35 + 0.08 * torch.rand((n, L), device="cuda", generator=g)
    true = torch.randint(L, (n,), device="cuda", generator=g)
    scores[torch.arange(n, device="cuda"), true] += 0.15 * torch.rand(n, device="cuda", generator=g)
    noisy = (scores + 0.01 * torch.randn((n, L), device="cuda", generator=g)).argmax(1)
    return scores.cpu().numpy(), noisy.int().cpu().numpy()


def _network(scores, targets, L, seed, hidden=256, steps=240, batch=4096):
    """Parameters of the proposal network, trained by the caller beforehand and loaded (abi.mlp_load)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.from_numpy(scores).cuda()
    x = ((x - x.amax(1, keepdim=True)) * 20.0).clamp(min=-8.0)
    y = torch.from_numpy(targets).cuda().long()
    p = []
    for rows, cols in ((hidden, L), (hidden, hidden), (L, hidden)):
        p += [(2 * torch.rand((rows, cols), device="cuda", generator=g) - 1) / math.sqrt(cols),
              torch.zeros(rows, device="cuda")]
    p = [t.requires_grad_() for t in p]
    opt = torch.optim.AdamW(p, lr=2e-3, weight_decay=0.01)
    for _ in range(steps):
        at = torch.randint(len(y), (min(batch, len(y)),), device="cuda", generator=g)
        h = torch.nn.functional.gelu(x[at] @ p[0].T + p[1])
        h = torch.nn.functional.gelu(h @ p[2].T + p[3])
        opt.zero_grad(set_to_none=True)
        torch.nn.functional.cross_entropy(h @ p[4].T + p[5], y[at]).backward()
        opt.step()
    return torch.cat([t.detach().reshape(-1) for t in p]).cpu().numpy()


def _select_scores(case, seed):
    """Score rows (queries x reference cells, labels in column ranges) as a correlation gives them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    Q, R, L = case["n_qry"], case["n_ref"], case["n_labels"]
    share = torch.rand(L, device="cuda", generator=g) + 0.1
    lens = (1 + (share / share.sum() * (R - L)).floor()).long()
    lens[0] += R - lens.sum()
    lens = lens.tolist()
    centre = 0.4 + 0.05 * torch.randn((Q, L), device="cuda", generator=g)
    at = torch.repeat_interleave(torch.arange(L, device="cuda"), torch.tensor(lens, device="cuda"))
    scores = centre[:, at] + 0.03 * torch.randn((Q, R), device="cuda", generator=g)
    starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    return scores, np.stack([starts, lens], 1).astype(np.uint32).reshape(-1)


# ---- the cases -----------------------------------------------------------------------------------


def _trained(case, ref):
    names, genes = synth.names("CT", case["n_labels"]), synth.names("G", case["n_genes"])
    a = abi.Annotator(mode=abi.MODE_FP32REF if case["kind"] == "fp32ref" else abi.MODE_EXACT)
    return a.train(_host(ref), ref.labels.cpu().numpy(), names, genes, genes)


def _query(c, host):
    if host:
        return _host(c)
    return abi.device_csr(c.n_rows, c.n_cols, c.data.data_ptr(), c.indices.data_ptr(), c.indptr.data_ptr())


def prepare(case, seed):
    kind, L = case["kind"], case["n_labels"]
    s = {"kind": kind, "case": dict(case)}
    if kind == "mlp_train":
        s["scores"], s["targets"] = _mlp_rows(case, seed)
        # the context's label count comes from a trained reference: the least one
        tiny = dict(case, n_ref=20 * L, n_qry=0, n_genes=2000, density=0.1)
        s["annotator"] = _trained(tiny, _dataset(tiny, seed)[1])
        s["seed"] = seed % 1000
        return s
    if kind == "select":
        s["rows"], s["ranges"] = _select_scores(case, seed)
        Q = case["n_qry"]
        s["out"] = (torch.empty((Q, L), device="cuda"), torch.empty(Q, dtype=torch.int32, device="cuda"),
                    torch.empty((Q, L), dtype=torch.uint8, device="cuda"))
        return s
    world, ref, qry = _dataset(case, seed)
    s["names"], s["genes"] = synth.names("CT", L), synth.names("G", case["n_genes"])
    if kind in ("train", "run"):
        s["ref"], s["celltypes"] = _host(ref), ref.labels.cpu().numpy().astype(np.int32)
        if kind == "train":
            s["annotator"] = abi.Annotator()
        else:
            s["qry"], s["cells"] = _host(qry[0]), synth.names("cell", case["n_qry"])
            s["code"] = {name: i for i, name in enumerate(s["names"])}
        return s
    s["annotator"] = a = _trained(case, ref)
    if kind == "stream":
        s["batches"] = [_host(q, pinned=True) for q in qry]
        return s
    s["keep"], s["qry"] = qry[0], _query(qry[0], case["host"])
    if kind == "learned":
        sample = _cells(world, 16384, 3 * seed + 3)
        _, final, scores = a.annotate(_query(sample, False), with_scores=True)
        a.mlp_load(_network(scores, final, L, seed), L, 256)
    return s


def _marker_tables(a, case):
    """What the training found, in arrays whose shape the case alone decides."""
    L, out = case["n_labels"], {}
    for name, what in (("common", 0), ("thre", 1)):
        out[name] = np.zeros(case["n_genes"], np.uint8)
        out[name][a.u32(what)] = 1
    for name, what in (("pair_genes", 2), ("finetune_genes", 4)):  # concatenated lists, then -1
        genes = a.u32(what)
        out[name] = np.full(512 * L * L, -1, np.int32)
        out[name][:len(genes)] = genes
    for name, what in (("pair_ranges", 3), ("finetune_ranges", 5), ("label_ranges", 6), ("row_order", 7)):
        out[name] = a.u32(what).view(np.int32)
    return out


def run(s):
    kind = s["kind"]
    if kind in ("annotate", "fp32ref"):
        first, final, scores = s["annotator"].annotate(s["qry"], QUANTILE, THRE, with_scores=True)
        return {"first": first, "final": final, "scores": scores}
    if kind == "score":
        first, scores, flags = s["annotator"].score_first(s["qry"], QUANTILE, THRE)
        return {"first": first, "scores": scores, "flags": flags}
    if kind == "learned":
        first, final, stats = s["annotator"].annotate_learned(s["qry"], QUANTILE, THRE)
        return {"first": first, "final": final, "stats": stats}
    if kind == "stream":
        first, final, _, _ = s["annotator"].annotate_stream(s["batches"], QUANTILE, THRE)
        return {"first": first, "final": final}
    if kind == "train":
        a = s["annotator"].train(s["ref"], s["celltypes"], s["names"], s["genes"], s["genes"])
        return _marker_tables(a, s["case"])
    if kind == "run":
        from cusingler import cusingler

        r, q = s["ref"], s["qry"]
        rows = cusingler.run(8, 0, r.n_rows, r.n_cols, r.data, r.indices, r.indptr, q.n_rows, q.n_cols, q.data,
                             q.indices, q.indptr, s["names"], s["celltypes"], s["cells"], s["genes"], s["genes"])
        return np.array([(s["code"][first], s["code"][final]) for _, first, final in rows], dtype=np.int32)
    if kind == "mlp_train":
        loss = s["annotator"].mlp_train(s["scores"], s["targets"], epochs=1, seed=s["seed"])
        return {"loss": loss, "params": s["annotator"].mlp_params()[0]}
    scores, first, flags = s["out"]
    status = abi.select_labels_noalloc(s["rows"].data_ptr(), s["rows"].shape[1], s["rows"].shape[0], s["ranges"],
                                       QUANTILE, THRE, scores.data_ptr(), first.data_ptr(), flags.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream)
    if status:
        raise RuntimeError(abi.STATUS_NAMES[status])
    return {"first": first, "scores": scores, "flags": flags}


def work(case):
    """Inputs read once, outputs written once; the score step's products, 2 per query, reference cell and
    marker gene (the fine-tune's depend on the data and come on top)."""
    kind, Q, R, L = case["kind"], case["n_qry"] * case["batches"], case["n_ref"], case["n_labels"]
    if kind == "select":
        return {"bytes": 4.0 * Q * R + Q * (5.0 * L + 4), "flops": 0.0}
    if kind == "mlp_train":
        params = 256 * (2 * L + 256 + 2) + L
        return {"bytes": 4.0 * Q * (L + 1) + 4.0 * params, "flops": 6.0 * Q * params}
    entry, W = 8.0 * case["density"] * case["n_genes"], case["n_genes"]
    ref = R * entry + 4.0 * R
    if kind == "train":
        return {"bytes": ref + 4.0 * L * W, "flops": 0.0}
    G = min(W, MARKERS_PER_LABEL * L)
    ref = ref if kind == "run" else 2.0 * R * G
    return {"bytes": ref + Q * (entry + 4.0 + 8.0 + 4.0 * L), "flops": 2.0 * Q * R * G}


# ---- 64-bit results ------------------------------------------------------------------------------


def _dense(c, rows, columns=None):
    """Rows [a, b) of a CSR as a dense float32 matrix, all columns or the given ones."""
    a, b = rows
    at = c.indptr[a:b + 1].long()
    out = torch.zeros((b - a, c.n_cols), device="cuda")
    row = torch.repeat_interleave(torch.arange(b - a, device="cuda"), at[1:] - at[:-1])
    out[row, c.indices[at[0]:at[-1]].long()] = c.data[at[0]:at[-1]]
    return out if columns is None else out[:, columns]


def _marker_genes(ref, L):
    """The score step's genes: per ordered label pair the first n of the genes by difference of medians."""
    n = int(math.floor(500.0 * (2.0 / 3.0) ** math.log2(L) + 0.5))
    dense = _dense(ref, (0, ref.n_rows))
    med = []
    for lab in range(L):
        v = dense[ref.labels == lab].sort(0).values
        k = len(v)
        med.append((v[k // 2] + v[k // 2 - 1]) / 2 if k % 2 == 0 else v[k // 2])
    med = torch.stack(med)
    chosen = torch.zeros(ref.n_cols, dtype=torch.bool, device="cuda")
    for lab in range(L):
        d = ((med[lab][None, :] - med).double() * 1e6).round()
        order = torch.sort(d, dim=1, descending=True, stable=True).indices[:, :n]
        order[lab] = order[lab - 1]  # a label is not compared with itself
        chosen[order.reshape(-1)] = True
    return chosen.nonzero().reshape(-1)


def _unit_ranks(c, genes):
    """Tie-averaged ranks of every row over the genes, centred and scaled to length one, in 64 bits."""
    out = []
    for a in range(0, c.n_rows, 8192):
        x = _dense(c, (a, min(a + 8192, c.n_rows)), genes).contiguous()
        order = x.sort(1).values
        rank = (torch.searchsorted(order, x) + torch.searchsorted(order, x, right=True)).double()
        rank -= rank.mean(1, keepdim=True)
        out.append(rank / rank.norm(dim=1, keepdim=True))
    return torch.cat(out)


def _quantiles(scores, pieces):
    """Per row and label the quantile of the label's scores, interpolated linearly."""
    out = []
    for columns in pieces:
        v = scores[:, columns].sort(1).values
        at = float(np.float32(QUANTILE)) * (v.shape[1] - 1)
        k = int(at)
        out.append(v[:, k] + (at - k) * (v[:, min(k + 1, v.shape[1] - 1)] - v[:, k]))
    return torch.stack(out, 1)


def exact(case, seed):
    kind, L = case["kind"], case["n_labels"]
    if kind == "select":
        rows, ranges = _select_scores(case, seed)
        pieces = [slice(int(a), int(a) + int(n)) for a, n in ranges.reshape(-1, 2)]
        got = torch.cat([_quantiles(rows[a:a + 2048].double(), pieces) for a in range(0, len(rows), 2048)])
        return {"first": None, "scores": got, "flags": None}
    if kind not in ("annotate", "fp32ref", "score"):
        return None
    _, ref, qry = _dataset(case, seed)
    genes = _marker_genes(ref, L)
    r = _unit_ranks(ref, genes)
    q = _unit_ranks(qry[0], genes)
    pieces = [(ref.labels == lab).nonzero().reshape(-1) for lab in range(L)]
    step = max(1, (1 << 27) // case["n_ref"])
    scores = torch.cat([_quantiles(q[a:a + step] @ r.T, pieces) for a in range(0, len(q), step)]).cpu().numpy()
    if kind == "score":
        return {"first": None, "scores": scores, "flags": None}
    return {"first": None, "final": None, "scores": scores}
