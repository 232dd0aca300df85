"""The per-cell fine-tune kernels that remain for gene pools too wide for the rounds over all cells: the work
queue and the spread path, on their three row scans, and the FP32-order form from host lists.  Whole numbers
equal to the oracle's."""

import functools

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

THRE = 0.15


@functools.lru_cache(maxsize=None)
def _problem(L=50, block=300):
    """Labels of six cells with genes (block) of their own each; queries that mix the genes of four labels."""
    rng = np.random.default_rng(11)
    n_genes = L * block

    def cells(labels, others):
        ptr, idx, val = [0], [], []
        for lab in labels:
            p = np.full(n_genes, 0.002)
            for m in [lab, *rng.choice(L, others, replace=False)]:
                p[m * block:(m + 1) * block] = 0.5 if others else 0.75
            c = np.flatnonzero(rng.random(n_genes) < p)
            idx.append(c)
            val.append(np.log2(1 + rng.integers(1, 40, len(c))))
            ptr.append(ptr[-1] + len(c))
        return synth.CSR(len(labels), n_genes, np.concatenate(val).astype(np.float32),
                         np.concatenate(idx).astype(np.int32), np.asarray(ptr, np.int32), np.asarray(labels, np.int32))

    ref = cells(np.repeat(np.arange(L), 6), 0)
    qry = cells(rng.integers(0, L, 40), 3)
    genes = synth.names("G", n_genes)
    return O.Problem(ref, qry, synth.names("CT", L), ref.labels, genes, genes)


@functools.lru_cache(maxsize=None)
def _solved(mode, **sizes):
    orc = O.Oracle(_problem(**sizes))
    orc.train()
    flags = orc.score(mode=mode, thre=THRE)[2].astype(np.uint8)
    final, rounds = orc.finetune(mode=mode, thre=THRE)
    assert rounds.max() >= 3
    return flags, final, rounds


def _trained(mode=abi.MODE_EXACT):
    prob = _problem()
    a = abi.Annotator(gpuid=0, mode=mode)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    assert 16 * (len(a.u32(1)) + 1) > 221 * 1024  # no table of e-values fits shared memory
    return a, prob


@pytest.mark.parametrize("scan", [0, 1, 2])
@pytest.mark.parametrize("heavy", [2, 1 << 30])
def test_spread_and_queue_paths(scan, heavy):
    """Two-register (0), packed (1) and packed scan with 32-bit run sums (2), every cell spread over the GPU or
    every cell on the work queue."""
    a, prob = _trained()
    a.set_tuning(3, scan)
    a.set_tuning(1, heavy)
    flags, final, rounds = _solved(1)
    a.reset_timings()
    got, got_rounds = a.finetune(prob.qry, flags, thre=THRE)
    t = a.timings()
    multi = int((flags.sum(1) >= 2).sum())
    assert t["ft_split_cells"] == (multi if heavy == 2 else 0)
    assert t["ft_queue_cells"] == (len(flags) - multi if heavy == 2 else len(flags))
    assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)


def test_fp32_order_from_host_lists():
    a, prob = _trained(abi.MODE_FP32REF)
    flags, final, rounds = _solved(0)
    got, got_rounds = a.finetune(prob.qry, flags, thre=THRE)
    assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)


@pytest.mark.parametrize("kind", ["tiny", "families", "small"])
@pytest.mark.parametrize("heavy", [2, 1 << 30])
@pytest.mark.parametrize("times", [0, 2])
def test_spread_and_queue_paths_on_narrow_pools(kind, heavy, times):
    """The same kernels where the two-register scan is asked for."""
    prob = H.problem(kind)
    res = H.oracle_run(kind, 1, times)
    a = abi.Annotator(gpuid=0)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    a.set_tuning(3, 0)
    a.set_tuning(1, heavy)
    a.reset_timings()
    got, got_rounds = a.finetune(prob.qry, res["flags"].astype(np.uint8), times=times)
    multi = int((res["flags"].sum(1) >= 2).sum())
    assert a.timings()["ft_split_cells"] == (multi if heavy == 2 else 0)
    assert np.array_equal(got, res["final"]) and np.array_equal(got_rounds, res["rounds"])
