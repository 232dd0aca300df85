"""Contexts keep their device memory in slabs of their own: calls of growing and shrinking sizes on one
context, retraining, failed calls in between, and contexts in several threads give the oracle's labels."""

import threading

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _trained(kind, mode=abi.MODE_EXACT):
    prob = H.problem(kind)
    a = abi.Annotator(gpuid=0, mode=mode)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    return a, prob


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
def test_sizes_up_and_down_with_retraining_and_errors(mode):
    a, prob = _trained("families", mode)
    bad = synth.CSR(1, prob.qry.n_cols, np.ones(1, np.float32), np.array([prob.qry.n_cols + 1], np.int32),
                    np.array([0, 1], np.int32), np.zeros(1, np.int32))
    for kind in ("families", "tiny", "small", "families"):
        p = H.problem(kind)
        want = H.oracle_run(kind, 0 if mode == abi.MODE_FP32REF else 1)
        a.train(p.ref, p.celltypes, p.label_names, p.ref_genes, p.qry_genes)
        for n in (1, 90, p.qry.n_rows, 7, p.qry.n_rows):
            first, final = a.annotate(p.qry.rows(0, n))
            assert np.array_equal(first, want["first"][:n]) and np.array_equal(final, want["final"][:n])
        with pytest.raises(abi.SgrError):
            a.score_first(bad if kind == "families" else synth.CSR(1, p.qry.n_cols + 1, bad.data, bad.indices,
                                                                    bad.indptr, bad.labels))


def test_contexts_in_threads():
    wrong = []

    def work(kind):
        try:
            a, prob = _trained(kind)
            want = H.oracle_run(kind, 1)
            for n in (40, prob.qry.n_rows, 3, prob.qry.n_rows):
                first, final = a.annotate(prob.qry.rows(0, n))
                if not (np.array_equal(first, want["first"][:n]) and np.array_equal(final, want["final"][:n])):
                    wrong.append((kind, n))
            a.close()
        except Exception as e:  # noqa: BLE001
            wrong.append((kind, e))

    for kind in ("tiny", "families", "small"):
        H.oracle_run(kind, 1)
    threads = [threading.Thread(target=work, args=(k,)) for k in ("tiny", "families", "small", "tiny")]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("heavy", [2, 1 << 30])
def test_per_cell_kernels_in_threads(heavy):
    """The per-cell fine-tune kernels take shared memory by the gene pool's size: contexts of several sizes in
    several threads do not lower the limit under one another's launches."""
    wrong = []
    start = threading.Barrier(4)

    def work(kind):
        try:
            a, prob = _trained(kind)
            a.set_tuning(3, 0)
            a.set_tuning(1, heavy)
            res = H.oracle_run(kind, 1)
            q, flags = prob.qry.rows(0, 8), res["flags"][:8].astype(np.uint8)
            start.wait()
            for _ in range(150):
                final, rounds = a.finetune(q, flags)
                if not (np.array_equal(final, res["final"][:8]) and np.array_equal(rounds, res["rounds"][:8])):
                    wrong.append(kind)
            a.close()
        except Exception as e:  # noqa: BLE001
            wrong.append((kind, e))
            start.abort()

    kinds = ("tiny", "small", "families", "small")
    for kind in kinds:
        H.oracle_run(kind, 1)
    threads = [threading.Thread(target=work, args=(k,)) for k in kinds]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
