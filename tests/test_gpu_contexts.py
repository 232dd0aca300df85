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
