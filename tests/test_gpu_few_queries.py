"""Scores of a few queries (the CUDA-core correlation, up to 8 rows) and of one row more (the tensor cores)
equal the oracle's exact scores bit for bit, for either limb split; the selection by number of rows."""

import numpy as np
import pytest
import torch

from cusingler_b200 import abi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["tiny", "families", "small"])
@pytest.mark.parametrize("base128", [0, 1])
def test_few_queries(kind, base128):
    prob = H.problem(kind)
    res = H.oracle_run(kind, 1)
    a = abi.Annotator(gpuid=0)
    a.set_tuning(11, base128)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    for n in (1, 2, 3, 4, 5, 8, 9):
        for at in (0, 37):
            q = prob.qry.rows(at, at + n)
            assert H.ulp_diff(a.debug_scores(q), res["raw"][at:at + n]).max() == 0
            first, scores, flags = a.score_first(q)
            assert H.ulp_diff(scores, res["scores"][at:at + n]).max() == 0
            assert np.array_equal(first, res["first"][at:at + n])
            assert np.array_equal(flags, res["flags"][at:at + n].astype(np.uint8))


@pytest.mark.parametrize("rows", ["one", "sms", "sms + 1", "all"])
def test_selection_by_size(rows):
    """A row per SM is selected by row CTAs, more rows by warps per row and label: the same label scores, first
    labels and flags as the oracle's, chosen by size or set."""
    prob = H.problem("small")
    res = H.oracle_run("small", 1)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = min({"one": 1, "sms": sms, "sms + 1": sms + 1, "all": prob.qry.n_rows}[rows], prob.qry.n_rows)
    a = abi.Annotator(gpuid=0)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    for form in (None, 0, 16):
        if form is not None:
            a.set_tuning(7, form)
        first, scores, flags = a.score_first(prob.qry.rows(0, n))
        assert H.ulp_diff(scores, res["scores"][:n]).max() == 0
        assert np.array_equal(first, res["first"][:n])
        assert np.array_equal(flags, res["flags"][:n].astype(np.uint8))


def _launches_of_one_row(a, prob):
    a.reset_timings()
    a.score_first(prob.qry.rows(0, 1))
    return a.timings()["launches"]


def test_selection_by_size_can_be_set_again():
    """A set form holds for every size (one row: the items take one launch more); -1 chooses by size again, and
    tuning on a large sample leaves a one-row call its own form."""
    prob = H.problem("small")
    a = abi.Annotator(gpuid=0)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    by_size = _launches_of_one_row(a, prob)
    a.set_tuning(7, 0)
    assert _launches_of_one_row(a, prob) == by_size + 1
    a.set_tuning(7, -1)
    assert _launches_of_one_row(a, prob) == by_size
    for bad in (-2, 2, 32):
        with pytest.raises(abi.SgrError):
            a.set_tuning(7, bad)
    a.autotune(prob.qry)
    assert _launches_of_one_row(a, prob) == by_size
