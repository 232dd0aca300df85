"""The fine-tune by rounds over all cells at the sizes where its layout has edges: lookup tables of 8, 4,
2 and 1 copies (gene pools of about 1,100 to 8,000), labels around 32-row blocks, and cell counts around
quads.  Labels and round counts are whole numbers and equal the oracle's."""

import functools

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

POOLS = {  # reference rows, genes, labels, density, marker block
    "8 copies": (1200, 9000, 14, 0.05, (150, 220, 4.0, 6.0)),
    "4 copies": (1500, 12000, 30, 0.03, (200, 300, 5.0, 8.0)),
    "2 copies": (2000, 16000, 45, 0.02, (250, 330, 6.0, 10.0)),
    "1 copy": (2600, 24000, 72, 0.015, (250, 330, 6.0, 10.0)),
}


WIDE = 0.4  # a threshold that keeps many candidates on well separated labels


def _solve(prob, thre=0.05, mode=1):
    orc = O.Oracle(prob)
    orc.train()
    flags = orc.score(mode=mode, thre=thre)[2].astype(np.uint8)
    final, rounds = orc.finetune(mode=mode, thre=thre)
    return flags, final, rounds


def _annotator(prob, mode=abi.MODE_EXACT):
    a = abi.Annotator(gpuid=0, mode=mode)
    return a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)


@functools.lru_cache(maxsize=None)
def _pool(kind):
    n_ref, n_genes, L, density, block = POOLS[kind]
    w, ref, qry = synth.custom_dataset(n_ref, 40, n_genes, L, density, block=block, seed=5)
    genes = synth.names("G", n_genes)
    prob = O.Problem(ref, qry, synth.names("CT", L), ref.labels, genes, genes)
    return prob, _solve(prob, WIDE)


@pytest.mark.parametrize("kind", list(POOLS))
@pytest.mark.parametrize("scan", [1, 2])
def test_table_copies(kind, scan):
    """Each table width, with 64-bit (1) and 32-bit (2) run sums."""
    prob, (flags, final, rounds) = _pool(kind)
    a = _annotator(prob)
    copies = {"8 copies": 8, "4 copies": 4, "2 copies": 2, "1 copy": 1}[kind]
    bytes_of = [16 * c * (len(a.u32(1)) + 1) for c in (copies, 2 * copies)]
    assert bytes_of[0] <= 221 * 1024 and (copies == 8 or bytes_of[1] > 222 * 1024)
    a.set_tuning(3, scan)
    got, got_rounds = a.finetune(prob.qry, flags, thre=WIDE)
    assert rounds.max() >= 2
    assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)


@pytest.mark.parametrize("kind", ["8 copies", "4 copies", "2 copies"])
def test_fp32_order(kind):
    """The FP32-order scan: gene sets of several lengths of its 128 chunks, over pools of 1,100 to 5,200 genes."""
    prob = _pool(kind)[0]
    flags, final, rounds = _solve(prob, WIDE, mode=0)
    got, got_rounds = _annotator(prob, abi.MODE_FP32REF).finetune(prob.qry, flags, thre=WIDE)
    assert rounds.max() >= 2
    assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 33, 131])
def test_cell_counts_around_quads(n):
    """The first n cells of a query alone: each cell's result depends on its own row only."""
    prob = H.problem("families")
    res = H.oracle_run("families", 1)
    a = _annotator(prob)
    got, rounds = a.finetune(prob.qry.rows(0, n), res["flags"][:n].astype(np.uint8))
    assert np.array_equal(got, res["final"][:n]) and np.array_equal(rounds, res["rounds"][:n])


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
def test_label_sizes_around_blocks(mode):
    """Labels of 1, 2, 31, 32, 33, 64, 65 and 129 reference cells."""
    sizes = [1, 2, 31, 32, 33, 64, 65, 129]
    w, ref, qry = synth.custom_dataset(3000, 150, 3000, len(sizes), 0.08, seed=23)
    rows = np.concatenate([np.flatnonzero(ref.labels == lab)[:n] for lab, n in enumerate(sizes)])
    ref = ref.take(rows)
    assert [int(x) for x in np.bincount(ref.labels)] == sizes
    genes = synth.names("G", ref.n_cols)
    prob = O.Problem(ref, qry, synth.names("CT", len(sizes)), ref.labels, genes, genes)
    flags, final, rounds = _solve(prob, mode=0 if mode == abi.MODE_FP32REF else 1)
    got, got_rounds = _annotator(prob, mode).finetune(qry, flags)
    assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)


@pytest.mark.parametrize("kind", list(POOLS))
@pytest.mark.parametrize("scan", [1, 2])
@pytest.mark.parametrize("times", [2, 7])
def test_table_copies_in_quads(kind, scan, times):
    """Each table width with four cells to a pass: 80 cells (more than are scanned one by one), and 280, from which
    on a label that one cell of a quad needs goes to the label's work list."""
    prob, (flags, final, rounds) = _pool(kind)
    a = _annotator(prob)
    a.set_tuning(3, scan)
    got, got_rounds = a.finetune(prob.qry.take(np.tile(np.arange(40), times)), np.tile(flags, (times, 1)), thre=WIDE)
    assert (flags.sum(1) >= 2).sum() * times > 64
    assert np.array_equal(got, np.tile(final, times)) and np.array_equal(got_rounds, np.tile(rounds, times))


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
@pytest.mark.parametrize("n", [63, 64, 65, 66, 67, 68, 69, 255, 256, 257, 300, 2047, 4097])
def test_cell_counts_past_the_direct_form(n, mode):
    """Around the most cells that are scanned one by one (64), quads that are not full, 64 quads (work lists from there
    on), 512 quads (items sized by the round) and 4,096 cells (ordered by counting from there on); the cells in an
    order of their own."""
    prob = H.problem("families")
    res = H.oracle_run("families", 0 if mode == abi.MODE_FP32REF else 1)
    assert (res["flags"].sum(1) >= 2).all()
    at = np.random.default_rng(n).permutation(n) * 7 % prob.qry.n_rows
    got, rounds = _annotator(prob, mode).finetune(prob.qry.take(at), res["flags"][at].astype(np.uint8))
    assert np.array_equal(got, res["final"][at]) and np.array_equal(rounds, res["rounds"][at])


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
@pytest.mark.parametrize("n", [40, 120, 400])
def test_score_lists_with_nan(n, mode):
    """Empty reference rows make NaN-bearing lists in every round, constant and empty query rows lists of NaN alone:
    cells scanned one by one, in quads, and with work lists."""
    ref, qry, L = H.dataset("tiny")
    keep = np.ones(len(ref.indices), bool)
    for i in (0, 1, 50, 51, 52, 300):
        keep[ref.indptr[i]:ref.indptr[i + 1]] = False
    ptr = np.concatenate([[0], np.cumsum(keep)])[ref.indptr].astype(np.int32)
    r = synth.CSR(ref.n_rows, ref.n_cols, ref.data[keep], ref.indices[keep], ptr, ref.labels)
    q = qry.take(np.arange(40))
    q.data[q.indptr[5]:q.indptr[6]] = 1.0
    genes = synth.names("G", ref.n_cols)
    prob = O.Problem(r, q, synth.names("CT", L), ref.labels, genes, genes)
    flags, final, rounds = _solve(prob, WIDE, mode=0 if mode == abi.MODE_FP32REF else 1)
    assert (flags.sum(1) >= 2).sum() >= 30
    at = np.random.default_rng(n).permutation(n) * 3 % 40
    got, got_rounds = _annotator(prob, mode).finetune(q.take(at), flags[at], thre=WIDE)
    assert np.array_equal(got, final[at]) and np.array_equal(got_rounds, rounds[at])


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
@pytest.mark.parametrize("scan", [0, 2])
def test_rounds_that_drop_no_candidate(scan, mode):
    """A NaN score of the first candidate lets a round drop none, so a cell can take more rounds than it has labels."""
    ref, qry, L = H.dataset("families")
    keep = np.ones(len(ref.indices), bool)
    for i in np.flatnonzero(np.random.default_rng(2).random(ref.n_rows) < 0.03):
        keep[ref.indptr[i]:ref.indptr[i + 1]] = False
    ptr = np.concatenate([[0], np.cumsum(keep)])[ref.indptr].astype(np.int32)
    r = synth.CSR(ref.n_rows, ref.n_cols, ref.data[keep], ref.indices[keep], ptr, ref.labels)
    genes = synth.names("G", ref.n_cols)
    prob = O.Problem(r, qry.rows(0, 150), synth.names("CT", L), ref.labels, genes, genes)
    flags, final, rounds = _solve(prob, 1e9, mode=0 if mode == abi.MODE_FP32REF else 1)
    assert rounds.max() >= L + 2
    a = _annotator(prob, mode)
    a.set_tuning(3, scan)
    for heavy in (2, 1 << 30):
        a.set_tuning(1, heavy)
        got, got_rounds = a.finetune(prob.qry, flags, thre=1e9)
        assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)
