"""NaN in a fine-tune gene that is no score-step gene, FP32 order: the fine-tune ranks the cells and the candidate
labels' rows over the round's gene set, and a NaN there is an error ("a CSR value is NaN"); a NaN outside the
set is never ranked."""

import functools

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LABELS = (1, 4)  # the candidates of every cell


@functools.lru_cache(maxsize=None)
def _problem():
    """More genes tell two labels apart than the score step keeps of a pair with eight labels (148)."""
    w, ref, qry = synth.custom_dataset(900, 90, 8000, 8, 0.08, block=(500, 560, 4.0, 6.0), seed=17)
    genes = synth.names("G", 8000)
    return O.Problem(ref, qry, synth.names("CT", 8), ref.labels, genes, genes)


def _trained(ref=None):
    prob = _problem()
    a = abi.Annotator(gpuid=0, mode=abi.MODE_FP32REF)
    a.train(ref if ref is not None else prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    return a, prob


def _gene_sets(a, L):
    """(genes of the first round's set, fine-tune genes outside it), both without the score-step genes."""
    thre, genes, idx = a.u32(1), a.u32(4), a.u32(5).reshape(-1, 2)
    most = int(round(500 * (2 / 3) ** np.log2(2)))
    inside = set()
    for i, j in (LABELS, LABELS[::-1]):
        pos, n = idx[i * L + j]
        inside |= set(thre[genes[pos:pos + min(n, most)]].tolist())
    common = set(a.u32(0).tolist())
    return sorted(inside - common), sorted(set(thre.tolist()) - inside - common)


def _flags(n, L):
    flags = np.zeros((n, L), np.uint8)
    flags[:, LABELS] = 1
    return flags


def _with_value(m, row, gene, value):
    """The CSR with the row's entry of the gene set to value (added where there is none; None: without it)."""
    a, b = int(m.indptr[row]), int(m.indptr[row + 1])
    keep = np.flatnonzero(m.indices[a:b] != gene) + a
    idx, val = m.indices[keep], m.data[keep]
    if value is not None:
        idx, val = np.append(idx, gene), np.append(val, value)
    indptr = m.indptr.copy()
    indptr[row + 1:] += len(idx) - (b - a)
    return synth.CSR(m.n_rows, m.n_cols, np.concatenate([m.data[:a], val, m.data[b:]]).astype(np.float32),
                     np.concatenate([m.indices[:a], idx, m.indices[b:]]).astype(np.int32), indptr, m.labels)


@pytest.mark.parametrize("nan", [np.float32(np.nan), -np.float32(np.nan)])
@pytest.mark.parametrize("n", [1, 90])
def test_query_nan(n, nan):
    a, prob = _trained()
    L = len(prob.label_names)
    inside, outside = _gene_sets(a, L)
    assert inside and outside
    q = prob.qry.rows(0, n)
    for gene in (inside[0], inside[-1]):
        for row in (0, n - 1):
            with pytest.raises(abi.SgrError) as e:
                a.finetune(_with_value(q, row, gene, nan), _flags(n, L))
            assert e.value.status == 1 and "NaN" in str(e.value)
    got = a.finetune(_with_value(q, n - 1, outside[0], nan), _flags(n, L))
    want = a.finetune(_with_value(q, n - 1, outside[0], None), _flags(n, L))
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    # a cell with one candidate is not ranked
    flags = _flags(n, L)
    flags[n - 1, LABELS[0]] = 0
    a.finetune(_with_value(q, n - 1, inside[0], nan), flags)


@pytest.mark.parametrize("nan", [np.float32(np.nan), -np.float32(np.nan)])
def test_reference_nan(nan):
    clean, prob = _trained()
    L = len(prob.label_names)
    inside, outside = _gene_sets(clean, L)
    ref = prob.ref
    dense = np.zeros((ref.n_rows, ref.n_cols), np.float32)
    for r in range(ref.n_rows):
        dense[r, ref.indices[ref.indptr[r]:ref.indptr[r + 1]]] = ref.data[ref.indptr[r]:ref.indptr[r + 1]]

    def entry(genes, label):
        """An entry of the label at which a NaN leaves the label's median, and so the markers, as they are."""
        for gene in genes:
            rows = np.flatnonzero(ref.labels == label)
            col = np.sort(dense[rows, gene])
            half = len(col) // 2
            if not np.signbit(nan):
                rows_at = rows[dense[rows, gene] > col[min(half + 1, len(col) - 1)]]
            else:
                rows_at = rows[dense[rows, gene] < col[max(half - 2, 0)]]
            if len(rows_at):
                return int(rows_at[-1]), gene
        return None

    seen = 0
    for genes, label, bad in ((inside, LABELS[0], True), (inside, LABELS[1], True), (outside, LABELS[0], False),
                              (inside, 2, False)):
        at = entry(genes, label)
        if at is None:
            continue
        a, _ = _trained(_with_value(ref, at[0], at[1], nan))
        if any(not np.array_equal(a.u32(w), clean.u32(w)) for w in (0, 1, 4, 5)):
            continue
        seen += bad
        for n in (1, 90):
            q = prob.qry.rows(0, n)
            if bad:
                with pytest.raises(abi.SgrError) as e:
                    a.finetune(q, _flags(n, L))
                assert e.value.status == 1 and "NaN" in str(e.value)
            else:
                a.finetune(q, _flags(n, L))
    assert seen or np.signbit(nan)
