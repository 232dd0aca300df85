"""The allocation-free label selection (sgr_select_labels_noalloc) against sgr_score_first.

It serves callers that cannot allocate device memory (their framework owns the GPU's memory, or
they are recording a CUDA graph): it works on device buffers the caller passes and keeps its only
temporary space in a fixed array inside the library.  This file is collected last so that a run
stopping at the first failure has already run every other test; it also passes on its own in a
fresh process.
"""

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _case(kind, constant_rows=False):
    prob = H.problem(kind)
    ref, qry = prob.ref, prob.qry
    if constant_rows:
        # empty reference rows make NaN-bearing score lists (the path that uses the fixed scratch)
        ptr = ref.indptr.copy()
        cut = {0, 1, 40}
        rows = [(ref.indices[ptr[i]:ptr[i + 1]], ref.data[ptr[i]:ptr[i + 1]]) if i not in cut else
                (np.zeros(0, np.int32), np.zeros(0, np.float32)) for i in range(ref.n_rows)]
        ind = np.concatenate([r[0] for r in rows]).astype(np.int32)
        dat = np.concatenate([r[1] for r in rows]).astype(np.float32)
        ip = np.zeros(ref.n_rows + 1, np.int32)
        ip[1:] = np.cumsum([len(r[0]) for r in rows])
        ref = synth.CSR(ref.n_rows, ref.n_cols, dat, ind, ip, ref.labels)
        prob = O.Problem(ref, qry, prob.label_names, prob.celltypes, prob.ref_genes, prob.qry_genes)
    a = abi.Annotator(gpuid=0, mode=abi.MODE_EXACT)
    a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)
    return a, prob


@pytest.mark.parametrize("kind,constant_rows", [("tiny", False), ("tiny", True), ("small", False)])
def test_noalloc_matches_score_first(kind, constant_rows):
    import torch

    a, prob = _case(kind, constant_rows)
    first, scores, flags = a.score_first(prob.qry)
    raw = a.debug_scores(prob.qry)                # Q x R correlations, the same the score step uses
    ranges = a.u32(6)                             # (start, len) of each label's reference columns
    Q, R = raw.shape
    L = len(prob.label_names)
    dev = torch.device("cuda", 0)
    d_scores = torch.from_numpy(raw).to(dev)
    for call in range(2):                         # two calls in a row share the fixed scratch
        d_ls = torch.full((Q, L), -7.0, dtype=torch.float32, device=dev)
        d_first = torch.full((Q,), -1, dtype=torch.int32, device=dev)
        d_flags = torch.full((Q, L), 9, dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()
        free_before = torch.cuda.mem_get_info(0)[0]
        st = abi.select_labels_noalloc(d_scores.data_ptr(), R, Q, ranges, 0.8, 0.05, d_ls.data_ptr(),
                                       d_first.data_ptr(), d_flags.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream)
        assert st == 0
        torch.cuda.synchronize()
        if call == 1:  # (the first call may load the library's module that holds the fixed array)
            assert torch.cuda.mem_get_info(0)[0] == free_before  # the call allocated no device memory
        ls = d_ls.cpu().numpy()
        assert H.ulp_diff(ls, scores).max() == 0, call
        assert np.array_equal(d_first.cpu().numpy(), first), call
        assert np.array_equal(d_flags.cpu().numpy(), flags), call
        if not constant_rows:  # and the oracle's exact-mode labels directly
            res = H.oracle_run(kind, 1)
            assert H.ulp_diff(ls, res["scores"]).max() == 0 and np.array_equal(d_first.cpu().numpy(), res["first"])


def test_noalloc_rejects_oversized_and_bad_ranges():
    # validated on the host before any device work
    big = np.array([0, 200000], np.uint32)
    assert abi.select_labels_noalloc(1, 200000, 1, big, 0.8, 0.05, 1, 1, None) == 6   # UNSUPPORTED
    bad = np.array([0, 10, 10, 10], np.uint32)
    assert abi.select_labels_noalloc(1, 15, 1, bad, 0.8, 0.05, 1, 1, None) == 1       # out of range
    empty = np.array([0, 0], np.uint32)
    assert abi.select_labels_noalloc(1, 15, 1, empty, 0.8, 0.05, 1, 1, None) == 5     # EMPTY_LABEL


@pytest.mark.parametrize("n_rows,L,pad", [(2400, 5, 0), (2401, 7, 3), (4999, 1, 1)])
def test_noalloc_many_rows_with_nan_lists(n_rows, L, pad):
    """Enough rows for the warp-per-row launch: rows without NaN, rows that are all NaN, rows with a NaN-bearing
    list (left to the CTA-per-row launch), one-score labels and a row stride off 16 bytes, against the
    oracle's percentile (std::sort order with NaN, as the reference's)."""
    import torch

    rng = np.random.default_rng(n_rows)
    lens = rng.integers(1, 90, L)
    if L > 1:
        lens[0] = 1
    starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    ld = int(lens.sum()) + pad
    raw = np.full((n_rows, ld), -5.0, np.float32)
    raw[:, :lens.sum()] = rng.normal(0.4, 0.1, (n_rows, lens.sum())).astype(np.float32)
    raw[::7, starts[-1]:starts[-1] + max(1, lens[-1] // 2)] = raw[::7, [starts[-1]]]  # ties
    raw[11::311, :] = np.nan
    for q in range(5, n_rows, 97):
        raw[q, starts[-1] + int(rng.integers(lens[-1]))] = np.nan
    ranges = np.stack([starts, lens], 1).astype(np.uint32).reshape(-1)
    dev = torch.device("cuda", 0)
    d = torch.from_numpy(raw).to(dev)
    ls = torch.empty((n_rows, L), device=dev)
    first = torch.empty(n_rows, dtype=torch.int32, device=dev)
    flags = torch.empty((n_rows, L), dtype=torch.uint8, device=dev)
    assert abi.select_labels_noalloc(d.data_ptr(), ld, n_rows, ranges, 0.8, 0.05, ls.data_ptr(), first.data_ptr(),
                                     flags.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ls, first, flags = ls.cpu().numpy(), first.cpu().numpy(), flags.cpu().numpy()
    for q in sorted(set(range(0, n_rows, 41)) | set(range(5, n_rows, 97)) | set(range(11, n_rows, 311))):
        want = np.array([O.percentile(raw[q, s:s + n], 0.8) for s, n in zip(starts, lens)], np.float32)
        assert H.ulp_diff(ls[q], want).max() == 0, q
        top = O.minmax(want)[1]
        assert first[q] == top
        with np.errstate(invalid="ignore"):
            assert np.array_equal(flags[q], (want >= np.float32(want[top] - np.float32(0.05))).astype(np.uint8)), q


@pytest.mark.parametrize("n_rows,L,longest", [(296, 9, 800), (297, 9, 800), (40, 3, 30000), (300, 256, 40)])
def test_noalloc_rows_around_the_turn_of_the_ctas(n_rows, L, longest):
    """As many rows as CTAs fit, and more of them (a warp per label and row): lists with and without NaN, ties and
    a row that is all NaN, against the oracle's percentile."""
    import torch

    rng = np.random.default_rng(n_rows + L)
    lens = rng.integers(1, longest, L)
    lens[L // 2] = longest
    starts = np.concatenate([[0], np.cumsum(lens)[:-1]])
    ld = int(lens.sum())
    raw = rng.normal(0.4, 0.1, (n_rows, ld)).astype(np.float32)
    raw[3] = np.nan
    raw[5, starts[L // 2] + longest // 2] = np.nan
    raw[7, starts[L // 2]:starts[L // 2] + longest // 2] = raw[7, starts[L // 2]]
    ranges = np.stack([starts, lens], 1).astype(np.uint32).reshape(-1)
    dev = torch.device("cuda", 0)
    d = torch.from_numpy(raw).to(dev)
    ls = torch.empty((n_rows, L), device=dev)
    first = torch.empty(n_rows, dtype=torch.int32, device=dev)
    flags = torch.empty((n_rows, L), dtype=torch.uint8, device=dev)
    assert abi.select_labels_noalloc(d.data_ptr(), ld, n_rows, ranges, 0.8, 0.05, ls.data_ptr(), first.data_ptr(),
                                     flags.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    ls, first, flags = ls.cpu().numpy(), first.cpu().numpy(), flags.cpu().numpy()
    for q in (0, 3, 5, 7, n_rows // 2, n_rows - 1):
        want = np.array([O.percentile(raw[q, s:s + n], 0.8) for s, n in zip(starts, lens)], np.float32)
        assert H.ulp_diff(ls[q], want).max() == 0, q
        top = O.minmax(want)[1]
        assert first[q] == top
        with np.errstate(invalid="ignore"):
            assert np.array_equal(flags[q], (want >= np.float32(want[top] - np.float32(0.05))).astype(np.uint8)), q
