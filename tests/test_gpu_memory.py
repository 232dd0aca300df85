"""A GPU that another framework has nearly filled: calls take less workspace instead of failing, and give the
same results.  Device memory is filled by ordinary allocations and given back after each test."""

import contextlib

import numpy as np
import pytest

from cusingler_b200 import abi, synth
from tests import helpers as H

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _free_mib(mib):
    """Only this much device memory free inside."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        for step in (1 << 30, 1 << 26, 1 << 21):
            while torch.cuda.mem_get_info(0)[0] - (mib << 20) >= step:
                spare = (torch.cuda.mem_get_info(0)[0] - (mib << 20)) // step * step
                held.append(torch.empty(spare, dtype=torch.uint8, device="cuda"))
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _trained(prob, mode=abi.MODE_EXACT):
    a = abi.Annotator(gpuid=0, mode=mode)
    return a.train(prob.ref, prob.celltypes, prob.label_names, prob.ref_genes, prob.qry_genes)


def _tiled_query(m, times):
    """The rows, `times` times over, on the device."""
    import torch

    nnz = int(m.indptr[-1])
    indptr = np.concatenate([[0]] + [m.indptr[1:].astype(np.int64) + nnz * t for t in range(times)])
    keep = [torch.from_numpy(x).cuda() for x in (m.data, m.indices.astype(np.int32))]
    keep = [t.repeat(times) for t in keep] + [torch.from_numpy(indptr.astype(np.int32)).cuda()]
    return abi.device_csr(m.n_rows * times, m.n_cols, *(t.data_ptr() for t in keep)), keep


@pytest.mark.parametrize("mode", [abi.MODE_EXACT, abi.MODE_FP32REF])
def test_finetune_in_several_batches(mode):
    """100,000 cells' round buffers take several times the free memory: the call runs them in batches."""
    prob = H.problem("families")
    res = H.oracle_run("families", 0 if mode == abi.MODE_FP32REF else 1)
    times = 500
    a = _trained(prob, mode)
    flags = res["flags"].astype(np.uint8)
    a.finetune(prob.qry, flags)
    q, keep = _tiled_query(prob.qry, times)
    many = np.tile(flags, (times, 1))
    batched = []
    with _free_mib(250):
        for _ in range(2):
            a.reset_timings()
            final, rounds = a.finetune(q, many)
            batched.append(a.timings()["ft_split_rounds"])
            assert np.array_equal(final, np.tile(res["final"], times))
            assert np.array_equal(rounds, np.tile(res["rounds"], times))
    a.reset_timings()
    final, rounds = a.finetune(q, many)  # and again in one
    assert min(batched) >= 2 * a.timings()["ft_split_rounds"] > 0
    assert np.array_equal(final, np.tile(res["final"], times))
    assert np.array_equal(rounds, np.tile(res["rounds"], times))
    a.close()
    del q, keep


def test_small_context():
    """A small training and call where less than one slab of buffers is free."""
    prob = H.problem("tiny")
    res = H.oracle_run("tiny", 1)
    _trained(prob).annotate(prob.qry)  # the kernels are loaded
    with _free_mib(60):
        a = _trained(prob)
        first, final = a.annotate(prob.qry)
        assert np.array_equal(first, res["first"]) and np.array_equal(final, res["final"])
        a.close()


def test_training_without_room_for_the_optional_tables():
    """The pairs' masks per candidate count (147 MiB here) do not fit: the rounds use the lists."""
    from tests import test_gpu_wide_pool as T

    sizes = dict(L=60, block=100)
    prob, (flags, final, rounds) = T._problem(**sizes), T._solved(1, **sizes)
    _trained(prob).finetune(prob.qry, flags, thre=T.THRE)
    with _free_mib(100):
        a = _trained(prob)
        got, got_rounds = a.finetune(prob.qry, flags, thre=T.THRE)
        assert np.array_equal(got, final) and np.array_equal(got_rounds, rounds)
        a.close()


def test_training_without_room_for_a_second_copy():
    """The reference as given and regrouped (120 MB each) do not fit together."""
    rng = np.random.default_rng(3)
    R, W, k, L = 10000, 4000, 1500, 4
    keys = rng.random((R, W), np.float32)
    labels = rng.integers(0, L, R).astype(np.int32)
    for lab in range(L):  # genes that a label's cells store more often
        keys[labels == lab, 100 * lab:100 * (lab + 1)] *= 0.5
    indices = np.sort(keys.argpartition(k, axis=1)[:, :k], axis=1).astype(np.int32)
    data = rng.integers(1, 60, (R, k)).astype(np.float32)
    ref = synth.CSR(R, W, data.reshape(-1), indices.reshape(-1), (np.arange(R + 1) * k).astype(np.int32), labels)
    names, genes = synth.names("CT", L), synth.names("G", W)
    q = ref.rows(0, 50)
    a = abi.Annotator(gpuid=0).train(ref, labels, names, genes, genes)
    tables, labels_of = [a.u32(what) for what in range(8)], a.annotate(q)
    a.close()
    bad = indices.reshape(-1).copy()
    bad[-1] = W
    with _free_mib(245):
        a = abi.Annotator(gpuid=0)
        for _ in range(2):  # the second training finds the first one's buffers
            a.train(ref, labels, names, genes, genes)
            assert all(np.array_equal(a.u32(what), tables[what]) for what in range(8))
        with pytest.raises(abi.SgrError) as e:
            a.train(synth.CSR(R, W, ref.data, bad, ref.indptr, labels), labels, names, genes, genes)
        assert e.value.status == 1
    assert all(np.array_equal(x, y) for x, y in zip(a.annotate(q), labels_of))
    a.close()


def test_held_round_buffers_are_given_back():
    """The score step needs more than what the fine-tune of an earlier call left free."""
    prob = H.problem("families")
    res = H.oracle_run("families", 1)
    times = 500
    a = _trained(prob)
    a.set_tuning(2, 16)
    a.annotate(prob.qry)
    q, keep = _tiled_query(prob.qry, times)
    flags = np.tile(res["flags"].astype(np.uint8), (times, 1))
    with _free_mib(500):
        for _ in range(2):
            final, rounds = a.finetune(q, flags)
            assert np.array_equal(final, np.tile(res["final"], times))
            first, final = a.annotate(q)
            assert np.array_equal(first, np.tile(res["first"], times))
            assert np.array_equal(final, np.tile(res["final"], times))
    a.close()
    del q, keep
