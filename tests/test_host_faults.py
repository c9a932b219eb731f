"""Failure paths of the host code, with the library's objects linked to a CUDA
runtime that needs no GPU (tests/fake): a launch that fails, memory that runs out."""
import numpy as np
import pytest

from dbsr_gb300 import SPLIT_BF16, Assembler, _lib, synth
from dbsr_gb300._lib import DbsrgError

from fake import library


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return library(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def fake(lib, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", lib)
    lib.fake_limit(2**63)
    lib.fake_fail(None)
    lib.fake_clear_log()
    return lib


def context(w):
    a = Assembler(w.t, w.ks, w.ksp, w.ksq, tuning=None)
    a.set_orbitals(w.pq, w.ipbs)
    a.alloc_matrix(w.nch, w.icc, w.iicc, w.mk)
    a.set_precision(SPLIT_BF16)
    return a


def all_bound(w):
    io = np.zeros((w.nbf, w.nch), dtype=np.int32, order="F")
    io[: w.nbound, :] = 1
    return io


CALLS = {
    "k_moment_sums R": lambda a, w: a.get_table(0, 2, 1),
    "k_moment_sums S": lambda a, w: a.get_table(1, 1, 1),
    "k_fill_r": lambda a, w: a.get_table(0, 2, 1),
    "k_fill_s": lambda a, w: a.get_table(1, 1, 1),
    "k_triang": lambda a, w: a.get_table(1, 0, 1),
    "k_vch": lambda a, w: a.orth_channels(all_bound(w)),
    "k_bound_rows": lambda a, w: a.backward([1], [1], [1], [2], [2], [1.0]),
}


@pytest.mark.parametrize("case", CALLS)
def test_a_failed_launch_leaves_nothing_that_reads_as_built(fake, case):
    """A build whose launch fails: the call reports it, what it was to fill is not
    taken for filled by the next call, and its memory comes back."""
    kernel, call = case.split()[0], CALLS[case]
    w = synth.small(ns=40, nch=2, mk=1, n_entries=20, breit=False, seed=3)
    a = context(w)
    call(a, w)  # the scratch of such a call
    a.release_tables()
    used = fake.fake_used()
    fake.fake_fail(kernel.encode())
    with pytest.raises(DbsrgError, match="ECUDA"):
        call(a, w)
    fake.fake_fail(None)
    fake.fake_clear_log()
    call(a, w)
    assert kernel in fake.fake_log().decode()
    a.release_tables()
    assert fake.fake_used() == used
    a.close()
    assert fake.fake_used() == 0


def test_builds_after_a_queued_replay_wait_for_it(fake):
    """Asynchronous mode: a replay rewrites the tables and orbital products of its
    graph on the contraction stream, so what a later list builds from them on a
    table stream is queued behind it."""
    w = synth.structures_case()
    a = context(w)
    a.alloc_perturbers(w.npert, w.icb, w.ibb)
    a.set_targets(w.ntarg, w.iptar, w.iitar, 1)
    lists = {L.kpol: (L.icase, L.itype, L.kpol, L.k1, L.k2, L.k3, L.k4, L.c)
             for L in w.lists if (L.icase, L.itype) == (2, 1)}
    a.set_async(True)
    a.graph_capture([lists[0]])
    a.graph_launch(w.pq)
    fake.fake_clear_log()
    a.graph_launch(w.pq)
    a.gen_matrix(*lists[2])
    log = [x.split() for x in fake.fake_log().decode().splitlines()]
    main = next(x[1] for x in log if x[0] == "graph")
    log = log[[x[0] for x in log].index("graph") + 1:]
    build = next(i for i, x in enumerate(log) if x[0] == "launch" and "k_pair" in x[2])
    assert log[build][1] != main
    after = {x[2] for x in log[:build] if x[:2] == ["record", main]}
    assert any(x[0] == "wait" and x[1] == log[build][1] and x[2] in after for x in log[:build])
    a.close()


def blocks(nch, pairs):
    """icc of the diagonal blocks (none) and of the given channel pairs."""
    icc = np.zeros((nch, nch), dtype=np.int32, order="F")
    for b, (i, j) in enumerate(pairs):
        icc[i, j] = icc[j, i] = b + 1
    return icc, len(pairs)


def basis_context(ns, nch, pairs):
    w = synth.small(ns=40, nch=2, mk=1, n_entries=20, breit=False, seed=3)
    t = np.concatenate([np.zeros(8), np.linspace(0.0, 10.0, ns - 7), np.full(8, 10.0)])
    a = Assembler(t, w.ks, w.ksp, w.ksq, tuning=None)
    icc, iicc = blocks(nch, pairs)
    a.alloc_matrix(nch, icc, iicc, 0)
    a.set_precision(SPLIT_BF16)
    sol = np.zeros((2 * ns, 2 * ns, nch), order="F")
    return a, sol, np.full(nch, 2 * ns, dtype=np.int32)


def test_channel_basis_takes_fewer_blocks_at_once_when_memory_is_short(fake):
    """The workspace follows the free memory: with room for a few blocks beside the
    channels' digits the call works through them a few at a time, and releasing the
    tables gives back what it kept."""
    pairs = [(i, j) for i in range(8) for j in range(i)]
    a, sol, nsol = basis_context(40, 8, pairs)
    a.channel_basis(sol, nsol)
    whole = fake.fake_log().decode().count("k_sgemm")
    a.release_tables()
    used = fake.fake_used()
    a.channel_basis(sol, nsol)
    kept = fake.fake_used() - used
    a.release_tables()
    assert fake.fake_used() == used
    fake.fake_limit(used + sol.nbytes + kept // 3)
    fake.fake_clear_log()
    a.channel_basis(sol, nsol)
    assert fake.fake_log().decode().count("k_sgemm") > whole
    # a matrix that needs the memory of the workspace kept takes it
    fake.fake_limit(fake.fake_used() + 1000)
    icc, iicc = blocks(8, pairs + [(0, 0)])
    a.alloc_matrix(8, icc, iicc, 0)
    a.close()


def test_a_large_channel_basis_workspace_is_given_back(fake):
    """A workspace beyond a gigabyte lives for the call only."""
    a, sol, nsol = basis_context(420, 70, [(i, 0) for i in range(1, 33)])
    used = fake.fake_used()
    a.channel_basis(sol, nsol)
    assert fake.fake_used() == used
    a.close()
