"""The batched form's wide-shape heuristic (host code, no device): how many of the
longest reads take the 512-thread shape for batch shapes measured on a GB300."""
import ctypes as C
import os

import numpy as np

from conftest import abea


def wide_threshold(bands, blocks=152):
    if not os.path.exists(abea.LIB_PATH):
        abea.build()
    L = abea.lib()
    f = L.abea_internal_wide_threshold
    f.argtypes = [C.c_void_p, C.c_int32, C.c_int32]
    f.restype = C.c_int64
    b = np.ascontiguousarray(bands, dtype=np.int64)
    return f(b.ctypes.data, len(b), blocks)


def n_wide(bands, blocks=152):
    thr = wide_threshold(bands, blocks)
    return 0 if thr >= 2**62 else int(np.sum(np.asarray(bands) >= thr))


def test_latency_bound_batch_goes_all_wide():
    """The f5c batch shape: its longest read bounds the batch whatever the split,
    and with every read on the wide shape (the blocks pulling them longest first)
    nothing else is longer (measured 8.46 ms, against 8.49-9.10 ms for the best
    one-wide-read-per-block split and 36.1 ms with none)."""
    from abea_gb300 import synth
    nb = synth.make_batch("f5c_batch", seed=1).n_bands()
    assert n_wide(nb) == len(nb)


def test_few_reads_per_sm_go_all_wide_many_stay_on_the_warp_shape():
    """1,024 reads of 1-10 kb (about 7 per SM): every read wide, 18.5 ms against
    20.8 ms with none.  4,096 such reads (27 per SM): none, 35.5 ms against 68.5
    with every read wide, because 16 warp-shape reads per SM issue more per SM
    than one wide read."""
    rng = np.random.default_rng(11)
    lens = rng.integers(1000, 10001, 1024)
    nb = lens - 5 + (lens * 1.71).astype(np.int64) + 2
    assert n_wide(nb) == 1024
    lens = rng.integers(1000, 10001, 4096)
    nb = lens - 5 + (lens * 1.71).astype(np.int64) + 2
    assert n_wide(nb) == 0
    assert n_wide(np.full(4096, 27000)) == 0


def test_serving_batches_keep_the_split():
    """A serving-stream device batch (about 4,000 reads, lognormal median 8 kb):
    26 reads per SM, not bound by its longest read, so not every read goes wide
    (measured: 1.23 s for the 200 Mbase stream every read wide, 0.99 s split)."""
    rng = np.random.default_rng(5)
    lens = np.clip(rng.lognormal(np.log(8000), 0.6, 3987), 500, 200000).astype(np.int64)
    nb = lens - 5 + (lens * 1.71).astype(np.int64) + 2
    k = n_wide(nb)
    assert 0 <= k < 152, k


def test_fewer_reads_than_blocks_and_edge_inputs():
    assert n_wide([54382]) == 1                        # one read alone: the wide shape
    assert wide_threshold([]) >= 2**62                 # nothing to do
    assert wide_threshold([10, -1]) == -1              # bad input
    assert wide_threshold([10], blocks=0) == -1


def test_short_reads_that_leave_sms_free_are_wide():
    """A read's first bands are where the warp shape's cells most often need FP64: one read of
    20 to 300 bases, or up to four per SM, is two to five times as fast on the wide shape
    (one of 100 bases 0.11 ms against 0.51; 304 of 300 bases 0.45 against 1.12)."""
    for bands in (40, 145, 263, 407, 842):
        assert n_wide([bands]) == 1, bands
    for n in (4, 64, 152):
        assert n_wide([276] * n) == n
    assert n_wide([58] * 152) == 152
    assert n_wide([878] * 304) == 304
    assert n_wide([304] * 608) == 608
    # with 16 reads and more per SM the warps' number wins again (0.88 ms; 3.2 against 7.9)
    assert n_wide([110] * 4000) == 0
    assert n_wide([1759] * 2432) == 0


def test_checkpointed_reads_keep_the_split():
    """A latency-bound batch with checkpointed reads (trace over the budget): those
    run on the warp shape and would start last behind every wide read, so the
    heuristic keeps at most one wide read per block and never a checkpointed one."""
    if not os.path.exists(abea.LIB_PATH):
        abea.build()
    f = abea.lib().abea_internal_wide_threshold_ck
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_int32]
    f.restype = C.c_int64
    from abea_gb300 import synth
    nb = np.ascontiguousarray(synth.make_batch("f5c_batch", seed=1).n_bands(), dtype=np.int64)
    ck = np.zeros(len(nb), dtype=np.int32)
    assert f(nb.ctypes.data, ck.ctypes.data, len(nb), 152) == 1          # no checkpointed read: every read wide
    ck[np.argsort(-nb)[200:210]] = 1                                     # ten mid-length reads checkpointed
    thr = f(nb.ctypes.data, ck.ctypes.data, len(nb), 152)
    k = int(np.sum((nb >= thr) & (ck == 0)))
    assert thr > 1 and 0 < k < 152, (thr, k)


def threshold_any(nb, ck, blocks=152):
    if not os.path.exists(abea.LIB_PATH):
        abea.build()
    f = abea.lib().abea_internal_wide_threshold_any
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_int32]
    f.restype = C.c_int64
    nb = np.ascontiguousarray(nb, dtype=np.int64)
    ck = np.ascontiguousarray(ck, dtype=np.int32)
    return f(nb.ctypes.data, ck.ctypes.data, len(nb), blocks)


def test_checkpointed_reads_may_be_wide():
    """The rule without the cluster pair: a long checkpointed read, and every read of a
    latency-bound batch with or without them, go wide (one read of 9 kb checkpointed 5.3 ms
    wide, 31 on a warp); many short checkpointed reads per SM stay on the warp shape (2,400 of
    1 kb: 13.0 ms against 18.7)."""
    from abea_gb300 import synth
    assert threshold_any([24928], [1]) == 1
    nb = synth.make_batch("f5c_batch", seed=1).n_bands()
    none = np.zeros(len(nb), dtype=np.int32)
    assert threshold_any(nb, none) == 1 == threshold_any(nb, none + 1)
    some = none.copy()
    some[np.argsort(-nb)[:10]] = 1  # the ten longest
    assert threshold_any(nb, some) == 1
    # one long checkpointed read among many short ones: it alone where the short ones would
    # then be the longer part, every read where it bounds the batch
    ck = np.array([1] + [0] * 2432, dtype=np.int32)
    assert 1759 < threshold_any([24928] + [1759] * 2432, ck) <= 24928
    assert threshold_any([54000] + [1759] * 2432, ck) == 1
    assert threshold_any([3413] * 2400, [1] * 2400) >= 2**62


def test_checkpointed_part_of_a_large_batch_is_wide():
    """4,096 reads of 1-10 kb, those over 8 kb checkpointed (six per SM): all of these wide, none
    of the others; without checkpoints none."""
    rng = np.random.default_rng(1)
    lens = rng.integers(1000, 10001, 4096)
    nb = lens - 5 + (lens * 1.71).astype(np.int64) + 2
    ck = (lens > 8000).astype(np.int32)
    thr = threshold_any(nb, ck)
    assert nb[ck == 0].max() < thr <= nb[ck == 1].min()
    assert threshold_any(nb, 0 * ck) >= 2**62
