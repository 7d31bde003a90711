"""Band-score checkpoints (ABEA_OPT_TRACE_BUDGET): reads whose trace exceeds the
budget keep checkpoints every 256 bands instead, and their traceback recomputes
the trace segment by segment.  Results must not change at all."""
import numpy as np
import pytest

from conftest import abea

pytestmark = pytest.mark.gpu

BYTES_PER_BAND = 128  # trace bytes per band (one byte per slot)


def align(batch, mode, budget, scores=False):
    ctx = abea.Context(0, mode, store_scores=scores)
    ctx.set_option(abea.OPT_TRACE_BUDGET, budget)
    dev = ctx.upload(batch)
    dev.run()
    pairs, counts = dev.results()
    return ctx, dev, pairs, counts


def same_alignments(batch, p1, c1, p2, c2):
    assert np.array_equal(c1, c2)
    for x, y in zip(abea.split_pairs(batch, p1, c1), abea.split_pairs(batch, p2, c2)):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("mode", [abea.MODE_PLAIN, abea.MODE_BATCHED])
def test_checkpointed_reads_match_the_oracle(oracle_mod, mode):
    """A budget that splits the batch: reads over ~5,400 bands checkpointed."""
    from abea_gb300 import synth
    batch = synth.make_batch("small", seed=3)
    budget = 5400 * BYTES_PER_BAND
    n_ck = int(np.sum(((batch.n_bands() + 3) // 4) * 4 * BYTES_PER_BAND > budget))
    assert 0 < n_ck < batch.n_reads
    _, dev, gp, gc = align(batch, mode, budget)
    op, oc, obest = oracle_mod.align_batch(batch)
    same_alignments(batch, gp, gc, op, oc)
    assert np.array_equal(dev.best_scores().view(np.uint32), obest.view(np.uint32))


@pytest.mark.parametrize("mode", [abea.MODE_PLAIN, abea.MODE_BATCHED])
def test_every_read_checkpointed_on_the_edge_cases(ref_synthetic, mode):
    """Budget of one byte: every read recomputes its trace, including tiny reads,
    paths that outgrow their output slot (tiny_20_5, few_events_400: the QC sum
    then needs a second recomputed walk) and reads over several segments."""
    batch, names, counts, pairs, _ = ref_synthetic
    _, dev, gp, gc = align(batch, mode, 1)
    assert np.array_equal(gc, counts)
    got = abea.split_pairs(batch, gp, gc)
    for i, name in enumerate(names):
        assert np.array_equal(got[i], pairs[i]), name
    # the trace is not kept, the band origins and scores are
    with pytest.raises(abea.AbeaError):
        dev.read_bands(len(names) - 1)


def test_checkpoints_leave_scores_origins_and_gradients_unchanged():
    from abea_gb300 import synth
    batch = synth.make_batch("small", seed=4)
    _, d0, p0, c0 = align(batch, abea.MODE_BATCHED, 0, scores=True)
    _, d1, p1, c1 = align(batch, abea.MODE_BATCHED, 1, scores=True)
    same_alignments(batch, p0, c0, p1, c1)
    assert np.array_equal(d0.best_scores().view(np.uint32), d1.best_scores().view(np.uint32))
    for i in (0, batch.n_reads // 2, batch.n_reads - 1):
        b0, _, o0 = d0.read_bands(i, scores=True)
        b1 = np.zeros_like(b0)
        o1 = np.zeros_like(o0)
        # scores and band origins only: a checkpointed read has no trace to give
        abea._check(abea.lib().abea_batch_read_bands(d1.ctx.h, d1.h, i, abea._p(b1), None, abea._p(o1)))
        assert np.array_equal(b0.view(np.uint32), b1.view(np.uint32))
        assert np.array_equal(o0, o1)
    g0, g1 = d0.backward(), d1.backward()
    assert np.array_equal(g0["grad_scalings"], g1["grad_scalings"])
    assert np.array_equal(g0["path_emission"], g1["path_emission"])


@pytest.mark.parametrize("mode", [abea.MODE_PLAIN, abea.MODE_BATCHED])
def test_f5c_batch_with_reads_over_8kb_checkpointed(oracle_mod, mode):
    """The 1.3 Mbase workload with the trace budget of an 8 kb read: the longest
    reads recompute, the rest keep their trace; the batched form's wide shape
    takes only reads that keep their trace."""
    from abea_gb300 import synth
    import os
    batch = synth.make_batch("f5c_batch", seed=1)
    budget = (8000 + int(8000 * 1.71) + 2) * BYTES_PER_BAND
    _, dev, gp, gc = align(batch, mode, budget)
    op, oc, _ = oracle_mod.align_batch(batch, threads=os.cpu_count())
    same_alignments(batch, gp, gc, op, oc)


@pytest.mark.parametrize("kept", [0, 2])
def test_checkpointed_reads_on_the_wide_shape(oracle_mod, kept):
    """Reads whose band counts lie around one checkpoint (256), a traceback slot's least
    read (512) and one round of sixteen recomputed segments (4,096), every read on the
    wide shape: all checkpointed, or only the longest ones."""
    from abea_gb300 import synth
    rng = np.random.default_rng(5)
    model = synth.make_model(rng)
    reads = []
    for target in (254, 256, 257, 511, 512, 513, 516, 4093, 4095, 4096, 4097, 4100, 8192, 8193):
        seq, ev = synth.make_read(rng, model, int(target / 2.4), 1.02, 2.0, 1.2, skip_p=0.01, mean_events=1.8)
        over = len(ev) + len(seq) - 5 + 2 - target  # a longer read, less its end
        assert over >= 0
        reads.append((seq.tobytes()[:len(seq) - over * 10 // 27], ev[:len(ev) - (over - over * 10 // 27)]))
    sc = np.zeros(len(reads), dtype=abea.types.SCALINGS_DTYPE)
    sc["scale"], sc["shift"], sc["var"], sc["log_var"] = 1.02, 2.0, 1.2, np.log(1.2)
    batch = abea.from_reads([r[0] for r in reads], [r[1] for r in reads], sc, model)
    assert 4096 in batch.n_bands() and 512 in batch.n_bands()
    budget = int(np.sort(batch.n_bands())[-kept - 1]) // 4 * 4 * BYTES_PER_BAND if kept else 1
    ctx = abea.Context(0, abea.MODE_BATCHED)
    ctx.set_option(abea.OPT_TRACE_BUDGET, budget)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1)
    dev = ctx.upload(batch)
    dev.run()
    pairs, counts = dev.results()
    op, oc, obest = oracle_mod.align_batch(batch)
    same_alignments(batch, pairs, counts, op, oc)
    assert np.array_equal(dev.best_scores().view(np.uint32), obest.view(np.uint32))


def test_more_checkpointed_reads_than_blocks(oracle_mod):
    from abea_gb300 import synth
    batch = synth.make_batch("small", seed=6, lengths=[230, 260, 90] * 150)
    _, dev, gp, gc = align(batch, abea.MODE_BATCHED, 1)
    op, oc, obest = oracle_mod.align_batch(batch)
    same_alignments(batch, gp, gc, op, oc)
    assert np.array_equal(dev.best_scores().view(np.uint32), obest.view(np.uint32))


@pytest.mark.parametrize("scores", [False, True])
@pytest.mark.parametrize("n", [2432, 2433, 3000])
def test_checkpointed_and_other_reads_in_more_than_a_wave(oracle_mod, n, scores):
    """Up to 16 warp-shape reads per SM of a GB300's 152, and more (their fills then share one
    copy of the code), every third read checkpointed, over one and over two segments."""
    from abea_gb300 import synth
    lengths = np.tile([40, 100, 230], 1000)[:n]
    batch = synth.make_batch("small", seed=7, lengths=lengths)
    budget = (int(np.sort(batch.n_bands())[-(n // 3)]) + 3) // 4 * 4 * BYTES_PER_BAND - 1
    ck = (batch.n_bands() + 3) // 4 * 4 * BYTES_PER_BAND > budget
    assert 0 < ck.sum() < n and (batch.n_bands()[ck] > 512).any()
    ctx = abea.Context(0, abea.MODE_BATCHED, store_scores=scores)
    ctx.set_option(abea.OPT_TRACE_BUDGET, budget)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1 << 40)
    dev = ctx.upload(batch)
    dev.run()
    pairs, counts = dev.results()
    op, oc, obest = oracle_mod.align_batch(batch, threads=8)
    same_alignments(batch, pairs, counts, op, oc)
    assert np.array_equal(dev.best_scores().view(np.uint32), obest.view(np.uint32))
