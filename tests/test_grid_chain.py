"""The wide shape's two engines, and the warp shape's two loops, against the oracle, with
every score, backpointer and band origin: reads that end around the points where the
exact chain hands over to the grid chain and back, emissions that no grid serves or that
lie far below its range, and events that are not finite.  All comparisons are exact: the
results are the reference's floats, whichever engine computes a band."""
import numpy as np
import pytest

from conftest import abea

pytestmark = pytest.mark.gpu


def make(rng, length, stdv=(1.0, 3.0), var=1.2, mean_events=1.8, skip=0.01):
    from abea_gb300 import synth
    model = synth.make_model(rng)
    model["level_stdv"] = rng.uniform(*stdv, len(model)).astype(np.float32)
    model["level_log_stdv"] = np.log(model["level_stdv"].astype(np.float64)).astype(np.float32)
    seq, ev = synth.make_read(rng, model, length, 1.02, 2.0, var, skip_p=skip, mean_events=mean_events)
    return model, seq.tobytes(), ev


def batch_of(model, reads):
    sc = np.zeros(len(reads), dtype=abea.types.SCALINGS_DTYPE)
    sc["scale"], sc["shift"], sc["var"], sc["log_var"] = 1.02, 2.0, 1.2, np.log(1.2)
    return abea.from_reads([r[0] for r in reads], [r[1] for r in reads], sc, model)


def check(oracle_mod, batch, shape):
    ctx = abea.Context(0, abea.MODE_BATCHED, store_scores=True)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1 if shape == "wide" else 1 << 40)
    dev = ctx.upload(batch)
    dev.run()
    pairs, counts = dev.results()
    opairs, ocounts, _ = oracle_mod.align_batch(batch, threads=8)
    assert np.array_equal(counts, ocounts)
    for got, exp in zip(abea.split_pairs(batch, pairs, counts), abea.split_pairs(batch, opairs, ocounts)):
        assert np.array_equal(got, exp)
    for i in range(batch.n_reads):
        b, t, bll = dev.read_bands(i, scores=True)
        _, _, info = oracle_mod.align(batch.sequence(i), batch.read_events(i), batch.model, batch.scalings[i],
                                      want_bands=True)
        assert np.array_equal(b.view(np.uint32), info["bands"].view(np.uint32)), i
        assert np.array_equal(t, info["trace"]), i
        assert np.array_equal(bll, info["bll"]), i


@pytest.mark.parametrize("shape", ["wide", "warp"])
@pytest.mark.parametrize("mean_events", [1.05, 1.8, 4.0])
def test_hand_over_between_the_engines(oracle_mod, mean_events, shape):
    """Reads of 6 bases up to ones with long grid runs, around the 800 bands after which
    the grid chain is first tried, at three event rates (few moves right, and many)."""
    rng = np.random.default_rng(11)
    model, _, _ = make(rng, 50)
    from abea_gb300 import synth
    reads = []
    for length in (6, 7, 60, 133, 160, 290, 296, 302, 330, 420, 550, 700, 1201, 2503, 4999):
        seq, ev = synth.make_read(rng, model, length, 1.02, 2.0, 1.2, skip_p=0.01, mean_events=mean_events)
        if len(ev):
            reads.append((seq.tobytes(), ev))
    check(oracle_mod, batch_of(model, reads), shape)


@pytest.mark.parametrize("shape", ["wide", "warp"])
@pytest.mark.parametrize("stdv", [(0.05, 0.4), (0.3, 1.0), (0.8, 1.1), (8.0, 30.0)])
def test_emissions_a_grid_does_not_serve(oracle_mod, stdv, shape):
    """Deviations so small that emissions are positive (no grid) or lie thousands below
    (their cells must lose or be done again), and so large that scores fall slowly."""
    rng = np.random.default_rng(12)
    model, seq, ev = make(rng, 1800, stdv=stdv)
    check(oracle_mod, batch_of(model, [(seq, ev)]), shape)


@pytest.mark.parametrize("shape", ["wide", "warp"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, 1e30, -1e5, 4000.0])
def test_outlier_events(oracle_mod, value, shape):
    """Single events far out or infinite, in and around the grid chain's bands."""
    rng = np.random.default_rng(13)
    model, seq, ev = make(rng, 2400)
    ev = ev.copy()
    for at in (700, 1500, 1501, 2600, len(ev) - 40):
        ev["mean"][at] = value
    check(oracle_mod, batch_of(model, [(seq, ev)]), shape)


@pytest.mark.parametrize("shape", ["wide", "warp"])
@pytest.mark.parametrize("mean_events", [1.05, 1.8, 4.0])
def test_bands_at_the_edges_of_a_read(oracle_mod, mean_events, shape):
    """Bands that lose the path: scalings off (the band follows the trim cells through the
    events, then the last event through the k-mers, and on the way is done again for events
    far out), and reads with 700 events or bases that do not belong to them at either end."""
    from abea_gb300 import synth
    rng = np.random.default_rng(14)
    model, _, _ = make(rng, 50)
    reads, scale = [], []
    for length, s in ((300, 1.1), (420, 0.9), (1203, 1.06), (2501, 1.1), (2502, 0.7), (2503, 1.5), (1900, 1.02)):
        seq, ev = synth.make_read(rng, model, length, 1.02, 2.0, 1.2, skip_p=0.01, mean_events=mean_events)
        reads.append((seq.tobytes(), ev))
        scale.append(s)
    seq, ev = reads[3][0], reads[3][1].copy()
    for at, value in ((900, np.inf), (1201, 1e30), (1300, -1e5), (1777, 4000.0), (len(ev) - 1, 4000.0), (len(ev) - 2, -np.inf)):
        ev["mean"][at] = value
    reads.append((seq, ev))
    scale.append(1.1)
    seq, ev = reads[6]
    junk, junk_ev = synth.make_read(rng, model, 500, 1.02, 2.0, 1.2, skip_p=0.01, mean_events=1.8)
    reads += [(seq, np.concatenate([ev, junk_ev[:700]])), (seq, np.concatenate([junk_ev[:700], ev])),
              (seq + junk.tobytes(), ev), (junk.tobytes() + seq, ev)]
    scale += [1.02] * 4
    batch = batch_of(model, reads)
    batch.scalings["scale"] = scale
    check(oracle_mod, batch, shape)


def test_many_entries_into_the_grid_chain(oracle_mod):
    """More reads than SMs, each with an event far out every few hundred, so that every
    block enters and leaves the grid chain time and again with all SMs at work: the whole
    block has to take each of these decisions alike."""
    from abea_gb300 import synth
    rng = np.random.default_rng(15)
    model, _, _ = make(rng, 50)
    reads = []
    for i in range(200):
        seq, ev = synth.make_read(rng, model, 2000 + 7 * i, 1.02, 2.0, 1.2, skip_p=0.01, mean_events=1.8)
        ev = ev.copy()
        ev["mean"][700 + i::150 + i] = 4000.0
        reads.append((seq.tobytes(), ev))
    batch = batch_of(model, reads)
    ctx = abea.Context(0, abea.MODE_BATCHED)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1)
    dev = ctx.upload(batch)
    opairs, ocounts, obest = oracle_mod.align_batch(batch, threads=8)
    for _ in range(3):
        dev.run()
        pairs, counts = dev.results()
        assert np.array_equal(counts, ocounts)
        for got, exp in zip(abea.split_pairs(batch, pairs, counts), abea.split_pairs(batch, opairs, ocounts)):
            assert np.array_equal(got, exp)
        assert np.array_equal(dev.best_scores().view(np.uint32), obest.view(np.uint32))


def counters(batch, shape):
    ctx = abea.Context(0, abea.MODE_BATCHED)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1 if shape == "wide" else 1 << 40)
    dev = ctx.upload(batch)
    dev.run()
    dev.results()
    return dev._counters()


def test_grid_candidates_selftest():
    """Candidates on every grid over the whole range of scores, aimed at the ends of their cells
    or not: none wrong, and the random ones hardly ever declined.  A k-mer is refused for an
    emission that may be positive: at most the 5% of deviations below 0.5, and with them
    margins and divisions of under 1 in 1,000 (as the division's own self-test asks)."""
    import ctypes as C
    out = np.zeros(7, dtype=np.int64)
    f = abea.lib().abea_internal_selftest_grid
    f.argtypes, f.restype = [C.c_int64, C.c_uint64, C.c_void_p], C.c_int
    assert f(1 << 26, 7, out.ctypes.data) == 0
    wrong, cases, on_grid, proven, skips, skips_on_grid, aimed = out.tolist()
    assert wrong == 0
    assert on_grid > 0.94 * cases and proven > 0.999 * on_grid
    assert skips_on_grid > 0.999 * skips
    assert aimed > 1 << 20


@pytest.mark.parametrize("shape", ["wide", "warp"])
def test_an_ordinary_read_runs_on_the_grid(shape):
    """All but the first and last bands: scores pass -2^11 after some 950 bands (the wide shape
    tries after 800, then every 128), and a read's last 170 k-mers are the exact engine's."""
    rng = np.random.default_rng(18)
    model, seq, ev = make(rng, 6000)
    batch = batch_of(model, [(seq, ev)])
    c = counters(batch, shape)
    bands = int(batch.n_bands()[0])
    assert c["grid"] > 0.9 * (bands - 1200 - 170 * bands / 6000) / 4
    assert c["grid_again"] < 0.1 * c["grid"]


@pytest.mark.parametrize("shape", ["wide", "warp"])
@pytest.mark.parametrize("every", [4000, 1500, 400, 60])
def test_a_grid_between_kmers_that_none_serves(oracle_mod, every, shape):
    """k-mers whose emissions may be positive (a deviation of 0.2), one in `every` bases: the
    bands between them still run on a grid where 128-slot windows fit between them (not at one
    in 60), and every score is the oracle's."""
    rng = np.random.default_rng(19)
    model, seq, ev = make(rng, 6000)
    model = model.copy()
    codes = np.searchsorted(np.frombuffer(b"ACGT", np.uint8), np.frombuffer(seq, np.uint8)).astype(np.int64)
    ranks = sum(codes[i:len(codes) - 5 + i] << (2 * (5 - i)) for i in range(6))
    hits = np.bincount(ranks, minlength=4096)
    for at in range(every // 2, len(ranks), every):
        once = at + int(np.argmin(hits[ranks[at:at + 40]]))  # a k-mer that is rare in the read
        model["level_stdv"][ranks[once]] = 0.2
        model["level_log_stdv"][ranks[once]] = np.log(0.2)
    batch = batch_of(model, [(seq, ev)])
    check(oracle_mod, batch, shape)
    c = counters(batch, shape)
    if shape == "wide":
        assert c["grid"] > 100 if every >= 400 else c["grid"] < 100


@pytest.mark.parametrize("shape", ["wide", "warp"])
def test_cells_without_a_proof_are_done_again_in_fp64(shape):
    """An infinite event's emissions are proven by nothing: its cells (one in each of the 100
    bands or more that hold it) are computed in FP64."""
    rng = np.random.default_rng(13)
    model, seq, ev = make(rng, 2400)
    plain = counters(batch_of(model, [(seq, ev)]), shape)
    ev = ev.copy()
    ev["mean"][[700, 1500, 2600, 3300]] = np.inf
    c = counters(batch_of(model, [(seq, ev)]), shape)
    assert c["fp64"] >= plain["fp64"] + 4 * 90
    assert c["fp64"] <= c["slow"]


@pytest.mark.parametrize("budget", [0, 400_000])
def test_a_wait_out_of_polls_ends_in_a_timeout(oracle_mod, budget):
    """With a limit of one poll the grid chain's waits give up: the run reports a timeout
    and returns no alignment, and the next run with the usual limit is the oracle's (the
    same batch, whose captured graph holds the limit)."""
    rng = np.random.default_rng(16)
    model, seq, ev = make(rng, 2400)
    batch = batch_of(model, [(seq, ev)])
    ctx = abea.Context(0, abea.MODE_BATCHED)
    ctx.set_option(abea.OPT_LONG_READ_BANDS, 1)
    ctx.set_option(abea.OPT_TRACE_BUDGET, budget)
    limit = ctx.get_option(abea.OPT_SPIN_LIMIT)
    dev = ctx.upload(batch)
    op, oc, _ = oracle_mod.align_batch(batch)
    for _ in range(2):
        ctx.set_option(abea.OPT_SPIN_LIMIT, 1)
        with pytest.raises(abea.AbeaError) as e:
            dev.run()
            dev.results()
        assert e.value.status == -5
        ctx.set_option(abea.OPT_SPIN_LIMIT, limit)
        dev.run()
        pairs, counts = dev.results()
        assert np.array_equal(counts, oc)
        assert np.array_equal(abea.split_pairs(batch, pairs, counts)[0], abea.split_pairs(batch, op, oc)[0])
