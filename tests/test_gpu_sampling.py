"""The sampling kernel against the plain restatement of the reference's sampler."""
import numpy as np
import pytest
import torch

from plain import sampler as ps

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run_sampler(logits_row, n_draws, temperature, top_k, top_p, penalty, history=(), seed=0):
    """Draws ``n_draws`` tokens from one row of logits, each from a slot with a stream of its own."""
    from xeno_rt_b200.csrc import ops
    from xeno_rt_b200.sampling import sequence_key
    vocab = len(logits_row)
    logits = torch.tensor(np.asarray(logits_row, dtype=np.float32), device=DEV).repeat(n_draws, 1).contiguous()
    slots = torch.arange(n_draws, dtype=torch.int32, device=DEV)
    keys = np.array([sequence_key(seed * 100003 + i) for i in range(n_draws)], dtype=np.uint64).view(np.int64)
    rng_key = torch.from_numpy(keys).to(DEV)
    counter = torch.zeros(n_draws, dtype=torch.int32, device=DEV)
    words = (vocab + 31) // 32
    seen = torch.zeros(n_draws, words, dtype=torch.int32, device=DEV)
    if len(history):
        ids = torch.tensor(list(history) * n_draws, dtype=torch.int32, device=DEV)
        sl = slots.repeat_interleave(len(history)).contiguous()
        ops.mark_seen(seen, sl, ids, vocab)
    full = lambda v, dt: torch.full((n_draws,), v, dtype=dt, device=DEV)
    out = torch.empty(n_draws, dtype=torch.int32, device=DEV)
    ops.sample(out, logits, slots, full(temperature, torch.float32), full(top_k, torch.int32),
               full(top_p, torch.float32), full(penalty, torch.float32), seen, rng_key, counter)
    assert counter.eq(1).all()
    return out.cpu().numpy()


def test_greedy_is_argmax_first_maximum():
    logits = np.random.default_rng(0).normal(size=5000).astype(np.float32)
    logits[[77, 4000]] = 9.0
    assert run_sampler(logits, 3, 0.0, 40, 0.95, 1.0).tolist() == [77] * 3
    assert run_sampler(logits, 2, 1e-5, 0, 1.0, 1.0).tolist() == [77] * 2


def test_repetition_penalty_flips_greedy():
    logits = np.zeros(300, dtype=np.float32)
    logits[10], logits[20], logits[30] = 4.0, 3.0, -1.0
    assert run_sampler(logits, 1, 0.0, 0, 1.0, 2.0, history=[10, 10, 30])[0] == 20  # 4/2 < 3
    assert run_sampler(logits, 1, 0.0, 0, 1.0, 1.0, history=[10])[0] == 10  # penalty 1 = none
    assert run_sampler(logits, 1, 0.0, 0, 1.0, 2.0)[0] == 10  # empty history


@pytest.mark.parametrize("temperature,top_k,top_p,penalty,history", [
    (0.8, 40, 0.95, 1.1, (3, 5, 700)),      # the reference's defaults
    (1.0, 0, 1.0, 1.0, ()),                 # plain temperature sampling over everything
    (1.5, 5, 1.0, 1.0, ()),                 # top-k alone
    (0.7, 0, 0.6, 1.0, ()),                 # top-p alone
    (1.0, 3, 0.5, 1.3, (0, 1, 2)),
])
def test_support_and_frequencies_match_the_plain_sampler(temperature, top_k, top_p, penalty, history):
    rng = np.random.default_rng(42)
    vocab = 1000
    logits = (rng.normal(size=vocab) * 2.0).astype(np.float32)
    ids, probs = ps.candidate_distribution(logits, history, temperature, top_k, top_p, penalty)
    n = 20000
    got = run_sampler(logits, n, temperature, top_k, top_p, penalty, history)
    assert set(got.tolist()) <= set(ids.tolist()), "a token outside the kept set was drawn"
    expect = dict(zip(ids.tolist(), probs.tolist()))
    counts = np.bincount(got, minlength=vocab)
    for tok, p in expect.items():
        if p > 0.02:
            assert abs(counts[tok] / n - p) < 4 * np.sqrt(p * (1 - p) / n) + 1e-3, (tok, p, counts[tok] / n)
    big = [t for t, p in expect.items() if p > 0.02]
    assert all(counts[t] > 0 for t in big)


def test_top_k_keeps_the_earlier_of_equal_values():
    logits = np.full(200, -5.0, dtype=np.float32)
    logits[[50, 60, 70, 80]] = 2.0  # four equal maxima, top_k = 2 keeps ids 50 and 60
    got = run_sampler(logits, 4000, 1.0, 2, 1.0, 1.0)
    assert set(got.tolist()) == {50, 60}
    assert abs((got == 50).mean() - 0.5) < 0.05
    got = run_sampler(logits, 2000, 1.0, 0, 0.5, 1.0)  # mass 0.5 of 4 equal tokens (plus dust): 50, 60 (and 70 at most)
    assert 50 in got and 60 in got and 80 not in got


def test_a_seed_gives_the_same_tokens_and_another_seed_others():
    logits = np.random.default_rng(1).normal(size=4000).astype(np.float32)
    a = run_sampler(logits, 64, 1.0, 0, 1.0, 1.0, seed=7)
    b = run_sampler(logits, 64, 1.0, 0, 1.0, 1.0, seed=7)
    c = run_sampler(logits, 64, 1.0, 0, 1.0, 1.0, seed=8)
    assert np.array_equal(a, b) and not np.array_equal(a, c)


def test_big_vocabulary_and_padding_rows():
    from xeno_rt_b200.csrc import ops
    vocab = 151936
    logits = torch.randn(3, vocab, device=DEV)
    logits[0, 150000] = 50.0
    slots = torch.tensor([0, -1, 1], dtype=torch.int32, device=DEV)
    out = torch.empty(3, dtype=torch.int32, device=DEV)
    f = lambda v, dt: torch.full((3,), v, dtype=dt, device=DEV)
    ops.sample(out, logits, slots, f(0.8, torch.float32), f(40, torch.int32), f(0.95, torch.float32),
               f(1.0, torch.float32), None, torch.zeros(2, dtype=torch.int64, device=DEV),
               torch.zeros(2, dtype=torch.int32, device=DEV))
    got = out.tolist()
    assert got[0] == 150000 and got[1] == -1 and 0 <= got[2] < vocab
    top40 = set(torch.topk(logits[2], 40).indices.tolist())
    assert got[2] in top40


def test_small_top_k_over_a_big_vocabulary_gathered_or_not():
    """A small top_k gathers its candidates into shared memory first (everything in the bin of the
    k-th largest logit or above, at most 4,096); when more than that share the bin the kernel walks
    the vocabulary instead.  Both ways keep the same set: equal values at the cut in index order."""
    vocab = 70001
    rng = np.random.default_rng(5)
    # (1) gathered: ties at the cut.  300 equal logits share the 40th place; ids in rising order win
    logits = (rng.normal(size=vocab) * 0.5).astype(np.float32)
    high = rng.choice(vocab, size=30, replace=False)
    logits[high] = 6.0 + rng.random(30).astype(np.float32)
    tied = np.setdiff1d(rng.choice(vocab, size=320, replace=False), high)[:300]
    logits[tied] = 4.25
    got = run_sampler(logits, 3000, 1.0, 40, 1.0, 1.0)
    kept = set(high.tolist()) | set(np.sort(tied)[:10].tolist())
    assert set(got.tolist()) <= kept
    ids, probs = ps.candidate_distribution(logits, (), 1.0, 40, 1.0, 1.0)
    assert set(ids.tolist()) == kept
    # (2) not gathered: every logit equal, 70,001 elements in one bin; top_k 40 keeps ids 0 .. 39
    flat = np.full(vocab, 1.5, dtype=np.float32)
    got = run_sampler(flat, 2000, 1.0, 40, 1.0, 1.0)
    assert set(got.tolist()) <= set(range(40)) and len(set(got.tolist())) > 30
    # (3) the reference's defaults on the gathered path against the plain sampler's kept set
    logits = (rng.normal(size=vocab) * 3.0).astype(np.float32)
    ids, probs = ps.candidate_distribution(logits, (7, 8), 0.8, 40, 0.95, 1.1)
    got = run_sampler(logits, 4000, 0.8, 40, 0.95, 1.1, history=(7, 8))
    assert set(got.tolist()) <= set(ids.tolist())
    top = int(ids[np.argmax(probs)])
    assert abs((got == top).mean() - probs.max()) < 4 * np.sqrt(probs.max() * (1 - probs.max()) / 4000) + 1e-3


# one block a row, two, eight; a slice that just fits the blocks' shared memory and one that does not; rows of whole 16 bytes or not
@pytest.mark.parametrize("vocab", [1, 33, 4096, 4097, 16390, 128256, 327680, 327685])
@pytest.mark.parametrize("temperature,top_k,top_p", [(0.8, 40, 0.95), (1.0, 300, 0.9), (1.0, 0, 0.9), (0.7, 0, 1.0)])
def test_a_draw_lands_where_the_mass_says(vocab, temperature, top_k, top_p):
    """The id of a draw u is the one whose share of the kept mass, walked in index order, covers u.  The kernel's masses are
    rounded down to 2^-32 of the largest, and 32-bit exponentials are off by 2e-7 of their value: the walk may be off by
    vocab * 2^-32 + 1e-6; an id at the edge of the kept set, which either rounding may put in or out, holds less than 1e-5."""
    from xeno_rt_b200.sampling import sequence_key
    rng = np.random.default_rng(vocab + top_k)
    logits = (rng.normal(size=vocab) * 2.0).astype(np.float32)
    if vocab > 1000:
        logits[rng.random(vocab) < 0.3] = -np.inf
    n, mask = 24, (1 << 64) - 1
    got = run_sampler(logits, n, temperature, top_k, top_p, 1.0, seed=3)
    ids, probs = ps.candidate_distribution(logits.astype(np.float64), (), temperature, top_k, top_p, 1.0)
    order = np.argsort(ids)
    upper = dict(zip(ids[order].tolist(), np.cumsum(probs[order]).tolist()))
    share = dict(zip(ids.tolist(), probs.tolist()))

    def splitmix(x):
        x = (x + 0x9E3779B97F4A7C15) & mask
        x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & mask
        return x ^ (x >> 31)

    slack = vocab * 2.0 ** -32 + 1.2e-5
    for i, token in enumerate(got.tolist()):
        u = (splitmix((sequence_key(3 * 100003 + i) + 0x9E3779B97F4A7C15) & mask) >> 32) / 2.0 ** 32
        assert token in upper
        assert upper[token] - share[token] - slack <= u <= upper[token] + slack


def test_rows_without_a_finite_maximum_and_with_nan():
    """Only ids above minus infinity are drawn, also beside a NaN (a small top_k, greedy); a row without any value gives its first id."""
    for vocab in (300, 20001):
        logits = np.full(vocab, -np.inf, dtype=np.float32)
        assert set(run_sampler(logits, 8, 1.0, 40, 0.9, 1.0).tolist()) == {0}
        logits[[7, vocab - 2]] = 1.0
        assert set(run_sampler(logits, 64, 1.0, 40, 1.0, 1.0).tolist()) == {7, vocab - 2}
        assert set(run_sampler(logits, 64, 1.0, 0, 0.99, 1.0).tolist()) == {7, vocab - 2}
        logits[5] = np.nan
        assert set(run_sampler(logits, 64, 1.0, 2, 1.0, 1.0).tolist()) == {7, vocab - 2}
        assert set(run_sampler(logits, 8, 0.0, 0, 1.0, 1.0).tolist()) == {7}


@pytest.mark.parametrize("vocab", [300, 20001, 128256])
def test_infinities_take_the_row_and_a_nan_is_never_drawn(vocab):
    """The first infinity is the id, whatever else the row holds; beside finite values a NaN has no mass, with and without top_k
    and top_p, on one block and on a team."""
    rng = np.random.default_rng(vocab)
    options = [(1.0, 0, 1.0), (1.0, 0, 0.9), (0.7, 40, 0.95), (0.7, 280, 1.0), (0.0, 0, 1.0)]
    logits = rng.normal(size=vocab).astype(np.float32)
    logits[[3, vocab // 2, vocab - 1]] = np.nan
    for temperature, top_k, top_p in options:
        got = run_sampler(logits, 64, temperature, top_k, top_p, 1.0)
        assert np.isfinite(logits[got]).all()
        for infinite in ([vocab // 3], [vocab - 2, vocab // 3], [7, 8, vocab - 2]):
            row = logits.copy()
            row[infinite] = np.inf
            assert set(run_sampler(row, 8, temperature, top_k, top_p, 1.0).tolist()) == {min(infinite)}


# candidates that one block's room just holds and does not; values spread over the blocks of a team, and falling, so that one block has
# all of them
@pytest.mark.parametrize("falling", [False, True])
@pytest.mark.parametrize("vocab", [4096, 20001, 128256, 400000])
@pytest.mark.parametrize("top_k", [257, 500, 1900, 3500])
def test_a_large_top_k_over_one_block_and_a_team(vocab, top_k, falling):
    """Only ids of the k largest are drawn, and each half of their mass (by index) about as often as it says: 720 draws, most of
    them from batches whose rows get the largest teams, six standard deviations."""
    rng = np.random.default_rng(vocab + top_k)
    logits = (rng.normal(size=vocab) * 0.5).astype(np.float32)
    if falling:
        logits = np.sort(logits)[::-1].copy()
    ids, probs = ps.candidate_distribution(logits.astype(np.float64), (), 1.0, top_k, 1.0, 1.0)
    got = np.concatenate([run_sampler(logits, n, 1.0, top_k, 1.0, 1.0, seed=i) for i, n in enumerate([300] + [70] * 6)])
    assert set(got.tolist()) <= set(ids.tolist())
    order = np.argsort(ids)
    half = ids[order][np.searchsorted(np.cumsum(probs[order]), 0.5)]
    share = probs[ids <= half].sum()
    assert abs((got <= half).mean() - share) < 6 * np.sqrt(share * (1 - share) / len(got))


# a slice of the smallest size, of an odd one, rows of whole 16 bytes or not; teams of eight, four and two blocks; a top_k of one, the
# usual ones, the largest that each team serves and one more
@pytest.mark.parametrize("rows", [1, 37, 64, 149])
@pytest.mark.parametrize("vocab", [4096, 16385, 32000, 128256, 151937])
def test_the_small_form_gives_the_same_ids(rows, vocab):
    """Every id is the one that the kernel gives without being told the largest top_k: kept sets, masses and draws are whole numbers
    there.  Rows: plain logits, few different values (ties at the cut, also more than there is room for), both zeros, infinities
    and NaN, fewer finite values than top_k, falling values, greedy rows and padding among them, with a history."""
    from xeno_rt_b200.csrc import ops
    rng = np.random.default_rng(rows * 7 + vocab)
    logits = (rng.normal(size=(rows, vocab)) * 3.0).astype(np.float32)
    for i in range(rows):
        kind = (i + vocab) % 9 if rows > 1 else 0
        if kind == 1:
            logits[i] = np.round(logits[i])
        elif kind == 2:
            logits[i] = np.where(rng.random(vocab) < 0.5, -0.0, 0.0)
        elif kind == 3:
            logits[i, rng.choice(vocab, 3)] = np.inf
        elif kind == 4:
            logits[i, rng.random(vocab) < 0.5] = np.nan
        elif kind == 5:
            logits[i] = -np.inf
            logits[i, rng.choice(vocab, 11)] = 1.0
        elif kind == 6:
            logits[i] = np.sort(logits[i])[::-1]
        elif kind == 7:
            logits[i] = -np.inf
    logits = torch.from_numpy(logits).to(DEV)
    seen = torch.from_numpy(rng.integers(0, 2 ** 31, size=(rows, (vocab + 31) // 32), dtype=np.int32)).to(DEV)
    slots = torch.arange(rows, dtype=torch.int32, device=DEV)
    if rows > 1:
        slots[rows // 2] = -1
    as_rows = lambda v: torch.from_numpy(np.resize(np.asarray(v), rows)).to(DEV)
    key = torch.from_numpy(rng.integers(0, 2 ** 62, size=rows)).to(DEV)
    for top_k in (1, 40, 64, 65, 128, 129, 256, 257):
        ks = as_rows(np.array([top_k, max(1, top_k // 2), top_k, 1, top_k], dtype=np.int32))
        temps = as_rows(np.array([0.8, 1.0, 0.7, 1.3, 0.9, 0.8, 0.0] if rows > 1 else [0.8], dtype=np.float32))
        for top_p, penalty in ((0.95, 1.1), (1.0, 1.0), (0.5, 1.3)):
            args = (temps, ks, as_rows(np.array([top_p], dtype=np.float32)), as_rows(np.array([penalty], dtype=np.float32)), seen, key)
            got = []
            for told in (0, top_k):
                out = torch.full((rows,), -7, dtype=torch.int32, device=DEV)
                counter = torch.arange(rows, dtype=torch.int32, device=DEV)
                ops.sample(out, logits, slots, *args, counter, largest_top_k=told)
                got.append((out.tolist(), counter.tolist()))
            assert got[0] == got[1]


# teams of four and of two blocks, rows of whole 16 bytes or not
@pytest.mark.parametrize("rows,vocab", [(40, 32000), (76, 20001), (152, 9000)])
def test_rows_whose_first_cut_leaves_too_few_or_too_many(rows, vocab):
    """The small form gives the ids of the other one: rows masked down to fewer ids than top_k, to a run of neighbours that few groups
    of lanes hold, to as many as are ranked at once and one more, with the lowest number; more than that above the cut (values in order);
    equal values at the cut, as many as are listed, one more, and all of them; zeros of both signs there."""
    from xeno_rt_b200.csrc import ops
    rng = np.random.default_rng(vocab)
    logits = (rng.normal(size=(rows, vocab)) * 3.0).astype(np.float32)

    def masked(row, kept, lowest=-np.inf):
        values = row[kept].copy()
        row[:] = lowest
        row[kept] = values

    for i in range(rows):
        row, kind = logits[i], i % 18
        if kind in (0, 1, 2, 3):
            masked(row, rng.choice(vocab, (1, 11, 512, 513)[kind], replace=False))
        elif kind in (4, 5, 6):
            masked(row, slice(vocab // 3, vocab // 3 + (39, 400, 2500)[kind - 4]))
        elif kind == 7:
            row.sort()
        elif kind == 8:
            row[:] = np.sort(row)[::-1]
        elif kind in (9, 10, 11):  # equal values at the cut
            row[rng.choice(vocab, (600, 4096, 4097)[kind - 9], replace=False)] = 20.0
            row[rng.choice(vocab, 5, replace=False)] = 21.0
        elif kind == 12:
            row[:] = 1.0
        elif kind in (13, 14, 15):  # all zeros without a sign, few, half
            row[:] = np.where(rng.random(vocab) < (1.0, 0.001, 0.5)[kind - 13], 0.0, -0.0)
            row[rng.choice(vocab, 7, replace=False)] = 1.0
        elif kind == 16:
            masked(row, rng.choice(vocab, 11, replace=False), np.finfo(np.float32).min)
    logits = torch.from_numpy(logits).to(DEV)
    full = lambda v, dtype: torch.full((rows,), v, dtype=dtype, device=DEV)
    slots = torch.arange(rows, dtype=torch.int32, device=DEV)
    seen = torch.from_numpy(rng.integers(0, 2 ** 31, size=(rows, (vocab + 31) // 32), dtype=np.int32)).to(DEV)
    key = torch.from_numpy(rng.integers(0, 2 ** 62, size=rows)).to(DEV)
    for top_k in (1, 40, 64):
        for top_p, penalty in ((0.95, 1.0), (1.0, 1.2), (0.3, 1.0)):
            got = []
            for told in (0, top_k):
                out, counter = full(-7, torch.int32), torch.arange(rows, dtype=torch.int32, device=DEV)
                for draw in range(4):
                    ops.sample(out, logits, slots, full(0.9, torch.float32), full(top_k, torch.int32), full(top_p, torch.float32),
                               full(penalty, torch.float32), seen, key, counter, largest_top_k=told)
                    got.append(out.tolist())
            assert got[:4] == got[4:]


def _sampler_of(slots, vocab):
    from xeno_rt_b200.cache import Cache
    from xeno_rt_b200.core import DType
    from xeno_rt_b200.sampling import Sampler
    cache = Cache([], slots * 64, 1024, DType.BF16, DEV, slots)
    sampler, opened = Sampler(cache, vocab), [cache.open_slot() for _ in range(slots)]
    sampler.begin(opened, list(range(slots)))
    return sampler, opened, torch.tensor(opened, dtype=torch.int32, device=DEV)


def test_options_that_one_stream_brought_serve_another():
    """The options of a batch are kept from call to call: a call on a second stream, while the first is still busy, finds them."""
    from xeno_rt_b200.sampling import SamplerConfig
    logits = torch.zeros(2, 5000, device=DEV)
    greedy, hot = [SamplerConfig(0.0)] * 2, [SamplerConfig(1.0, 0, 1.0, 1.0)] * 2
    sampler, _, rows = _sampler_of(2, 5000)
    want = sampler.sample(logits, rows, hot).tolist()
    assert want != [0, 0]  # (what greedy rows give)
    sampler, _, rows = _sampler_of(2, 5000)
    nobody = torch.full_like(rows, -1)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(first):
        sampler.sample(logits, nobody, greedy)  # what the room of the next options may still hold
        sampler.sample(logits, nobody, [SamplerConfig(0.5), SamplerConfig(0.7)])
        torch.cuda._sleep(500_000_000)
        sampler.sample(logits, nobody, hot)
    with torch.cuda.stream(second):
        got = sampler.sample(logits, rows, hot)
    torch.cuda.synchronize()
    assert got.tolist() == want


@pytest.mark.parametrize("call", ["sample", "begin"])
def test_new_options_and_seeds_are_refused_inside_a_capture(call):
    """They come from the host: a graph would replay whatever the host's buffer holds then.  Known options may be captured."""
    from xeno_rt_b200.sampling import SamplerConfig
    logits = torch.zeros(2, 5000, device=DEV)
    sampler, slots, rows = _sampler_of(2, 5000)
    known = [SamplerConfig(0.9)] * 2
    sampler.sample(logits, rows, known)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            if call == "begin":
                sampler.begin(slots, [5, 6])
            else:
                sampler.sample(logits, rows, [SamplerConfig(0.6)] * 2)
    for turn in range(6):  # and all goes on
        sampler.begin(slots, [turn, turn])
        sampler.sample(logits, rows, [SamplerConfig(0.3 + turn)] * 2)
    sampler.sample(logits, rows, known)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        out = sampler.sample(logits, rows, known)
    sampler.begin(slots, [1, 2])
    sampler.rng_counter.zero_()
    graph.replay()
    got = out.tolist()
    sampler.rng_counter.zero_()
    assert got == sampler.sample(logits, rows, known).tolist()


def test_sequences_begun_by_several_threads_keep_their_seeds(monkeypatch):
    """``begin`` of other slots at the same time, the device busy: no thread's seeds pass through a buffer that another one writes."""
    import threading
    import time
    from xeno_rt_b200.core import staging
    from xeno_rt_b200.sampling.sampler import sequence_key
    take = staging.PinnedRing.take

    def slow_take(self, n):  # every thread has its buffer before the first one fills it
        got = take(self, n)
        time.sleep(0.05)
        return got

    sampler, slots, _ = _sampler_of(12, 100)
    torch.cuda.synchronize()
    monkeypatch.setattr(staging.PinnedRing, "take", slow_take)
    torch.cuda._sleep(500_000_000)
    threads = [threading.Thread(target=sampler.begin, args=([s], [1000 + s])) for s in slots]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    want = [k - (1 << 64) if k >> 63 else k for k in (sequence_key(1000 + s) for s in slots)]
    assert sampler.rng_key[torch.tensor(slots, device=DEV)].tolist() == want
