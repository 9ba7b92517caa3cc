"""The row kernel (csrc/split_kernel.cuh) at the sizes where its cut of a row can
go wrong, against the CPU oracle: vocabularies around a whole number of pieces
and of buckets, rows that do not start on 16 bytes, every number of blocks per row,
and every way of keeping the history. Ids and kept sets are exact, as everywhere."""
import numpy as np
import pytest

from gpu_util import assert_parity, make_params, np_u32, oracle_rows, run_batch, t_f32, t_logits
from test_sampler_gpu import check, make_batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def W(lily):
    import workloads as w
    return w


# 4 pieces per block at least (1024 bf16, 512 f32 logits); a bucket is 80 pieces.
EDGES = [2047, 2048, 2049, 16383, 16384, 16385, 20480 * 2 - 1, 20480 * 2 + 8, 60001]


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("vocab", EDGES)
def test_edges_of_the_cut(cuda, lily, W, vocab, bf16):
    rng = np.random.default_rng(vocab * 2 + bf16)
    for rows, k, kw in ((1, 1, {}), (2, 20, dict(history=300, rep=1.1)), (3, 64, dict(history=7, presence=0.4)),
                        (4, 0, dict(history=500, presence=0.5, frequency=0.2, n_bias=9, n_ban=3)),
                        (2, 65, dict(n_ban=5)), (1, 2, dict(history=4099, frequency=0.1))):
        b = make_batch(W, rng, rows, vocab, k, bf16, kind="zipf", **kw)
        check(cuda, lily, W, b, vocab, f"V={vocab} k={k} B={rows}")


@pytest.mark.parametrize("rows", [1, 18, 19, 37, 38, 74, 75, 148, 149])
def test_every_number_of_blocks_per_row(cuda, lily, W, rows):
    vocab = 20_011  # (odd: only every eighth bf16 row starts on 16 bytes)
    rng = np.random.default_rng(rows)
    for bf16, k, kw in ((True, 40, dict(history=5000, rep=1.2)), (False, 50, dict(history=600, frequency=0.3, n_bias=6))):
        b = make_batch(W, rng, rows, vocab, k, bf16, kind="zipf", **kw)
        check(cuda, lily, W, b, vocab, f"B={rows} bf16={bf16}")


def test_ties_fill_the_candidates(cuda, lily, W):
    # Coarse values: more logits reach the bound than one warp, then than the buffers
    # take (the general code draws those rows).
    rng = np.random.default_rng(5)
    for quantise in (16, 4, 1, 0.25):
        b = make_batch(W, rng, 2, 30_000, 50, True, kind="uniform", quantise=quantise, history=50, rep=1.1)
        check(cuda, lily, W, b, 30_000, f"steps of 1/{quantise}")


@pytest.mark.parametrize("rows", [16, 34, 65, 297, 315, 316, 620])
def test_rows_around_the_waves_and_the_argument_blocks(cuda, lily, W, rows):
    # 16 and 34: more clusters of eight or four than run at once; 65: the largest argument
    # block; from 149 on two blocks to an SM, the parameters stored by a launch of their own
    # (of 16 KB up to 315 rows, of 32 KB up to 615, then by a copy).
    vocab = 9_001
    rng = np.random.default_rng(rows)
    for bf16, k, kw in ((True, 64, dict(history=900, rep=1.2, n_bias=3, n_ban=2)), (False, 0, dict(presence=0.3, history=40)),
                        (False, 1, {}), (True, 30, dict(history=200, frequency=0.2))):
        b = make_batch(W, rng, rows, vocab, k, bf16, kind="zipf", **kw)
        check(cuda, lily, W, b, vocab, f"B={rows} bf16={bf16} k={k}")


def long_lists(W, rng, rows, vocab, k, bf16, length, **kw):
    """Rows of unequal lists up to `length` ids; the ids that a lost part of the list would change
    (each row's best logits, some of them several times) stand in the list's last quarter."""
    b = make_batch(W, rng, rows, vocab, k, bf16, kind="zipf", history=length, **kw)
    b.history_len = rng.integers(length - length // 8, length + 1, rows).astype(np.uint32)
    b.history_len[0] = length
    lf = b.logits_f32()
    for r in range(rows):
        n = int(b.history_len[r])
        best = np.argpartition(lf[r], vocab - 40)[vocab - 40:].astype(np.uint32)
        at = n - n // 4 + rng.choice(n // 4, 60, replace=False)
        b.history[r, at] = np.concatenate([best, best[:20]])
    return b


@pytest.mark.parametrize("rows,length,vocab,bf16", [
    (149, 6143, 20_011, True), (149, 6144, 20_480, False), (149, 6145, 50_304, True), (200, 8192, 20_011, False),
    (296, 8193, 20_011, True), (256, 20_000, 50_304, True), (160, 32_768, 20_011, False)])
def test_long_lists_with_two_blocks_per_sm(cuda, lily, W, rows, length, vocab, bf16):
    # More rows than SMs, not aligned (20011) or aligned but short: 6144 ids are what the
    # block's marking half has in flight at a time.
    rng = np.random.default_rng([rows, length, vocab])
    for k, kw in ((30, dict(rep=1.3)), (50, dict(presence=0.7)), (20, dict(frequency=0.4, rep=1.1)), (1, dict(presence=1.5))):
        b = long_lists(W, rng, rows, vocab, k, bf16, length, **kw)
        check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} n={length} {kw}", params_on_device=k == 50)


@pytest.mark.parametrize("vocab,bf16,owner", [(65_536, False, 0), (65_536, True, 3), (40_009, False, 7)])
def test_wide_rows_whose_candidates_are_one_blocks(cuda, lily, W, vocab, bf16, owner):
    # The blocks of a cluster send each other their sorted lists. Here one block has (nearly)
    # all candidates: the others have nothing to rank and are the first to be done, while
    # theirs and its lists are still on their way. Launch after launch, so that the next
    # one's blocks take their places.
    rng = np.random.default_rng([7, vocab, owner])
    rows, piece = 6, 256 if bf16 else 128
    x = rng.uniform(-8, -7, (rows, vocab)).astype(np.float32)
    mine = (np.arange(vocab) // piece) % 8 == owner
    x[:, mine] = rng.uniform(0, 8, (rows, int(mine.sum())))
    params = [dict(temperature=1.2, top_k=[0, 300, 1000][r % 3], top_p=0.98, min_p=0.0, seed=r) for r in range(rows)]
    b = W.Batch(W.to_bf16_bits(x) if bf16 else x, bf16, params, rng.random(rows, dtype=np.float32))
    want = oracle_rows(b)
    s = lily.SamplerScratch(vocab, max_rows=rows)
    logits, out = t_logits(cuda, b), cuda.zeros((40, rows), dtype=cuda.int32, device="cuda")
    prepared = [s.prepare_sample_batch(logits, make_params(lily, b), out[i], uniforms=t_f32(cuda, b.uniforms))
                for i in range(len(out))]
    for p in prepared:
        s.sample_prepared(p)
    cuda.cuda.synchronize()
    assert s.status() == lily.OK
    got = np_u32(out)
    assert all(list(row) == [d.token for d in want] for row in got)
    assert_parity(b, run_batch(cuda, lily, s, b), want, label=f"V={vocab} owner {owner}")
    s.close()


@pytest.mark.parametrize("barrier,block,lost", [(1, 0, True), (1, 1, False), (2, 0, True), (2, 1, False)])
def test_a_wait_of_a_narrow_row_that_runs_out(cuda, lily, W, barrier, block, lost):
    """A block that waits for the others of its row gives up after the handle's limit: the
    launch completes and its shared memory stays until nobody stores into it. Without the first
    block's own arrivals the row has no result, and the status says so once; with another
    block's missing the first one draws the row alone. The next launch is as ever."""
    vocab, rows = 60_001, 3
    b = make_batch(W, np.random.default_rng([barrier, block]), rows, vocab, 40, False, kind="zipf", history=300, rep=1.1)
    s = lily.SamplerScratch(vocab, max_rows=rows)
    s.set_wait_limit(2_000_000)
    s.inject_lost_arrival(barrier, block)
    res = run_batch(cuda, lily, s, b)
    want = oracle_rows(b)
    if lost:
        assert list(res.ids) == [0xFFFFFFFF] * rows and (res.status == 8).all() and not res.kept_n.any()
        assert s.status() == lily.ERR_TIMEOUT
    else:
        assert_parity(b, res, want)
    assert s.status() == lily.OK
    s.set_wait_limit(0)
    assert_parity(b, run_batch(cuda, lily, s, b), want)
    assert s.status() == lily.OK
    s.close()


@pytest.mark.parametrize("barrier,block,lost", [(1, 0, True), (3, 0, True), (3, 2, True), (5, 0, True), (5, 2, False)])
def test_a_wait_of_a_wide_row_that_runs_out(cuda, lily, W, barrier, block, lost):
    vocab, rows = 60_001, 2
    b = make_batch(W, np.random.default_rng([barrier, block, 1]), rows, vocab, 0, False, kind="zipf")
    s = lily.SamplerScratch(vocab, max_rows=rows)
    s.set_wait_limit(2_000_000)
    s.inject_lost_arrival(barrier, block)
    res = run_batch(cuda, lily, s, b)
    want = oracle_rows(b)
    if lost:
        assert list(res.ids) == [0xFFFFFFFF] * rows and (res.status == 8).all()
        assert s.status() == lily.ERR_TIMEOUT
    else:
        assert_parity(b, res, want)
    assert s.status() == lily.OK
    s.set_wait_limit(0)
    assert_parity(b, run_batch(cuda, lily, s, b), want)
    s.close()


def test_a_wait_for_an_argmax_and_for_a_shards_sums_that_runs_out(cuda, lily, W):
    vocab, rows = 60_001, 2
    b = make_batch(W, np.random.default_rng(3), rows, vocab, 40, False, kind="zipf")
    logits, out = t_logits(cuda, b), cuda.zeros(rows, dtype=cuda.int32, device="cuda")
    s = lily.SamplerScratch(vocab, max_rows=rows)
    s.set_wait_limit(2_000_000)
    s.inject_lost_arrival(1, 0)
    s.argmax_batch(logits, out)
    assert s.status() == lily.ERR_TIMEOUT and list(np_u32(out)) == [0xFFFFFFFF] * rows
    s.argmax_batch(logits, out)
    assert s.status() == lily.OK and list(np_u32(out)) == list(b.logits.argmax(1))
    # (the candidates are there, their sum is not)
    records = [cuda.zeros((rows, lily.SHARD_RECORD_BYTES), dtype=cuda.uint8, device="cuda") for _ in range(2)]
    s.shard_candidates(logits, make_params(lily, b), records[0], want_sums=True)
    assert s.status() == lily.OK
    s.inject_lost_arrival(4, 0)
    s.shard_candidates(logits, make_params(lily, b), records[1], want_sums=True)
    assert s.status() == lily.ERR_TIMEOUT
    good, bad = (r.cpu().numpy() for r in records)
    assert np.array_equal(good[:, :516], bad[:, :516]) and not bad[:, 516:].any() and good[:, 516:].any()
    s.close()


@pytest.mark.parametrize("barrier,block,k,share", [
    (1, 0, 40, 0.5), (2, 0, 40, 1.0), (1, 0, 1, 1.0),
    (1, 0, 0, 0.25), (3, 0, 0, 1.0), (3, 2, 0, 1.0), (5, 0, 0, 1.0), (5, 2, 0, 1.0)])
def test_a_lost_arrival_is_given_up_within_the_limit(cuda, lily, W, barrier, block, k, share):
    """However late in the row the meeting is: the limit bounds the wait, and the row's other waits
    for a block that gave up end with it. (What is missing costs the share of the limit its meeting has; a
    block that lost the lists keeps the others, which wait for its receipt, for the whole.)"""
    vocab, rows, limit = 60_001, 2, 40e6
    b = make_batch(W, np.random.default_rng([barrier, block, k]), rows, vocab, k, False, kind="zipf")
    s = lily.SamplerScratch(vocab, max_rows=rows)
    logits, out = t_logits(cuda, b), cuda.zeros(rows, dtype=cuda.int32, device="cuda")
    p = s.prepare_sample_batch(logits, make_params(lily, b), out, uniforms=t_f32(cuda, b.uniforms))
    s.sample_prepared(p)
    s.set_wait_limit(int(limit))
    s.inject_lost_arrival(barrier, block)
    t0, t1 = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
    cuda.cuda.synchronize()
    t0.record()
    s.sample_prepared(p)
    t1.record()
    cuda.cuda.synchronize()
    took = t0.elapsed_time(t1) * 1e6 / limit
    # (Beside the waits the launch takes microseconds; a quarter of the limit, 10 ms, is room for a busy host.)
    assert 0.95 * share < took < share + 0.25, took
    assert s.status() == (lily.OK if (barrier, block) == (5, 2) else lily.ERR_TIMEOUT)
    s.close()


RAISING = [dict(history=700, presence=-0.6), dict(history=3000, rep=0.7), dict(history=2000, frequency=-0.2, rep=1.1),
           dict(history=900, frequency=0.1, presence=-1.0, n_bias=9, n_ban=3), dict(history=5, presence=-40.0)]


@pytest.mark.parametrize("rows,vocab,bf16", [(1, 1024, False), (3, 2048, True), (4, 60_001, True), (20, 9_001, False),
                                             (70, 9_001, True), (149, 9_001, False)])
def test_penalties_that_raise_a_logit(cuda, lily, W, rows, vocab, bf16):
    # An emitted id may be among the best whatever its logit: with lists in every way of
    # keeping them, narrow, wide and greedy rows, parameters on either side.
    rng = np.random.default_rng([rows, vocab])
    for i, kw in enumerate(RAISING):
        b = make_batch(W, rng, rows, vocab, [40, 1, 0, 20, 64][i], bf16, kind="zipf", **kw)
        for r in range(0, rows, 3):  # the row's worst ids are on its list
            b.history[r, :4] = np.argpartition(b.logits_f32()[r], 4)[:4].astype(np.uint32)
        for dev in (False, True):
            check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} {kw}", params_on_device=dev)
        b = make_batch(W, rng, rows, vocab, [0, 40, 64, 1, 2][i], bf16, kind="uniform", **kw)
        check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} {kw} uniform")


@pytest.mark.parametrize("rows,vocab,bf16", [(1, 1024, True), (6, 8448, True), (5, 16_001, False), (40, 8200, False)])
def test_lists_that_cover_the_vocabulary(cuda, lily, W, rows, vocab, bf16):
    # Most ids have been emitted, some of them often: their multiplicities decide the bound.
    rng = np.random.default_rng([rows, vocab])
    for k, kw in ((20, dict(frequency=0.2, presence=0.5)), (0, dict(frequency=0.2)), (1, dict(frequency=0.7)),
                  (500, dict(frequency=0.05, n_bias=6, n_ban=2))):
        for n in (vocab // 7, 15_953, 32_000):
            b = make_batch(W, rng, rows, vocab, k, bf16, kind="zipf", history=n, **kw)
            b.history[::2] = rng.integers(0, vocab, b.history[::2].shape)  # (the other rows': mostly a few ids)
            b.history_len[:] = n
            check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} k={k} n={n}")


@pytest.mark.parametrize("same,length", [(16_383, 17_000), (16_384, 17_000), (33_000, 65_535), (65_535, 65_535),
                                         (15_358, 70_000), (15_359, 70_000), (66_000, 70_000)])
def test_one_id_as_often_as_a_mark_counts(cuda, lily, W, same, length):
    # (A half word less two flags; lists beyond 65535 ids are looked at one by one.)
    rng = np.random.default_rng([same, length])
    for frequency in (0.0001, -0.0001):
        b = make_batch(W, rng, 2, 9_001, 40, True, kind="zipf", history=length, frequency=frequency)
        top = b.logits_f32().argmax(1)
        for r in range(2):
            b.history[r] = rng.integers(0, 9_000, length)
            b.history[r] += b.history[r] >= top[r]  # (any id but the row's best)
            b.history[r, rng.choice(length, same, replace=False)] = top[r]
        b.history_len[:] = length
        s = lily.SamplerScratch(9_001, max_rows=2, max_history=70_000)
        assert_parity(b, run_batch(cuda, lily, s, b), oracle_rows(b), label=f"{same} times one id of {length}")
        s.close()


def test_more_ids_than_a_raising_count_holds(cuda, lily, W):
    # Lists of mostly one id, around the most that a half word counts: the longer one is the
    # general code's.
    rng = np.random.default_rng(8)
    b = make_batch(W, rng, 3, 9_001, 40, True, kind="zipf", history=40_000, frequency=-0.001)
    b.history[:, :16_300] = 17
    b.history_len[:] = [40_000, 16_383, 16_384]
    check(cuda, lily, W, b, 9_001, "long list")


@pytest.mark.parametrize("lists", [{}, dict(n_bias=7, n_ban=4)])
@pytest.mark.parametrize("pen", [dict(presence_penalty=-0.7), dict(frequency_penalty=-0.1, repetition_penalty=1.2)])
def test_penalties_that_raise_a_logit_of_a_slot(cuda, lily, W, pen, lists):
    rng = np.random.default_rng(12)
    rows, vocab = 5, 60_001
    b = make_batch(W, rng, rows, vocab, 40, False, kind="zipf", **lists)
    for p in b.params:
        p.update(pen)
    counts = np.zeros((rows, vocab), dtype=np.uint32)
    s = lily.SamplerScratch(vocab, max_rows=rows, max_history=0, counts_table=True)
    for r in range(rows):
        ids = rng.integers(0, vocab, 3000)
        ids[:4] = np.argpartition(b.logits[r], 4)[:4]
        if lists:
            ids[4:8] = b.bias_ids[r, :4]
        np.add.at(counts[r], ids, 1)
        s.write_counts(counts[r], slot=r)
    for dev in (False, True):
        res = run_batch(cuda, lily, s, b, count_slots=list(range(rows)), params_on_device=dev)
        assert_parity(b, res, oracle_rows(b, counts=counts))
        for r in range(rows):
            counts[r, res.ids[r]] += 1
            assert np.array_equal(s.read_counts(slot=r), counts[r])
    s.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("vocab", [511, 512, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097, 6000, 7300, 8192,
                                   9000, 10_001])
def test_short_rows(cuda, lily, W, vocab, bf16):
    # Around the least that the kernel takes (four pieces: 512 f32, 1024 bf16 logits), where
    # half of a block's warps have nothing, few blocks share a row and a wide row's bound comes
    # from parts of a thread's logits; with tens of rows few blocks share any row.
    rng = np.random.default_rng([vocab, bf16])
    for rows, k, kw in ((1, 20, dict(history=300, rep=1.1)), (2, 64, dict(history=9, presence=0.4, n_bias=5, n_ban=2)),
                        (3, 0, dict(history=400, rep=1.3, frequency=0.1)), (2, 910, {}), (1, 300, dict(n_ban=4)),
                        (40, 0, dict(history=200, presence=-0.5)), (80, 500, dict(history=200, presence=0.5)),
                        (3, 1023, dict(kind="uniform")), (150, 700, {})):
        b = make_batch(W, rng, rows, vocab, k, bf16, **{"kind": "zipf", **kw})
        check(cuda, lily, W, b, vocab, f"V={vocab} k={k} B={rows}", params_on_device=rows == 2)


def cut_by_min_p(x, temp, cut):
    """A min-p that ends a row's kept set at rank `cut` or, where the weights there are too close to each
    other, four ranks or more later; and that rank."""
    w = np.sort(x.astype(np.float64))[::-1] / temp
    w = np.exp(w - w[0])
    while w[cut - 1] < w[cut] * (1.0 + 1e-4):
        cut += 4
    return float(np.float32(np.sqrt(w[cut - 1] * w[cut]))), cut


@pytest.mark.parametrize("rows,vocab,bf16,most", [(6, 60_001, False, 1024), (30, 30_001, False, 1024),
                                                  (60, 60_001, False, 455), (100, 9_001, False, 227),
                                                  (100, 9_001, True, 227)])
def test_rows_that_keep_many_at_the_edges_of_their_runs(cuda, lily, W, rows, vocab, bf16, most):
    """A wide row's lists are put in order by runs of 32, its weights added up four at a time, each
    thread cuts among four of them: kept counts around multiples of both, uncut, ended by top-p, and
    ended by min-p at every one of a thread's four ranks. A row over eight, four and two blocks and in
    one, with up to as many kept as the kernel ranks there by itself."""
    rng = np.random.default_rng([rows, vocab])
    ks = [65, 66, 67, 68, 95, 96, 97, 127, 128, 129, 191, 193, 225, 226, 227, 255, 256, 257, 453, 454, 455, 511, 513, 1021,
          1022, 1023, 1024, 0]
    ways = [(k, way, i) for i, k in enumerate(k for k in ks if (k or 1024) <= most)
            for way in ("uncut", "top-p", "min-p", "min-p, an odd rank")]
    ended = {0: 0, 1: 0, 2: 0, 3: 0}
    for at in range(0, len(ways), rows):
        x = rng.normal(0.0, 2.0, (rows, vocab)).astype(np.float32)
        bits = W.to_bf16_bits(x) if bf16 else x
        values = W.bf16_bits_to_f32(bits) if bf16 else x
        params, ends = [], []
        for r in range(rows):
            k, way, i = ways[(at + r) % len(ways)]
            p, end = dict(temperature=1.1, top_k=k, seed=r), k or 1024
            if way == "top-p":
                p["top_p"], end = (0.9, 0.6, 0.3)[i % 3], None
            elif way != "uncut":
                half = end // 2
                p["min_p"], end = cut_by_min_p(values[r], 1.1, half - half % 4 + (2 * i + way.endswith("odd rank")) % 4)
                assert end < (k or 1024)
                ended[end % 4] += 1
            params.append(p)
            ends.append(end)
        b = W.Batch(bits, bf16, params, rng.random(rows, dtype=np.float32))
        want = oracle_rows(b)
        for p, end, d in zip(params, ends, want):  # (what ends the set is what the test means to end it)
            assert len(d.kept_ids) == end if end else len(d.kept_ids) < (p["top_k"] or 1024)
        s = lily.SamplerScratch(vocab, max_rows=rows)
        assert_parity(b, run_batch(cuda, lily, s, b), want, label=f"from {at}")
        assert s.status() == lily.OK
        s.close()
    assert min(ended.values()) > 0, ended


@pytest.mark.parametrize("kind", ["flat", "coarse", "even", "steep", "beside a power of two"])
def test_sums_of_many_weights_bit_for_bit(cuda, lily, W, kind):
    """The prefix sums of a row that keeps more than 384 are not one chain of adds, but have its bits:
    draws at sums and the values beside them, and the kept probabilities (weight / sum of all) bit for
    bit. Equal weights; weights that tie when they are rounded to the sum's last place; a tail that
    leaves the sum at a power of two for hundreds of adds (a chain after all)."""
    vocab, rows = 40_000, 8
    i = np.arange(vocab)
    profile = {"flat": np.maximum(i - 1400, 0) * -0.01, "coarse": i // 100 / -8.0, "even": i * -0.0005, "steep": i * -0.02,
               "beside a power of two": np.where(i < 256, 0.0, -10.0 - 0.0005 * (i - 256))}[kind].astype(np.float32)
    rng = np.random.default_rng(len(kind))
    s = lily.SamplerScratch(vocab, max_rows=rows)
    for k in (384, 385, 388, 511, 778, 1023, 1024):
        x = np.stack([rng.permutation(profile) for _ in range(rows)])
        b = W.Batch(x, False, [dict(temperature=1.0, top_k=k, seed=r) for r in range(rows)], np.zeros(rows, np.float32))
        for at in (0.999, 0.51, 0.1, 0.003):
            for r, d in enumerate(oracle_rows(b)):  # u: a prefix sum over the mass, or up to three floats beside it
                n = len(d.kept_ids)  # (fewer than k where a tail adds nothing any more: the sum before it is all)
                assert n == k or kind == "steep"
                u = np.cumsum(d.kept_prob.astype(np.float32), dtype=np.float32)[int(at * n)].view(np.uint32)
                b.uniforms[r] = min((u + np.uint32(r) - np.uint32(4)).view(np.float32), np.float32(1 - 2.0 ** -24))
            want, res = oracle_rows(b), run_batch(cuda, lily, s, b)
            assert_parity(b, res, want, label=f"{kind} k={k} at {at}")
            for r, d in enumerate(want):
                bits = d.kept_prob.astype(np.float32).view(np.uint32)
                assert np.array_equal(res.kept_probs[r, :len(bits)].view(np.uint32), bits), f"{kind} k={k} row {r}"
    assert s.status() == lily.OK
    s.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,vocab", [(2, 5_000), (7, 40_003), (9, 20_000), (63, 9_001), (65, 9_001), (147, 9_001)])
def test_a_row_does_not_depend_on_what_the_others_bring(cuda, lily, W, rows, vocab, bf16):
    """The kernel is compiled for what a launch's rows bring: the same rows drawn among themselves, beside
    one that keeps many, one whose penalties can raise a logit, with (empty) lists, with their
    parameters on the device, the greedy ones by the argmax call too. (Shards and proposals have tests of
    their own.)"""
    rng = np.random.default_rng([rows, vocab, bf16])
    b = make_batch(W, rng, rows, vocab, 20, bf16, kind="zipf", history=600, presence=0.4, frequency=0.1)
    for r in range(0, rows, 3):  # every third is greedy, without penalties
        b.params[r].update(temperature=0.0, presence_penalty=0.0, frequency_penalty=0.0)
    want = oracle_rows(b)
    s = lily.SamplerScratch(vocab, max_rows=rows + 1, max_list=8)

    def drawn(b, extra, **kw):
        res = run_batch(cuda, lily, s, b, **kw)
        cut = W.Batch(b.logits[:rows], bf16, b.params[:rows], b.uniforms[:rows])
        res.ids, res.status = res.ids[:rows], res.status[:rows]
        assert_parity(cut, res, want, label=extra)

    drawn(b, "among themselves")
    drawn(b, "parameters on the device", params_on_device=True)
    for extra, more in (("keeps many", dict(top_k=0, temperature=1.1)), ("raises", dict(repetition_penalty=0.9, top_k=5))):
        one = make_batch(W, rng, 1, vocab, 20, bf16, kind="zipf", history=600)
        both = W.Batch(np.concatenate([b.logits, one.logits]), bf16, b.params + [dict(one.params[0], **more)],
                       np.concatenate([b.uniforms, one.uniforms]))
        both.history = np.concatenate([b.history, one.history])
        both.history_len = np.concatenate([b.history_len, one.history_len])
        drawn(both, extra)
    b.bias_ids, b.bias_vals = np.zeros((rows, 4), np.uint32), np.zeros((rows, 4), np.float32)
    b.bias_len = np.zeros(rows, np.uint32)
    drawn(b, "empty lists")
    ids = cuda.zeros(rows, dtype=cuda.int32, device="cuda")
    s.argmax_batch(t_logits(cuda, b), ids)
    greedy = np.arange(0, rows, 3)
    assert np.array_equal(np_u32(ids)[greedy], np.array([want[r].token for r in greedy], np.uint32))
    assert s.status() == lily.OK
    s.close()


@pytest.mark.parametrize("rows,vocab", [(75, 327_680), (75, 330_003), (149, 197_003)])
def test_more_buckets_than_a_word_has_bits(cuda, lily, W, rows, vocab):
    # A row in one block whose thread has 32 buckets, 33, and 33 with two blocks to an SM: those that reach the
    # bound are listed 32 at a time.
    rng = np.random.default_rng(rows + vocab)
    b = make_batch(W, rng, rows, vocab, 20, False, history=30, rep=1.1)
    for r in range(rows):  # (the best ones all over the row, its last bucket among them)
        b.logits[r, rng.integers(0, vocab, 12)] += 3.0
        b.logits[r, vocab - 1 - rng.integers(0, 400, 4)] += 4.0
    check(cuda, lily, W, b, vocab, f"B={rows} V={vocab}")


@pytest.mark.parametrize("rows,vocab,bf16", [
    (4, 81_920, False), (4, 81_921, False), (4, 82_304, False), (5, 151_937, False), (4, 163_840, False), (4, 163_843, False),
    (4, 163_840, True), (4, 163_841, True), (5, 262_143, True),
    (24, 40_960, False), (24, 41_003, False), (24, 100_353, True), (50, 20_483, False), (50, 40_001, False), (50, 60_007, True)])
def test_rows_that_keep_many_and_hold_their_second_bucket(cuda, lily, W, rows, vocab, bf16):
    """Rows without lists that keep more than 320 do not read the second of two
    buckets again: kept counts around that, shares of one, two and three buckets (in one cluster too: a
    bucket is 80 pieces of 512 bytes), rows over eight, four and two blocks that do not start on 16 bytes."""
    rng = np.random.default_rng([rows, vocab, bf16])
    ks = [65, 319, 320, 321, 384, 385, 1024, 640, 0]
    for kw in ({}, dict(history=700, rep=1.2)):
        b = make_batch(W, rng, rows, vocab, 0, bf16, kind="zipf", **kw)
        for r in range(rows):
            b.params[r].update(top_k=ks[(r + len(kw)) % len(ks)], top_p=1.0, min_p=0.0)
        check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} {kw}")
        for p in b.params:  # (all of them on one side)
            p["top_k"] = 448
        check(cuda, lily, W, b, vocab, f"B={rows} V={vocab} {kw} 448 kept")
