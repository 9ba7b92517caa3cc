"""One row with host parameters (`sample_f32`, lily_sample_one) against the CPU oracle and
the batch entry point: the history's length travels in the launch's arguments, and so do the
step and the seed that the uniform is taken from."""
import numpy as np
import pytest

import oracle
from gpu_util import make_params, np_u32, oracle_rows, t_logits, t_u32
from test_sampler_gpu import make_batch

pytestmark = pytest.mark.gpu

STEP = 41


def draw_one(cuda, lily, scratch, b, history):
    """The row's ids by sample_f32 and by sample_batch (no draw: 0xFFFFFFFF)."""
    logits, p = t_logits(cuda, b), make_params(lily, b)
    out = cuda.zeros(3, dtype=cuda.int32, device="cuda")
    lily.sample_f32(logits.view(-1), scratch, p[0], STEP, out[1:2], history_ids=history)
    kw = {}
    if history is not None and history.numel():  # (an empty list is refused there)
        kw = dict(history_ids=history.view(1, -1),
                  history_len=cuda.full((1,), history.numel(), dtype=cuda.int32, device="cuda"))
    scratch.sample_batch(logits, p, out[2:3], steps=[STEP], **kw)
    cuda.cuda.synchronize()
    got = np_u32(out)
    assert got[0] == 0
    return int(got[1]), int(got[2])


def check_one(cuda, lily, scratch, W, rng, vocab, bf16, n, at=0, k=40, label="", **kw):
    """n: ids of the history (None: no history), which start `at` words into their tensor."""
    b = make_batch(W, rng, 1, vocab, k, bf16, kind=kw.pop("kind", "zipf"), history=max(n or 0, 1), **kw)
    b.history_len[:] = n or 0
    b.params[0]["seed"] = int(rng.integers(0, 1 << 40))
    b.uniforms[0] = lily.uniform_for(b.params[0]["seed"], STEP)
    history = None
    if n is not None:
        whole = np.full(at + n, 0xFFFFFFFF, dtype=np.uint32)
        whole[at:] = b.history[0, :n]
        history = t_u32(cuda, whole)[at:]
    one, batch = draw_one(cuda, lily, scratch, b, history)
    want = oracle_rows(b)[0]
    token = want.token if want.status == oracle.OK else 0xFFFFFFFF
    assert one == token and batch == token, f"V={vocab} n={n} at={at} k={k} {kw} {label}: {one}, {batch}, oracle {token}"


@pytest.fixture(scope="module")
def W(lily):
    import workloads as w
    return w


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("vocab", [511, 512, 1023, 1024, 20_011, 151_936])
def test_one_row(cuda, lily, W, vocab, bf16):
    rng = np.random.default_rng([vocab, bf16])
    s = lily.SamplerScratch(vocab, max_history=10_000)
    for n, at in ((None, 0), (0, 0), (1, 0), (3, 0), (3, 1), (700, 3), (8193, 2), (10_000, 0)):
        check_one(cuda, lily, s, W, rng, vocab, bf16, n, at, k=[40, 1, 0, 64][(n or 0) % 4], rep=1.1, frequency=0.05)
    for kw in (dict(rep=0.8), dict(presence=-0.4), dict(presence=-0.4, frequency=0.1)):  # these can raise a logit
        check_one(cuda, lily, s, W, rng, vocab, bf16, 500, 1, **kw)
    assert s.status() == lily.OK
    s.close()


def test_one_row_that_the_general_code_draws(cuda, lily, W):
    # Ties by the hundred, and a history of one id more often than a raising count holds: the
    # row's parameters, step and history length go along.
    rng = np.random.default_rng(11)
    vocab = 30_000
    s = lily.SamplerScratch(vocab, max_history=40_000)
    for bf16 in (False, True):
        check_one(cuda, lily, s, W, rng, vocab, bf16, 50, k=50, kind="uniform", quantise=0.25, rep=1.1, label="ties")
        check_one(cuda, lily, s, W, rng, vocab, bf16, 20_000, k=50, frequency=-0.001, label="long")
    s.close()


def test_one_row_with_a_bad_list_or_a_nan(cuda, lily, W):
    rng = np.random.default_rng(12)
    vocab = 20_011
    b = make_batch(W, rng, 1, vocab, 40, False, kind="zipf", history=101, rep=1.1)
    s = lily.SamplerScratch(vocab, max_history=100)
    assert draw_one(cuda, lily, s, b, t_u32(cuda, b.history[0])) == (0xFFFFFFFF, 0xFFFFFFFF)
    assert s.status() == lily.ERR_DEVICE_ROW  # a list longer than max_history
    b.logits[0, 7] = np.nan
    assert draw_one(cuda, lily, s, b, t_u32(cuda, b.history[0, :100])) == (0xFFFFFFFF, 0xFFFFFFFF)
    assert s.status() == lily.ERR_DEVICE_ROW and s.status() == lily.OK
    s.close()
