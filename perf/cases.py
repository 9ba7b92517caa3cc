"""Performance cases of the token sampler: one decode step's work, as a server calls it.

Every case is one call sequence through the package's public entry points
(`SamplerScratch.sample_batch`, `sample_f32`, `argmax_batch`, `spec_verify`,
`lmhead_logits`, `shard.sharded_lmhead_draw`) on inputs that already lie on the GPU.
Handles, argument blocks and output buffers are made once, as a decode loop makes them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import lily_b200 as lily
from lily_b200 import shard

K_CAP = lily.K_CAP

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
ELEMENT = {"f32": 4, "bf16": 2}


def listed():
    """The cases of everyday use, smallest to largest."""
    return [
        # A greedy request on a small vocabulary: the least work a call can have.
        {"name": "greedy 1 row", "kind": "greedy", "rows": 1, "vocab": 32768, "dtype": "f32"},
        # One interactive user: a single f32 row with a repetition penalty over its history.
        {"name": "single row", "kind": "one", "vocab": 151936, "history": 4096},
        # A few requests with everything on: mixed parameters, bias, bans, a forced id.
        {"name": "server 4 rows", "kind": "server", "rows": 4, "vocab": 151936, "dtype": "bf16", "history": 8192},
        # Requests whose penalty state is a histogram slot that each draw updates.
        {"name": "histogram slots 8 rows", "kind": "slots", "rows": 8, "vocab": 248320, "dtype": "f32"},
        # A drafting step that hands on its whole kept distribution (top-k off: 1024 candidates).
        {"name": "draft export 3 rows", "kind": "wide", "rows": 3, "vocab": 151936, "dtype": "f32"},
        # Verification of two drafted tokens against a dense draft distribution.
        {"name": "speculative 3 rows", "kind": "spec", "rows": 3, "vocab": 151936, "dtype": "bf16", "dense": True,
         "history": 0},
        # An ordinary batch on a vocabulary that no vector width divides.
        {"name": "ragged batch 24 rows", "kind": "batch", "rows": 24, "vocab": 50257, "dtype": "f32",
         "history": 1024, "device_params": False},
        # Continuous batching: requests come and go, so the parameters are host values.
        {"name": "batch 64 rows", "kind": "batch", "rows": 64, "vocab": 151936, "dtype": "bf16", "history": 8192,
         "device_params": False},
        # The throughput batch: long contexts, parameters resident on the GPU.
        {"name": "batch 256 rows", "kind": "batch", "rows": 256, "vocab": 151936, "dtype": "bf16", "history": 32768,
         "device_params": True},
        # A 4-bit head in affine storage, then the draw from its logits.
        {"name": "4-bit head 32 tokens", "kind": "head", "rows": 32, "vocab": 151936, "hidden": 2048, "bits": 4},
        # The same with 8-bit codes and few tokens: a small batch decodes.
        {"name": "8-bit head 4 tokens", "kind": "head", "rows": 4, "vocab": 248320, "hidden": 4096, "bits": 8},
        # The fused step on a symmetric int8 head: projection, candidates, merged draw.
        {"name": "int8 head 64 tokens", "kind": "fused", "rows": 64, "vocab": 262144, "hidden": 4096},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _vocab(rng, low=8192, high=262144):
    """Half of them padded to a multiple of 128, as checkpoints are; the others as they fall."""
    v = _log(rng, low, high)
    return max(low, v // 128 * 128) if rng.random() < 0.5 else v


def draw(rng):
    """One more case of the listed kinds, over the ranges that serving meets."""
    kind = rng.choice(["greedy", "one", "server", "slots", "wide", "spec", "batch", "batch", "head", "fused"])
    dtype = rng.choice(["f32", "bf16"])
    if kind == "greedy":
        return {"kind": kind, "rows": _log(rng, 1, 64), "vocab": _vocab(rng), "dtype": dtype}
    if kind == "one":
        return {"kind": kind, "vocab": _vocab(rng), "history": rng.randint(0, 8192)}
    if kind == "server":
        return {"kind": kind, "rows": _log(rng, 1, 12), "vocab": _vocab(rng), "dtype": dtype,
                "history": rng.randint(1, 16384)}
    if kind in ("slots", "wide"):
        return {"kind": kind, "rows": _log(rng, 1, 12), "vocab": _vocab(rng), "dtype": dtype}
    if kind == "spec":
        return {"kind": kind, "rows": rng.randint(2, 8), "vocab": _vocab(rng), "dtype": dtype,
                "dense": rng.random() < 0.5, "history": rng.choice([0, rng.randint(1, 8192)])}
    if kind == "batch":
        rows = _log(rng, 9, 256)
        return {"kind": kind, "rows": rows, "vocab": min(_vocab(rng, 32000), 256 * 151936 // rows), "dtype": dtype,
                "history": rng.randint(1, 32768), "device_params": rng.random() < 0.5}
    hidden = 512 * rng.randint(2, 8)
    vocab = _vocab(rng, 16384, 248320)
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 1, 64), "vocab": vocab, "hidden": hidden, "bits": rng.choice([4, 8])}
    return {"kind": kind, "rows": _log(rng, 1, 64), "vocab": vocab, "hidden": hidden}


# ------------------------------------------------------------------ inputs --


class _Inputs:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.rng = np.random.default_rng(seed)
        self.seed = seed

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device="cuda")

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.g, device="cuda")

    def ids(self, high, *shape):
        return torch.randint(0, high, shape, generator=self.g, device="cuda", dtype=torch.int32)

    def skewed_ids(self, high, *shape):
        """Token ids as text has them: few are frequent (a power law of exponent 1.3)."""
        u = torch.rand(shape, generator=self.g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
        return (u.pow(-1.0 / 0.3).clamp_max(1e15).long() % high).int()

    def logits(self, rows, vocab, dtype):
        """N(0, 3^2) plus a Zipf(1.1) bump over a permutation of the vocabulary per row."""
        out = torch.empty((rows, vocab), dtype=DTYPES[dtype], device="cuda")
        bump = 1.1 * torch.log(vocab / torch.arange(1, vocab + 1, device="cuda", dtype=torch.float64)).float()
        for r in range(rows):
            order = torch.randperm(vocab, generator=self.g, device="cuda")
            out[r] = 3.0 * self.normal(vocab) + bump[order]
        return out

    def choice(self, rows, vocab, n):
        return torch.from_numpy(np.stack([self.rng.choice(vocab, n, replace=False) for _ in range(rows)])
                                .astype(np.int32)).cuda()


def _full(rows, value):
    return torch.full((rows,), value, dtype=torch.int32, device="cuda")


def _outputs(rows, kept=0):
    out = {"ids": _full(rows, 0), "status": _full(rows, 0)}
    if kept:
        out["kept_n"] = _full(rows, 0)
        out["kept_ids"] = torch.zeros((rows, kept), dtype=torch.int32, device="cuda")
        out["kept_probs"] = torch.zeros((rows, kept), device="cuda")
    return out


def _steps(x, rows):
    return [int(v) for v in x.rng.integers(0, 1 << 20, rows)]


def prepare(case, seed):
    x = _Inputs(seed)
    state = {"kind": case["kind"]}
    state.update(_PREPARE[case["kind"]](case, x))
    return state


def _greedy(case, x):
    return {"logits": x.logits(case["rows"], case["vocab"], case["dtype"]), "out": {"ids": _full(case["rows"], 0)},
            "scratch": lily.SamplerScratch(case["vocab"], max_rows=case["rows"], max_history=0)}


def _one(case, x):
    v, h = case["vocab"], case["history"]
    params = lily.SamplingParams(temperature=0.7, top_k=20, top_p=0.95, repetition_penalty=1.05, seed=x.seed)
    return {"logits": x.logits(1, v, "f32").view(-1), "params": params, "step": _steps(x, 1)[0],
            "history": x.ids(v, h) if h else None, "out": {"ids": _full(1, 0)},
            "scratch": lily.SamplerScratch(v, max_rows=1, max_history=8192)}


def _server(case, x):
    rows, v, h = case["rows"], case["vocab"], case["history"]
    params = [lily.SamplingParams(temperature=[0.0, 0.6, 0.8, 1.0][r % 4], top_k=[0, 20, 40][r % 3],
                                  top_p=[1.0, 0.95, 0.8][r % 3], presence_penalty=0.5, frequency_penalty=0.2,
                                  seed=x.seed + r) for r in range(rows)]
    forced = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    if rows > 2:  # one request's thinking budget has run out
        forced[2] = int(x.rng.integers(0, v))
    return {"scratch": lily.SamplerScratch(v, max_rows=rows, max_history=16384),
            "logits": x.logits(rows, v, case["dtype"]), "params": params, "out": _outputs(rows),
            "kw": {"steps": _steps(x, rows), "history_ids": x.skewed_ids(v, rows, h), "history_len": _full(rows, h),
                   "bias_ids": x.choice(rows, v, 64), "bias_vals": 10.0 * x.ids(2, rows, 64).float() - 5.0,
                   "bias_len": _full(rows, 64), "ban_ids": x.choice(rows, v, 8), "ban_len": _full(rows, 8),
                   "forced_ids": forced}}


def _slots(case, x):
    rows, v = case["rows"], case["vocab"]
    scratch = lily.SamplerScratch(v, max_rows=rows, max_history=0, counts_table=True)
    for r in range(rows):  # each request has emitted 2048 tokens so far
        scratch.write_counts(np.bincount(x.skewed_ids(v, 2048).cpu().numpy(), minlength=v), slot=r)
    params = [lily.SamplingParams(temperature=0.7 + 0.05 * (r % 4), top_k=20, top_p=0.95, presence_penalty=0.5,
                                  frequency_penalty=0.1, seed=x.seed + r) for r in range(rows)]
    return {"scratch": scratch, "logits": x.logits(rows, v, case["dtype"]), "params": params, "out": _outputs(rows),
            "kw": {"steps": _steps(x, rows), "count_slots": list(range(rows))}}


def _wide(case, x):
    rows, v = case["rows"], case["vocab"]
    params = [lily.SamplingParams(temperature=1.3, top_k=0, min_p=0.02, seed=x.seed + r) for r in range(rows)]
    return {"scratch": lily.SamplerScratch(v, max_rows=rows, max_history=0),
            "logits": x.logits(rows, v, case["dtype"]), "params": params, "out": _outputs(rows, K_CAP),
            "kw": {"steps": _steps(x, rows)}}


def _spec(case, x):
    m, v, h = case["rows"], case["vocab"], case["history"]
    target = 2.0 * x.normal(m, v)
    drafted = 0.8 * target[:-1] + 0.6 * 2.0 * x.normal(m - 1, v)  # the draft head follows the target
    penalty = {"presence_penalty": 0.5, "repetition_penalty": 1.05} if h else {}
    params = lily.SamplingParams(temperature=1.0, top_k=20, top_p=0.95, seed=x.seed, **penalty)
    scratch = lily.SamplerScratch(v, max_rows=m, max_history=8192 + 8)
    kw = {}
    if case["dense"]:
        kw["q_dense"] = torch.softmax(drafted, dim=1)
        ids = torch.multinomial(kw["q_dense"], 1, generator=x.g).view(-1).int()
    else:  # what the drafting steps exported
        d = _outputs(m - 1, K_CAP)
        ids = d["ids"]
        scratch.sample_batch(drafted, [lily.draft_params(params)] * (m - 1), ids,
                             steps=[lily.draft_step(j) for j in range(m - 1)], kept_n=d["kept_n"],
                             kept_ids=d["kept_ids"], kept_probs=d["kept_probs"])
        kw.update(q_n=d["kept_n"], q_ids=d["kept_ids"], q_probs=d["kept_probs"])
    if h:
        kw["history_ids"] = x.skewed_ids(v, h)
    out = _outputs(m)
    out["accepted"] = _full(1, 0)
    return {"scratch": scratch, "logits": target.to(DTYPES[case["dtype"]]), "params": params, "draft_ids": ids,
            "out": out, "step0": _steps(x, 1)[0], "kw": kw}


def _batch(case, x):
    rows, v, h = case["rows"], case["vocab"], case["history"]
    params = [lily.SamplingParams(temperature=0.8, top_k=50, top_p=0.9, min_p=0.05, repetition_penalty=1.1,
                                  seed=x.seed + r) for r in range(rows)]
    state = {"scratch": lily.SamplerScratch(v, max_rows=rows, max_history=32768),
             "logits": x.logits(rows, v, case["dtype"]), "out": _outputs(rows),
             "kw": {"history_ids": x.ids(v, rows, h), "history_len": _full(rows, h), "uniforms": x.uniform(rows)}}
    if case["device_params"]:  # the same buffers every step: the argument block is made once
        # (it holds addresses: the tensors behind them stay alive with the state)
        raw = np.frombuffer(b"".join(bytes(p) for p in params), dtype=np.uint8).copy()
        state["d_params"] = torch.from_numpy(raw).cuda()
        state["prepared"] = state["scratch"].prepare_sample_batch(
            state["logits"], state["d_params"], state["out"]["ids"], out_status=state["out"]["status"],
            params_on_device=True, **state["kw"])
    else:
        state["params"] = params
    return state


def _head(case, x):
    t, v, k, bits = case["rows"], case["vocab"], case["hidden"], case["bits"]
    top = 2 ** bits - 1
    scales = (0.0002 + 0.0018 * x.uniform(v, k // 64)) * (127.0 / top)
    biases = -scales * (top / 2) * (0.9 + 0.2 * x.uniform(v, k // 64))
    params = [lily.SamplingParams(temperature=0.7, top_k=40, top_p=0.95, seed=x.seed + r) for r in range(t)]
    return {"scratch": lily.SamplerScratch(v, max_rows=t, max_history=0), "bits": bits,
            "codes": torch.randint(0, 256, (v, k * bits // 8), generator=x.g, device="cuda", dtype=torch.uint8),
            "scales": scales.bfloat16(), "biases": biases.bfloat16(), "hidden": x.normal(t, k).bfloat16(),
            "params": params, "steps": _steps(x, t),
            "out": {**_outputs(t), "logits": torch.zeros((t, v), device="cuda")}}


def _fused(case, x):
    t, v, k = case["rows"], case["vocab"], case["hidden"]
    params = [lily.SamplingParams(temperature=0.7, top_k=40, top_p=0.95, seed=x.seed + r) for r in range(t)]
    out = _outputs(t, K_CAP)
    out["lse"] = torch.zeros(t, device="cuda")
    return {"scratch": lily.SamplerScratch(v, max_rows=t, max_history=0, lmhead=True),
            "weights": torch.randint(-127, 128, (v, k), generator=x.g, device="cuda", dtype=torch.int8),
            "scales": (0.0002 + 0.0018 * x.uniform(v, k // 64)).bfloat16(), "hidden": x.normal(t, k).bfloat16(),
            "params": params, "steps": _steps(x, t), "out": out,
            "records": torch.zeros((t, lily.SHARD_RECORD_BYTES), dtype=torch.uint8, device="cuda")}


_PREPARE = {"greedy": _greedy, "one": _one, "server": _server, "slots": _slots, "wide": _wide, "spec": _spec,
            "batch": _batch, "head": _head, "fused": _fused}


# -------------------------------------------------------------------- run --


def run(state):
    kind, out, scratch = state["kind"], state["out"], state["scratch"]
    if kind == "greedy":
        scratch.argmax_batch(state["logits"], out["ids"])
    elif kind == "one":
        lily.sample_f32(state["logits"], scratch, state["params"], state["step"], out["ids"],
                        history_ids=state["history"])
    elif kind == "spec":
        scratch.spec_verify(state["logits"], state["params"], state["draft_ids"], out["ids"], out["accepted"],
                            step0=state["step0"], out_status=out["status"], **state["kw"])
    elif kind == "head":
        scratch.lmhead_logits(state["codes"], state["scales"], state["hidden"], out["logits"],
                              biases=state["biases"], code_bits=state["bits"])
        scratch.sample_batch(out["logits"], state["params"], out["ids"], steps=state["steps"],
                             out_status=out["status"])
    elif kind == "fused":
        shard.sharded_lmhead_draw(scratch, state["weights"], state["scales"], state["hidden"], state["params"],
                                  out["ids"], 0, steps=state["steps"], records=state["records"], want_sums=True,
                                  out_lse=out["lse"], out_status=out["status"], kept_n=out["kept_n"],
                                  kept_ids=out["kept_ids"], kept_probs=out["kept_probs"])
    elif "prepared" in state:
        scratch.sample_prepared(state["prepared"])
    else:
        kept = {k: out[k] for k in ("kept_n", "kept_ids", "kept_probs") if k in out}
        scratch.sample_batch(state["logits"], state["params"], out["ids"], out_status=out["status"], **kept,
                             **state["kw"])
    return out


# ------------------------------------------------------------------- work --


def work(case):
    """Each input once, each output once. A draw's arithmetic (a few operations per
    logit) is not what bounds it and counts as none; a head's is its contraction."""
    kind, v = case["kind"], case["vocab"]
    rows = case.get("rows", 1)
    if kind in ("head", "fused"):
        k = case["hidden"]
        bits = case.get("bits", 8)
        per_row = k * bits / 8 + (k // 64) * 2 * (2 if kind == "head" else 1)
        bytes_ = v * per_row + rows * k * 2 + (rows * v * 4 if kind == "head" else 0)
        return {"bytes": bytes_, "flops": 2.0 * rows * v * k}
    bytes_ = rows * v * ELEMENT[case.get("dtype", "f32")]
    if kind == "spec":
        history = case["history"]
        if case["dense"]:  # the accept test reads single probabilities, a rejected row's residual its k candidates'
            bytes_ += (rows - 1) * 4 * 21
        else:
            bytes_ += (rows - 1) * 8 * 20
    else:
        history = rows * case.get("history", 0)
    if kind == "slots":  # the slot's bits of emitted ids
        bytes_ += rows * v / 8
    if kind == "server":
        bytes_ += rows * (64 * 8 + 8 * 4 + 4)
    if kind == "wide":
        bytes_ += rows * K_CAP * 8
    return {"bytes": bytes_ + 4 * history, "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("head", "fused"):
        # 32-bit sums over the columns; a logit's error over the temperature is a
        # probability's relative error, and equal ranks may change places.
        return {"rel": 2e-5, "max": 8e-4, "differ": 0.01}
    if case["kind"] == "wide":
        return {"rel": 1e-6, "max": 1e-5}
    return "exact"
