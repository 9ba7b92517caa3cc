"""Which kernel a call takes depends on what its rows bring. Whichever it is, it is on the device when the
handle is made: no call after that allocates there, and a call of a kind that the process has not made before
may be captured. In processes of their own, whose first calls these are."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = '''
import sys
import numpy as np, torch
import lily_b200 as lily

VOCAB, ROWS = 16_384, 160
g = torch.Generator(device="cuda").manual_seed(5)
full = lambda shape, v: torch.full(shape, v, dtype=torch.int32, device="cuda")
logits = {"f32": 3.0 * torch.randn((ROWS, VOCAB), generator=g, device="cuda")}
logits["bf16"] = logits["f32"].bfloat16()
uniforms = torch.rand(ROWS, generator=g, device="cuda")
history, length = torch.randint(0, VOCAB, (ROWS, 16), generator=g, device="cuda", dtype=torch.int32), full((ROWS,), 16)
ids = torch.randint(0, VOCAB, (ROWS, 4), generator=g, device="cuda", dtype=torch.int32)
values, four = torch.ones((ROWS, 4), device="cuda"), full((ROWS,), 4)
draft = [torch.softmax(logits["f32"][:2], 1), ids[:2, 0].contiguous()]
records = torch.zeros((ROWS, lily.SHARD_RECORD_BYTES), dtype=torch.uint8, device="cuda")
device_params = lambda ps: torch.from_numpy(np.frombuffer(b"".join(bytes(p) for p in ps), dtype=np.uint8).copy()).cuda()
NARROW, WIDE = dict(temperature=0.9, top_k=20), dict(temperature=0.9, top_k=0)
PENALTY, RAISES = dict(NARROW, presence_penalty=0.5), dict(NARROW, presence_penalty=-0.5)

def calls(s):
    """(name, call, its outputs)"""
    for rows in (3, 40, 120, 160):
        for dtype in ("f32", "bf16"):
            x, u, out = logits[dtype][:rows], uniforms[:rows], full((rows,), -1)
            lists = dict(bias_ids=ids[:rows], bias_vals=values[:rows], bias_len=four[:rows])
            past = dict(history_ids=history[:rows], history_len=length[:rows])
            for name, p, kw in (("narrow", NARROW, {}), ("wide", WIDE, {}), ("lists", NARROW, lists), ("penalty", PENALTY, past),
                                ("wide, lists", WIDE, lists), ("raises", RAISES, past)):
                host = [lily.SamplingParams(seed=r, **p) for r in range(rows)]
                yield (f"{rows} {dtype} {name}", lambda st, x=x, p=host, u=u, o=out, kw=kw:
                       s.sample_batch(x, p, o, uniforms=u, stream=st, **kw), out)
                yield (f"{rows} {dtype} {name}, on the device", lambda st, x=x, p=device_params(host), u=u, o=out, kw=kw:
                       s.sample_batch(x, p, o, uniforms=u, params_on_device=True, stream=st, **kw), out)
            yield f"{rows} {dtype} argmax", lambda st, x=x, o=out: s.argmax_batch(x, o, stream=st), out
            host = [lily.SamplingParams(seed=r, **NARROW) for r in range(rows)]
            yield (f"{rows} {dtype} shard", lambda st, x=x, p=host, r=rows:
                   s.shard_candidates(x, p, records[:r], want_sums=True, stream=st), records[:rows])
            if rows <= 64:
                yield (f"{rows} {dtype} merge", lambda st, p=host, u=u, o=out, r=rows:
                       s.merge_draw(records[None, :r], p, o, uniforms=u, stream=st), out)
    accepted = full((1,), 0)
    for dtype in ("f32", "bf16"):
        out = full((3,), -1)
        yield (f"{dtype} proposal", lambda st, x=logits[dtype][:3], o=out:
               s.spec_verify(x, lily.SamplingParams(seed=1, **NARROW), draft[1], o, accepted, step0=3, q_dense=draft[0],
                             stream=st), out)

free = lambda: torch.cuda.mem_get_info()[0]
scratch = lily.SamplerScratch(VOCAB, max_rows=ROWS, max_history=64, max_list=8)
todo = list(calls(scratch))
stream = torch.cuda.Stream()
torch.cuda.synchronize()
if sys.argv[1] == "memory":
    for name, call, _ in todo:
        before = free()
        call(stream)
        torch.cuda.synchronize()
        assert free() == before, f"{name}: {before - free()} bytes"
else:
    for name, call, out in todo:
        if name.startswith("160") and "device" not in name and "argmax" not in name:
            continue  # (more rows than a launch's arguments hold: their parameters are staged, which is not for a capture)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            call(stream)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        captured = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        call(stream)
        torch.cuda.synchronize()
        assert torch.equal(captured, out), name
        assert int(out.ne(0).sum()) > 0, name
        del graph
assert scratch.status() == lily.OK
print(len(todo), "calls")
'''


@pytest.mark.parametrize("what", ["memory", "capture"])
def test_first_calls(cuda, lily, what):
    r = subprocess.run([sys.executable, "-c", CHILD, what], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    assert r.stdout.strip().endswith("calls")
