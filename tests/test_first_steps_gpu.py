"""GPU: the first steps of several engines on several host threads at once, in a process that has launched none of their kernels."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.join(os.path.dirname(__file__), "..")

PROGRAM = r"""
import threading, torch
from asd_b200.engine import MezilixEngine, RivetarEngine
from asd_b200.models import mezilix, rivetar

def make(i):
    if i % 2:
        return MezilixEngine(mezilix.sized_config(2048, 1, 16, vocab=1024, ff=256), max_seqs=8, max_seq_len=64, max_tokens=64)
    return RivetarEngine(rivetar.sized_config(2048, 3, 16, vocab=1024, ff=2048), max_seqs=8, max_seq_len=64, max_tokens=64)

N = 8
engines = [make(i).load_random(seed=7 + i) for i in range(N)]
ids = torch.randint(0, 1024, (8, 1), generator=torch.Generator().manual_seed(1), dtype=torch.int32).cuda()
slots = torch.arange(8, dtype=torch.int32, device="cuda")
start = torch.zeros(8, dtype=torch.int32, device="cuda")
for e in engines:
    e._uniform_index_on(8, 1, ids.device)          # (index tensors: made on the default stream)
torch.cuda.synchronize()
gate, first, wrong = threading.Barrier(N), [None] * N, []

def step(i):
    try:
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            gate.wait()
            first[i] = engines[i].forward_uniform(ids, start, slots, 1)
        stream.synchronize()
    except Exception as e:
        wrong.append(f"engine {i}: {e}")

threads = [threading.Thread(target=step, args=(i,)) for i in range(N)]
for t in threads: t.start()
for t in threads: t.join()
for i, e in enumerate(engines):
    if first[i] is not None and not torch.equal(first[i], e.forward_uniform(ids, start, slots, 1)):
        wrong.append(f"engine {i}: other logits than alone")
    e.check_device()
print("\n".join(wrong) if wrong else "same")
"""


def test_first_steps_on_eight_threads():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=100)
    assert r.returncode == 0 and r.stdout.strip() == "same", (r.stdout, r.stderr[-2000:])
