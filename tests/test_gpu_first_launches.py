"""First launches of a kernel from several threads at once, with different amounts of shared memory: none may lower what another needs.
In a process of its own, where nothing has been launched yet."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu

_PROGRAM = """
import sys, threading
import torch
import dsv3_b200
from dsv3_b200 import _lib
from dsv3_b200.moe_seam import GroupedExperts
torch.set_default_dtype(torch.bfloat16)
THREADS = 8

def weight(n, k):
    w = torch.zeros(n, k, dtype=torch.float8_e4m3fn, device="cuda")
    w.scale = torch.ones(-(-n // 128), -(-k // 128), dtype=torch.float32, device="cuda")
    return w

def linear(m, n, k):
    x, w = torch.zeros(m, k, device="cuda"), weight(n, k)
    return lambda: dsv3_b200.fp8_linear(x, w, w.scale)

def experts(tokens, dim, inter):
    lin = lambda n, k: type("Lin", (), {"weight": weight(n, k), "scale_fmt": None})()
    e = [type("E", (), {"w1": lin(inter, dim), "w2": lin(dim, inter), "w3": lin(inter, dim)})() for _ in range(2)]
    grouped = GroupedExperts(e, e, 0)
    x, weights = torch.zeros(tokens, dim, device="cuda"), torch.ones(tokens, 2, device="cuda")
    indices = torch.tensor([[0, 1]] * tokens, device="cuda")
    return lambda: _lib.host.combine(grouped.run(x, weights, indices, 1024), None)

def at_once(calls):
    gate, failed = threading.Barrier(len(calls)), []
    def one(call):
        torch.set_default_dtype(torch.bfloat16)
        gate.wait()
        try:
            call()
        except Exception as e:
            failed.append(repr(e))
    threads = [threading.Thread(target=one, args=(c,)) for c in calls]
    for t in threads: t.start()
    for t in threads: t.join()
    for c in calls:                  # and whatever they left behind serves all of them
        try:
            c()
        except Exception as e:
            failed.append("later: " + repr(e))
    torch.cuda.synchronize()
    return failed

sizes = list(range(THREADS))
groups = [
    [linear(2, 3072, 8192 + 2048 * i) for i in sizes],             # eight warps
    [linear(2, 512, 65536 + 8192 * i) for i in sizes],             # four, clusters of eight
    [linear(12, 512, 32768 + 4096 * i) for i in sizes],
    [linear(2, 5120, 24576 + 4096 * i) for i in sizes],            # four row tiles
    [experts(1 + i % 8, 7168, 256 + 1024 * i) for i in sizes],
]
failed = [f for g in groups for f in at_once(g)]
print("\\n".join(failed))
sys.exit(1 if failed else 0)
"""


def test_first_launches_of_different_sizes():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([PKG, ROOT, os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", _PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
