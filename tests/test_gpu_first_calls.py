"""The first render calls of a process, made by several threads at once on jobs
of their own: the launch shapes that the first call works out are shared by all
threads. Images equal to those of the same jobs rendered one after the other."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import os, sys, threading
sys.path.insert(0, sys.argv[1])
import numpy as np
from hastyrenderer_gb300 import RenderJob
names = ["cornell", "field", "room", "room_nomis"] * 2
paths = [os.path.join(sys.argv[1], "tests", "golden", "scenes", n, "renderJob.json") for n in names]
jobs = [RenderJob(p) for p in paths]
start = threading.Barrier(len(jobs))
def call(j):
    start.wait()
    j.render_passes(3, sync=True)
threads = [threading.Thread(target=call, args=(j,)) for j in jobs]
for t in threads: t.start()
for t in threads: t.join()
for p, j in zip(paths, jobs):
    one = RenderJob(p)
    one.render_passes(3, sync=True)
    assert all(np.array_equal(one.read_sums(a)[0], j.read_sums(a)[0]) for a in range(3)), p
print("same")
"""


def test_first_calls_of_several_threads():
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
