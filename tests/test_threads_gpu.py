"""Calls from several threads of one process, in a process of its own so that they are the first on the device."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

FIRST_CALLS = """
import itertools, threading, torch
from helpers import Case
wrong = []
for H, k in itertools.product((8, 4, 2, 1), (0, 2, 4, 6, 8, 12)):
    # the same kernel with different ring and table sizes: what it may use of shared memory is set at the first call
    cases = [Case([360], H=H, Hq=4 * H, seed=3, k=k, page_size=ps) for ps in (8, 32)]
    out, barrier = [None, None], threading.Barrier(2)
    def first(i):
        barrier.wait()
        try:
            out[i] = cases[i].run(num_kv_splits=2)
        except Exception as e:
            wrong.append((H, k, "first", i, str(e)))
    threads = [threading.Thread(target=first, args=(i,)) for i in (0, 1)]
    for t in threads: t.start()
    for t in threads: t.join()
    for i, c in enumerate(cases):
        try:
            o, lse = c.run(num_kv_splits=2)
            if out[i] is not None and not (torch.equal(o, out[i][0]) and torch.equal(lse, out[i][1])):
                wrong.append((H, k, "differs", i))
        except Exception as e:
            wrong.append((H, k, "again", i, str(e)))
print(wrong)
raise SystemExit(1 if wrong else 0)
"""


def test_first_calls_of_two_threads_with_different_page_sizes():
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join((os.path.dirname(here), here)))
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
