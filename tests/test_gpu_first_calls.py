"""A context loads the common kernels when it is made: the first search of a fresh process costs about what the
second one does, whichever instance a row width, a degree and a batch size lead to."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes, json, sys
import numpy as np, torch
from glide_b200 import api
from glide_b200.params import Metric, SearchParameter
ctx = api.Context(0)
rng = np.random.default_rng(1)
t = lambda a: torch.from_numpy(a).to(ctx.torch_device)
out = {}
for dim in (128, 100, 960):
    for degree in (32, 64):
        for beam in (32, 64, 128) if degree == 32 else (64,):
            for nq in (1, 6000):
                n = 3000
                base, q = rng.random((n, dim), np.float32), rng.random((nq, dim), np.float32)
                graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
                sp = SearchParameter(top_k=10, beam=beam).derive(degree)
                args = (ctx, t(base), api.from_u32(ctx, graph), t(base[:2].copy()), api.from_u32(ctx, np.array([3, 77], np.uint32)), t(q), sp)
                times = []
                for _ in range(3):
                    api.search(*args)
                    split = (ctypes.c_float * 2)()
                    ctx.lib.glide_last_search_split_ms(ctx.handle, split)
                    times.append(split[1])
                out[f"dim {dim} degree {degree} beam {beam} queries {nq}"] = times
print("TIMES " + json.dumps(out))
"""


def test_the_first_search_of_a_process_takes_no_longer_than_the_next_ones():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    times = json.loads(r.stdout.split("TIMES ", 1)[1])
    # search kernels alone, by events on the stream. Loading one takes milliseconds; a first run also finds cold caches
    # and clocks, for which twice the later time and half a millisecond are allowed.
    slow = {k: v for k, v in times.items() if v[0] > 2 * max(v[1:]) + 0.5}
    assert not slow, slow
