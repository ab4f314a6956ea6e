"""An LBVH build whose sort gives up a look-back wait: with the poll limit at one, a build either
ends as usual or returns LTS_ERR_DEVICE and leaves no tree behind, and the passes after the one that
gave up touch nothing (their keys are no longer the counted ones).  In a child process, so that
the lowered limit stays out of the other tests."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
OK, ERR_STATE, ERR_DEVICE = 0, 7, 8  # LTS_ERR_* of include/lts_capi.h

_CHILD = r"""
import ctypes, json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import torch
import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes
lib = lts.library()
ctx = lts.Context(0)
sizes = [5000, 200003, 262144, 1000003]
tris = {n: scenes.random_triangles(n, seed=n) for n in sizes}
dev = {n: torch.from_numpy(t.reshape(-1).copy()).cuda() for n, t in tris.items()}
bufs = [torch.empty(262144, dtype=torch.int32, device="cuda") for _ in range(3)]
nodes = torch.empty((262144, 16), dtype=torch.int32, device="cuda")
root = torch.empty(6, device="cuda")
torch.cuda.synchronize()
ptr = lambda t: ctypes.c_void_p(t.data_ptr())
ctx.set_option("debug_spin_limit", 1)
calls = []
for _ in range(3):
    for n in sizes:
        ctx.check(lib.lts_bvh_build_device_async(ctx.h, ptr(dev[n]), n, lts.BVH_SORTED, -1))
        calls.append([lib.lts_bvh_dump_get(ctx.h, None), lib.lts_bvh_dump_get(ctx.h, None)])
        if n <= 262144:
            rc = lib.lts_bvh_build_noalloc(ptr(dev[n]), n, lts.BVH_SORTED, -1, ptr(bufs[0]), ptr(bufs[1]), ptr(nodes),
                                           ptr(bufs[2]), ptr(root), None)
            calls.append([rc, -1])
ctx.set_option("debug_spin_limit", 0)
same = True
for n in sizes:
    a = lts.build_bvh_triangles(ctx, tris[n])
    other = lts.Context(0)
    b = lts.build_bvh_triangles(other, tris[n])
    other.close()
    order = np.lexsort((a["sorted_ids"], a["sorted_codes"]))
    same = same and np.array_equal(order, np.arange(n)) and all(
        np.array_equal(a[k].view(np.int32), b[k].view(np.int32)) for k in a)
ctx.close()
print("RESULT " + json.dumps({"calls": calls, "same": bool(same)}))
"""


def test_a_look_back_that_runs_out(built_lib):
    p = subprocess.run([sys.executable, "-c", _CHILD, ROOT], capture_output=True, text=True, timeout=600, env=os.environ)
    assert p.returncode == 0, p.stderr[-3000:]
    r = json.loads([x for x in p.stdout.splitlines() if x.startswith("RESULT ")][-1][len("RESULT "):])
    print("builds that gave up:", sum(c[0] == ERR_DEVICE for c in r["calls"]), "of", len(r["calls"]))
    for first, second in r["calls"]:
        assert first in (OK, ERR_DEVICE), r["calls"]
        assert second in ((-1, OK) if first == OK else (-1, ERR_STATE)), r["calls"]
    assert r["same"]
