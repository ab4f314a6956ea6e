"""Device buffers that cannot grow: an allocation cap (LTS_MAX_DEVICE_MB, in a child process) makes a call
fail part way through its allocations; the context must not go on using what it has already given
back."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
ERR_OOM = 5  # LTS_ERR_OOM of include/lts_capi.h

_HEAD = r"""
import ctypes, json, sys, tempfile
sys.path.insert(0, sys.argv[1])
import numpy as np
import torch
import lighttransportsimulation_gb300 as lts
from lighttransportsimulation_gb300 import scenes
lib = lts.library()
out = {}
def code(call):
    try:
        return 0, call()
    except lts.LtsError as e:
        return e.code, str(e)
"""


def child(body, cap_mb):
    p = subprocess.run([sys.executable, "-c", _HEAD + body + "\nprint('RESULT ' + json.dumps(out))\n", ROOT],
                       capture_output=True, text=True, timeout=600, env={**os.environ, "LTS_MAX_DEVICE_MB": str(cap_mb)})
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads([x for x in p.stdout.splitlines() if x.startswith("RESULT ")][-1][len("RESULT "):])


def test_a_build_after_one_that_did_not_fit(built_lib):
    """500,000 triangles need 32 MB of nodes, 6 MB of arrays and 4 MB of sort buffers: with 40 MB the
    last allocations fail.  A small build then starts from nothing and is right."""
    r = child(r"""
ctx = lts.Context(0)
small = scenes.random_triangles(50000, seed=1)
big = torch.from_numpy(scenes.random_triangles(500000, seed=2).reshape(-1).copy()).cuda()
torch.cuda.synchronize()
a = lts.build_bvh_triangles(ctx, small)
out["big"] = lib.lts_bvh_build_device_async(ctx.h, ctypes.c_void_p(big.data_ptr()), 500000, lts.BVH_SORTED, -1)
b = lts.build_bvh_triangles(ctx, small)
out["same"] = all(np.array_equal(a[k].view(np.int32), b[k].view(np.int32)) for k in a)
order = np.lexsort((b["sorted_ids"], b["sorted_codes"]))
out["sorted"] = bool(np.array_equal(order, np.arange(50000)))
ctx.close()
""", 40)
    assert r["big"] == ERR_OOM and r["same"] and r["sorted"], r
