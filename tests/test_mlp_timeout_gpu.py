"""Radiance-cache kernels whose mbarrier waits run out: with the poll limit at one, inference and
training either end as usual or return LTS_ERR_DEVICE, having waited for the products and copies they
had issued before they freed their tensor memory; with the limit back, the same context gives the
results it gave before.  In a child process, so that the lowered limit stays out of the other tests."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
OK, ERR_DEVICE = 0, 8  # LTS_ERR_* of include/lts_capi.h

_CHILD = r"""
import json, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import lighttransportsimulation_gb300 as lts
ctx = lts.Context(0)
net = lts.RadianceCacheMLP(ctx, seed=5)
rng = np.random.default_rng(2)
n = 200001  # more than one round of tiles for inference and for training, the last one partial
f = (rng.random((n, 96)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
t = rng.random((n, 3)).astype(np.float32)
def code(call):
    try:
        return 0, call()
    except lts.LtsError as e:
        return e.code, None
before = net.forward(f)
_, (loss0, g0) = code(lambda: net.train_step(f, t, 0.0, want_grad=True))
ctx.set_option("debug_spin_limit", 1)
rc = [code(lambda: net.forward(f))[0] for _ in range(4)] + [code(lambda: net.train_step(f, t, 0.0))[0] for _ in range(4)]
ctx.set_option("debug_spin_limit", 0)
after = net.forward(f)
loss1, g1 = net.train_step(f, t, 0.0, want_grad=True)
# the gradient is summed over the SMs with atomics, in any order: n_sm roundings of partial sums of
# one sign or the other, bounded by 2^-24 x 152 x the largest gradient times a few
bound = 152 * 2.0**-24 * 16 * float(np.abs(g0).max())
print("RESULT " + json.dumps({"rc": rc, "forward_same": bool(np.array_equal(before, after)),
                              "grad": float(np.abs(g0 - g1).max()), "bound": bound, "loss": [loss0, loss1]}))
ctx.close()
"""


def test_waits_that_run_out_leave_the_context_usable(built_lib):
    p = subprocess.run([sys.executable, "-c", _CHILD, ROOT], capture_output=True, text=True, timeout=600, env=os.environ)
    assert p.returncode == 0, p.stderr[-3000:]
    r = json.loads([x for x in p.stdout.splitlines() if x.startswith("RESULT ")][-1][len("RESULT "):])
    print(r)
    assert all(c in (OK, ERR_DEVICE) for c in r["rc"]), r
    assert r["forward_same"] and r["grad"] <= r["bound"] and abs(r["loss"][0] - r["loss"][1]) <= 1e-4 * r["loss"][0], r
