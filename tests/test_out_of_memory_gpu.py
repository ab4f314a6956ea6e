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


def test_renders_after_ones_that_did_not_fit(built_lib):
    """A film (92 + 34 MB), the splats of a bidirectional render (47 MB beside a film of 63 + 24) and
    per-sample records (98 + 66 MB) that do not fit into 120 MB: the small renders after them are those
    before."""
    r = child(r"""
d = tempfile.mkdtemp()
sc, sub = scenes.write_tri_light_box(d, level=1)
ctx = lts.Context(0)
def render(w, h, which, spp=1, record=False):
    s = lts.Scene.parse(ctx, d, sc, sub, w, h)
    return lts.PathTracingIntegrator(2, 3, s, integrator=which).render(spp, 3, record=record, film=not record)
mega, bdpt = lts.INTEGRATOR_MEGAKERNEL, lts.INTEGRATOR_BDPT
close = lambda a, b: bool(np.allclose(a, b, rtol=1e-5, atol=1e-6))  # the film's sums are atomic, in doubles
a, b, c = render(64, 64, mega)["film"], render(64, 64, bdpt)["film"], render(64, 64, mega, record=True)["L"]
out["film"] = code(lambda: render(2048, 1400, mega))
out["a"] = close(render(64, 64, mega)["film"], a)
out["splat"] = code(lambda: render(1400, 1400, bdpt))
out["b"] = close(render(64, 64, bdpt)["film"], b)
out["record"] = code(lambda: render(64, 64, mega, spp=2000, record=True))
out["c"] = bool(np.array_equal(render(64, 64, mega, record=True)["L"], c))
out = {k: (v if isinstance(v, bool) else [v[0], v[1] if isinstance(v[1], str) else ""]) for k, v in out.items()}
ctx.close()
""", 120)
    for k in ("film", "splat", "record"):
        assert r[k][0] != 0 and "out of memory" in r[k][1], r
    assert r["a"] and r["b"] and r["c"], r


def test_a_dump_without_memory_for_the_flattened_tree(built_lib):
    """60,000 triangles: 4.9 MB of tree and sort buffers fit into 7 MB, the flattened tree's 3.8 MB beside them
    do not.  The dump is the one of a build with room, whole or in parts."""
    r = child(r"""
n = 60000
tris = scenes.random_triangles(n, seed=4)
dev = torch.from_numpy(tris.reshape(-1).copy()).cuda()
torch.cuda.synchronize()
ctx = lts.Context(0)
ctx.check(lib.lts_bvh_build_device_async(ctx.h, ctypes.c_void_p(dev.data_ptr()), n, lts.BVH_SORTED, -1))
a, d = lts._dump_arrays(n)
out["rc"] = lib.lts_bvh_dump_get(ctx.h, ctypes.byref(d))
left = np.zeros(2 * n - 1, np.int32)
part = lts.BvhDump(None, None, None, left.ctypes.data, None, None)
out["part"] = lib.lts_bvh_dump_get(ctx.h, ctypes.byref(part))
out["device_mb"] = ctx.metrics().device_bytes / 2**20
from oracle import lbvh_np
codes, ids = lbvh_np.stable_sort(*lbvh_np.morton_codes(tris, -1))
l, r = lbvh_np.karras_topology(codes)
out["order"] = bool(np.array_equal(a["sorted_codes"], codes) and np.array_equal(a["sorted_ids"], ids))
out["tree"] = bool(np.array_equal(a["node_left"][: n - 1], l) and np.array_equal(a["node_right"][: n - 1], r)
                   and np.all(a["node_left"][n - 1:] == -1) and np.all(a["node_right"][n - 1:] == -1)
                   and np.array_equal(left, a["node_left"]))
out["key"] = bool(np.array_equal(a["node_key"], np.concatenate([np.full(n - 1, -1), np.arange(n)]).astype(np.int32)))
mn, mx = lbvh_np.tri_bounds(tris)
lbvh_np.check_tree(a["node_left"], a["node_right"], a["node_bounds"], np.concatenate([mn, mx], 1)[ids])
ctx.close()
""", 7)
    assert r["rc"] == 0 and r["part"] == 0 and r["device_mb"] < 7, r
    assert r["order"] and r["tree"] and r["key"], r


def test_a_large_tree_without_memory_for_its_small_blocks(built_lib):
    """4,200,000 triangles: 391 MB with the forests of blocks of 256 leaves, 357 MB with those of 512, which is
    what 360 MB (377 million bytes) hold.  Both blocks build the same tree."""
    body = r"""
import hashlib
n = 4200000
g = torch.Generator(device="cuda").manual_seed(3)
x = (torch.rand((n, 1, 3), generator=g, device="cuda") + torch.randn((n, 3, 3), generator=g, device="cuda") * 1e-3).reshape(-1)
torch.cuda.synchronize()
ctx = lts.Context(0)
ctx.check(lib.lts_bvh_build_device_async(ctx.h, ctypes.c_void_p(x.data_ptr()), n, lts.BVH_SORTED, -1))
out["mb"] = ctx.metrics().device_bytes / 1e6
a, d = lts._dump_arrays(n)
ctx.check(lib.lts_bvh_dump_get(ctx.h, ctypes.byref(d)))
out["tree"] = hashlib.sha256(b"".join(a[k].tobytes() for k in sorted(a))).hexdigest()
ctx.close()
"""
    small, large = child(body, 360), child(body, 4096)
    assert small["mb"] < 377 < large["mb"], (small, large)
    assert small["tree"] == large["tree"]


def test_a_network_that_did_not_fit(built_lib):
    """A tree of 8,000 triangles leaves a third of 1 MB, the network needs half of it: its calls are then refused
    as they are without one, and a context with room has one."""
    r = child(r"""
x = torch.from_numpy(scenes.random_triangles(8000, seed=1).reshape(-1).copy()).cuda()
f, o = torch.zeros((64, 96), dtype=torch.bfloat16, device="cuda"), torch.zeros((64, 3), device="cuda")
torch.cuda.synchronize()
ctx = lts.Context(0)
ctx.check(lib.lts_bvh_build_device_async(ctx.h, ctypes.c_void_p(x.data_ptr()), 8000, lts.BVH_SORTED, -1))
call = lambda c: lib.lts_mlp_forward_device_async(c.h, ctypes.c_void_p(f.data_ptr()), 64, ctypes.c_void_p(o.data_ptr()))
out["init"] = [lib.lts_mlp_init(ctx.h, 1), lib.lts_mlp_init(ctx.h, 1)]
out["call"] = call(ctx)
ctx.close()
ctx = lts.Context(0)
out["again"] = [lib.lts_mlp_init(ctx.h, 1), call(ctx)]
torch.cuda.synchronize()
out["ones"] = bool((o == 1).all())  # every activation of zero features is 0, and exp(0) is 1
ctx.close()
""", 1)
    assert r["init"][0] != 0 and r["init"][1] != 0 and r["call"] == 7, r  # LTS_ERR_STATE
    assert r["again"] == [0, 0] and r["ones"], r
