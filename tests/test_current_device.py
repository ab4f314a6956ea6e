"""Entry points that work on a context's stream make the context's device current first: a program may
have another device current, where an allocation would land on the wrong GPU and a launch on the
context's stream would be refused.  Read from the source; no second GPU is needed."""
import os
import re

from conftest import ROOT

CAPI = os.path.join(ROOT, "lighttransportsimulation_gb300", "csrc", "capi.cu")
# what a body that touches the device mentions (helpers of the file included)
WORK = re.compile(r"ctx->stream\b|\bdo_build\(|\bdump_bvh\(|\bray_queries\(|\bdev_alloc\(|\bcheck_device_error\(|\bcudaM")


def functions(text):
    """(name, body) of the functions that take a context first: from their line to the closing brace in
    column 0."""
    for m in re.finditer(r"^(?:int|void) (\w+)\(lts_ctx\*? ?\*?ctx\b", text, re.M):
        yield m.group(1), text[m.end():text.index("\n}", m.end())]


def test_device_is_set_before_device_work():
    text = open(CAPI).read()
    bodies = dict(functions(text))
    assert len(bodies) > 30 and "lts_bvh_dump_get" in bodies
    missing = []
    for name, body in bodies.items():
        if not name.startswith("lts_"):
            continue  # helpers are called by entry points
        at = WORK.search(body)
        if not at:
            continue
        sets = body.find("cudaSetDevice(ctx->device)")
        if sets < 0:  # or the helper that begins the body does
            sets = min((body.find(h + "(ctx") for h in bodies if not h.startswith("lts_") and
                        "cudaSetDevice(ctx->device)" in bodies[h] and h + "(ctx" in body), default=-1)
        if sets < 0 or sets > at.start():
            missing.append(name)
    assert not missing, missing
