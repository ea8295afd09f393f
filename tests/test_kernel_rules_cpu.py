"""Rules of order that every kernel source keeps, checked on the text.

A kernel that breaks one of them may still give right results in a run, so
these are looked for in the sources and not in outputs.
"""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "parode_b200" / "csrc"


def _sources():
    for f in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"/\*.*?\*/", "", f.read_text(), flags=re.S)
        yield f.name, re.sub(r"//[^\n]*", "", text)


def _block(text, at):
    """The text from the brace at `at` to the one that closes it."""
    depth = 0
    for k in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[at:k + 1]
    raise AssertionError("unbalanced braces")


def _kernels():
    for name, text in _sources():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            brace = text.index("{", m.end())
            if ";" not in text[m.end():brace]:
                yield f"{name}:{m.group(1)}", _block(text, brace)


def _depth(body, at):
    return body.count("{", 0, at) - body.count("}", 0, at)


def test_peer_shared_memory_is_written_between_cluster_barriers():
    """A peer's shared memory is written only once every CTA of the cluster is
    known to run, and no CTA leaves while another may still write to it: a
    cluster wait outside every loop comes before the first remote store and
    one after the last."""
    store = re.compile(r"store_remote\(|shared::cluster\.")
    wait = re.compile(r"cluster_(?:barrier|wait)\(\)")
    seen = 0
    for name, body in _kernels():
        stores = [m.start() for m in store.finditer(body)]
        if not stores:
            continue
        seen += 1
        waits = [m.start() for m in wait.finditer(body) if _depth(body, m.start()) == 1]
        assert waits and waits[0] < stores[0], f"{name}: a remote store before the cluster's first barrier"
        assert waits[-1] > stores[-1], f"{name}: no barrier after the last remote store"
    assert seen >= 2


def test_shared_memory_limits_are_constants():
    """The dynamic shared memory limit belongs to the function on the device, not
    to the launch: a host thread that sets the size of its own launch lowers
    the limit under another thread's.  Every limit is a constant."""
    constant = re.compile(r"^(?:\(int\))?\s*(?:k[A-Z]\w*|C::smem|\d+(?: \* \d+)*)$")
    seen = 0
    for name, text in _sources():
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)\);", text):
            seen += 1
            assert constant.match(m.group(1).strip()), f"{name}: limit {m.group(1).strip()} of one launch"
    assert seen >= 10


def test_dependent_kernels_wait_before_they_read():
    """A kernel launched as a dependent sees the results of the grids before it
    after griddepcontrol.wait only.  Every thread waits once, at the top level
    of the kernel or at the start of its warp's role, not in a helper called
    where the reads happen to be."""
    seen = 0
    for name, body in _kernels():
        waits = [m.start() for m in re.finditer(r"grid_dep_wait\(\)", body)]
        if not waits:
            continue
        seen += 1
        for at in waits:
            # the enclosing blocks: none may be a lambda's
            starts, depth = [], 0
            for k in range(at - 1, -1, -1):
                if body[k] == "}":
                    depth += 1
                elif body[k] == "{":
                    if depth == 0:
                        starts.append(k)
                    else:
                        depth -= 1
            for k in starts[:-1]:
                assert not re.search(r"\[[&=]?\]\s*(?:\([^()]*\)\s*)?$", body[:k]), f"{name}: waits inside a lambda"
    assert seen >= 10
