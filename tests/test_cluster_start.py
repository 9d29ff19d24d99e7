"""Stores into another block's shared memory (sk_cluster.cuh) are legal only once that block has started,
which a completed cluster barrier shows and nothing else does. Read off the sources: in every kernel
that reaches storeRemote, an arrive and a wait stand before the first call that reaches it."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "splatkit-ios_b200" / "csrc"


def functions(text):
    """name -> (is a kernel, body) of every device function with a body."""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"__(global|device)__", text):
        head = re.compile(r"([A-Za-z_]\w*)\s*\(").finditer(text, m.end())
        name = next(h for h in head if h.group(1) not in ("__launch_bounds__", "__align__"))
        open_ = text.find("{", name.end())
        semicolon = text.find(";", name.end())
        if open_ < 0 or 0 <= semicolon < open_:
            continue
        depth, end = 1, open_ + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[name.group(1)] = (m.group(1) == "global", text[open_:end])
    return out


def first_call(body, names):
    found = [m.start() for n in names for m in re.finditer(rf"\b{n}\s*(<[^;()]*>)?\s*\(", body)]
    return min(found, default=None)


def sources():
    return [p for p in sorted(CSRC.glob("*.cu")) if "storeRemote" in p.read_text()]


def test_some_sources_store_into_other_blocks():
    assert sources()


@pytest.mark.parametrize("source", sources(), ids=lambda p: p.stem)
def test_a_cluster_barrier_completes_before_the_first_remote_store(source):
    found = functions(source.read_text())
    reaching = {"storeRemote"}
    while True:
        more = {n for n, (kernel, body) in found.items() if not kernel and first_call(body, reaching) is not None}
        if more <= reaching:
            break
        reaching |= more
    kernels = {n: body for n, (kernel, body) in found.items() if kernel and first_call(body, reaching) is not None}
    assert kernels
    for name, body in kernels.items():
        arrive, wait = first_call(body, ["clusterArrive"]), first_call(body, ["clusterWait"])
        assert arrive is not None and wait is not None, name
        assert arrive < wait < first_call(body, reaching), name
