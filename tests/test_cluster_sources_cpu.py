"""Kernels whose blocks store into their cluster peers' shared memory: a peer's memory exists only
from the moment that peer runs, and nothing but a cluster barrier shows that it does. A store that
comes too early is undefined and need not show up in any result, so the order is checked in the
source: each such kernel meets its cluster, unconditionally, before the first statement that can
reach a store, and the routine that stores ends with a barrier, so that no block leaves early."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "magma_b200" / "csrc"
REMOTE = re.compile(r"\b(?:st|ld|atom|red)\.shared::cluster|\bmap_shared_rank\b")


def _code(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    return re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)


def _body(text, start):
    """The braces' contents from the first '{' at or after start."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i + 1:j - 1]


def _functions(text, kind):
    """(name, body) of each function whose declaration holds `kind` and that is defined here."""
    out = []
    for m in re.finditer(kind + r"\b[^;{}]*?\b(\w+)\s*\([^;{}]*\)\s*\{", text):
        out.append((m.group(1), _body(text, m.end() - 1)))
    return out


def _remote_functions():
    """Device functions that reach a peer's shared memory, directly or through one another."""
    bodies = {}
    for f in sorted(CSRC.glob("*.cu*")):
        for name, body in _functions(_code(f), "__device__"):
            bodies[name] = bodies.get(name, "") + body
    hit = {n for n, b in bodies.items() if REMOTE.search(b)}
    while True:
        more = {n for n, b in bodies.items() if n not in hit and any(re.search(rf"\b{h}\b", b) for h in hit)}
        if not more:
            return hit, bodies
        hit |= more


def _kernels():
    hit, _ = _remote_functions()
    out = []
    for f in sorted(CSRC.glob("*.cu*")):
        for name, body in _functions(_code(f), "__global__"):
            if any(re.search(rf"\b{h}\b", body) for h in hit):
                out.append((f"{f.name}:{name}", body))
    return out


def test_the_cluster_kernel_is_found():
    assert [n for n, _ in _kernels()] == ["getrf_cluster.cu:getrf_cluster_kernel"]


@pytest.mark.parametrize("name,body", _kernels(), ids=[n for n, _ in _kernels()])
def test_cluster_meets_before_the_first_peer_store(name, body):
    hit, _ = _remote_functions()
    first = min(m.start() for h in hit for m in re.finditer(rf"\b{h}\b", body))
    sync = re.search(r"if constexpr \(CS > 1\)\s*cluster_sync<CS>\(\);", body)
    assert sync and sync.start() < first, f"{name}: no cluster barrier before the first access to a peer"
    before = body[:sync.start()]
    assert before.count("{") == before.count("}"), f"{name}: the barrier stands inside a branch or a loop"
    assert not re.search(r"\b(?:for|while|if\s*\(|return|continue)\b", before)


def test_each_matrix_ends_with_a_cluster_barrier():
    _, bodies = _remote_functions()
    loop = bodies["cluster_getrf"].rstrip()
    assert loop.endswith("}")
    inner = loop[:-1].rstrip()                      # the panel loop's last statement
    assert inner.endswith("cluster_sync<CS>();")
