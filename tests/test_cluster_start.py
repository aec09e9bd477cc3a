"""Kernels that write a peer CTA's shared memory wait for the cluster to have started.

A CTA of a cluster may access another's shared memory only once that CTA runs; being
scheduled together does not order their starts.  No run can show a missing barrier
reliably, so the rule is checked where it is written: in every kernel, a wait at a cluster
barrier stands before the first store to a peer."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tenet-py_b200" / "csrc"
REMOTE = r"st\.shared::cluster|st\.async|red\.shared::cluster|atom\.shared::cluster"
WAIT = r"barrier\.cluster\.wait"


def _functions(text, mark):
    """``{name: text}`` of the functions marked ``mark``, each up to a brace in column 0."""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(rf"^{mark}.*?^}}", text, re.M | re.S):
        name = re.search(r"(\w+)\s*\(", m.group().replace("__launch_bounds__(", ""))
        out[name.group(1)] = m.group()
    return out


def _first(pattern, text):
    m = re.search(pattern, text)
    return len(text) if m is None else m.start()


def _unguarded(text):
    """Kernels of ``text`` that store to a peer before any wait at a cluster barrier."""
    helpers = _functions(text, "__device__")

    def uses(pattern):  # directly or through a helper
        names = [n for n, body in helpers.items() if re.search(pattern, body)]
        return "|".join([pattern, *(rf"\b{n}\(" for n in names)])

    return [n for n, body in _functions(text, "__global__").items()
            if _first(uses(REMOTE), body) < _first(uses(WAIT), body)]


SEND = 'asm("st.shared::cluster.f64 [%0], %1;");'
MEET = 'asm("barrier.cluster.arrive;" "barrier.cluster.wait;");'


@pytest.mark.parametrize("body, ok", [
    (SEND + MEET, False), (MEET + SEND, True), ("put(1); meet();", False), (SEND, False),
    ("meet(); put(1);", True), ("// meet();\nput(1);", False), ("meet();", True)])
def test_the_check_sees_a_missing_barrier(body, ok):
    text = (f"__device__ void meet() {{\n{MEET}\n}}\n__device__ void put(int x) {{\n{SEND}\n}}\n"
            f"__global__ void __launch_bounds__(64)\nkernel(int x) {{\n{body}\n}}\n")
    assert _unguarded(text) == ([] if ok else ["kernel"])


@pytest.mark.parametrize("name", ["tnb_vec.cu", "tnb_svd_cluster.cu"])
def test_peers_are_written_after_a_cluster_barrier(name):
    text = (CSRC / name).read_text()
    assert re.search(REMOTE, text) and _unguarded(text) == []
