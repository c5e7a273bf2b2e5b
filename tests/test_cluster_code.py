"""Device code, read on the host.  No kernel touches another CTA's shared memory before a barrier over the whole cluster has
said that all of its CTAs run.  And what a kernel of a chain reads behind its wait, because the kernel before it wrote it, is not
declared as data that nobody writes: such a load may be moved ahead of the wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "megaqwen_b200", "csrc")
ACCESS = re.compile(r"\b(?:cluster_map|st_cluster_f32|ld_cluster|leader_addr)\(")
BARRIER = re.compile(r"\b(?:cluster_wait|cluster_sync|cluster_sync_all)\(\);")


def bodies(text):
    """(name, body) of every function, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\b(\w+)\(([^;{}]*)\) \{\n", text):
        if text[text.rfind("\n", 0, m.start()) + 1].isspace():               # a statement inside a function
            continue
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        kernel = re.search(r"\b(k_\w+)\(", m.group(0))              # behind its launch bounds
        yield kernel.group(1) if kernel else m.group(1), text[m.end():at - 1]


def first_access_without_barrier(body):
    """Whether an access stands before any barrier that every thread of every variant passes (one at the outermost level)."""
    depth = 0
    for token in re.finditer(r"[{}]|" + ACCESS.pattern + "|" + BARRIER.pattern, body):
        t = token.group(0)
        if t in "{}":
            depth += 1 if t == "{" else -1
        elif BARRIER.match(t):
            if depth == 0:
                return False
        else:
            return True
    return False


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_cluster_barrier_before_the_first_access(name):
    text = open(os.path.join(CSRC, name)).read()
    helpers = {"cluster_map", "st_cluster_f32", "ld_cluster", "leader_addr"}
    bad = [f for f, body in bodies(text) if f not in helpers and first_access_without_barrier(body)]
    assert not bad, bad


def test_the_rule_sees_the_kernels():
    seen = {f for n in ("sk_chain.cuh", "tc_gemm2.cuh", "hy_attention.cu") for f, body in bodies(open(os.path.join(CSRC, n)).read()) if ACCESS.search(body)}
    assert {"k_sk", "k_gemm2", "merge_pieces"} <= seen
    assert first_access_without_barrier("x(); if (a) { cluster_wait(); } st_cluster_f32(p, v);")


WEIGHTS = {"embed", "audio", "w", "wq", "wk", "cos", "sin"}            # written by nothing on the stream


@pytest.mark.parametrize("name", ["prefill.cu", "sk_chain.cuh", "mma_attention.cuh", "tc_attention.cuh", "tc_gemm.cuh", "tc_gemm2.cuh"])
def test_only_weights_are_read_only(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    found = 0
    for m in re.finditer(r"\b(\w+)\(([^;{}]*)\) \{\n", text):
        if text[text.rfind("\n", 0, m.start()) + 1].isspace() or re.search(r"\bk_kv_quantize", m.group(0)):      # the latter is launched without overlap
            continue
        for p in re.finditer(r"const \w+\* __restrict__ (\w+)", m.group(0)):
            found += 1
            assert p.group(1) in WEIGHTS, (m.group(1), p.group(1))
    assert found or name != "prefill.cu"
