"""A CTA of a cluster may store into another one's shared memory only once that one has started: every kernel that does so takes a
cluster barrier in front of its first such store.  Read from the source, since a store that comes too early goes right on nearly every run."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "homura_b200", "csrc")
FILES = ["attention.cu", "gemm_tc.cu", "gemv_kernel.cuh", "gla.cuh", "gqa_attn.cu", "gqa_talk.cuh", "kquant.cu", "kquant_gemm.cu", "moe.cu", "quant.cu", "recur.cu", "sampler.cu"]
PRIMITIVE = re.compile(r"\b(?:st_dsmem|st_async|red_dsmem)_\w+\(")
# (one behind a condition counts where the condition says that there is a cluster)
BARRIER = re.compile(r"(?<!\) )(?:if \((?:CL|\w+ > 1)\) )?\bcluster_(?:wait_acquire|sync_all)\(\)")
HEAD = re.compile(r"^[\w:<>,&* ]*?\b(\w+)\([^;{}]*\)\s*\{", re.M)


def functions(source):
    """(name, body, is a kernel) of the functions of a file, comments removed."""
    source = re.sub(r"//[^\n]*|/\*.*?\*/", "", source, flags=re.S)
    source = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", source)
    for m in HEAD.finditer(source):
        if "__device__" not in m.group(0) and "__global__" not in m.group(0):
            continue
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[end], 0)
            end += 1
        yield m.group(1), source[m.end() : end], "__global__" in m.group(0)


def unguarded(source):
    """Kernels whose first remote store, their own or a helper's, has no cluster barrier in front of it."""
    found = list(functions(source))
    early = set()  # helpers that store before they take a barrier themselves

    def stores_first(name, body):
        calls = "|".join(map(re.escape, sorted(early - {name})))
        store = min((m.start() for p in ([PRIMITIVE] + ([re.compile(rf"\b(?:{calls})(?:<[^;()]*>)?\(")] if calls else [])) for m in [p.search(body)] if m), default=None)
        barrier = BARRIER.search(body)
        return store is not None and not (barrier and barrier.start() < store)

    while True:
        more = {name for name, body, kernel in found if not kernel and name not in early and not PRIMITIVE.match(name + "(") and stores_first(name, body)}
        if not more:
            return [name for name, body, kernel in found if kernel and stores_first(name, body)]
        early |= more


@pytest.mark.parametrize("name", FILES)
def test_clusters_have_started_before_stores_into_them(name):
    with open(os.path.join(CSRC, name)) as f:
        source = f.read()
    assert PRIMITIVE.search(source)
    assert unguarded(source) == []


def test_the_reader_finds_a_store_in_front_of_the_barrier():
    helper = "template <int N>\n__device__ __forceinline__ void push(float* p, float v) {\n    if (v > 0) st_dsmem_f32(dsmem_addr(p, 0u), v);\n    cluster_arrive_release();\n    cluster_wait_acquire();\n}\n"
    kernel = "template <int N>\n__global__ void __launch_bounds__(256, N == 1 ? 3 : 1) k(const Args a) {\n    %s\n    push<N>(a.p, 1.f);\n}\n"
    assert unguarded(helper + kernel % "cluster_sync_all();") == []
    assert unguarded(helper + kernel % "__syncthreads();  // cluster_sync_all();") == ["k"]
    assert unguarded(helper + kernel % "if (alias) cluster_sync_all();") == ["k"]
