"""How the attention launches of steps and small passes are cut (csrc/attn_plan.h), compiled for the host: what holds for every shape."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "attn_plan.h"
using namespace hm;
extern "C" void cut(int batch, int group, int kvh, int hd, int bf16, int pages, int clusters, int M, int decode, int* out) {
    const AttnPlan p(batch, group * kvh, kvh, hd, bf16 != 0, pages, 148, clusters != 0, 16);
    const AttnCut c = p.cut(M, decode != 0);
    out[0] = c.nsplit; out[1] = c.cluster; out[2] = c.early_pages; out[3] = p.scratch_splits();
    out[4] = attn_pick_nsplit(M, kvh, pages, 148, bf16 != 0); out[5] = attn_pick_nsplit(batch, kvh, pages, 148, bf16 != 0);
}
"""
SOURCE += '''
extern "C" int stream_from(int hd, int bf16, int group, int M, int ctas, int early, int two_fit) { return attn_stream_from(hd, bf16 != 0, group, M, ctas, early != 0, two_fit != 0, 148); }
'''
SHAPES = [(batch, group, kvh, hd, bf16, pages) for batch in (1, 2, 4, 8, 40) for group in (1, 3, 8) for kvh in (1, 2, 4, 8) for hd in (64, 128) for bf16 in (0, 1) for pages in (1, 2, 17, 64, 65, 80, 81, 100, 125, 157, 256, 257, 1000)]


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "homura_b200", "csrc"), "-o", str(d / "plan.so"), str(d / "plan.cpp")])
    lib = C.CDLL(str(d / "plan.so"))

    def call(shape, M, decode, clusters=True):
        out = (C.c_int * 6)()
        lib.cut(*shape, int(clusters), M, int(decode), out)
        return dict(zip(("nsplit", "cluster", "early", "scratch", "model", "batch_model"), out))

    call.lib = lib
    return call


def test_launches_fit_their_merge(cut):
    for shape in SHAPES:
        for clusters in (True, False):
            for M, decode in ((shape[0], True), (1, False), (8, False), (40, False), (64, False)):
                c = cut(shape, M, decode, clusters)
                assert 1 <= c["nsplit"] <= (16 if c["cluster"] else c["scratch"]), (shape, M, decode, c)
                assert (c["early"] > 0) == decode
                assert clusters or not c["cluster"]


def test_passes_over_several_rows_of_a_sequence_are_cut_as_without_clusters(cut):
    """Beyond 1024 tokens only steps are clusters; the splits of the other passes know nothing of that."""
    for shape in SHAPES:
        if shape[-1] > 64:
            for M in (1, 2, 8, 40, 64):
                c = cut(shape, M, False)
                assert not c["cluster"] and c["nsplit"] == min(c["model"], c["batch_model"]), (shape, M, c)


def test_pages_kept_in_shared_memory(cut):
    """Through global scratch a split of 128-wide heads keeps its pages as long as two CTAs fit an SM, and splits of two pages keep them in clusters too."""
    for shape in SHAPES:
        batch, group, kvh, hd, _, pages = shape
        c = cut(shape, batch, True)
        ctas = batch * kvh * c["nsplit"]
        if ctas > 2 * 148:
            assert c["early"] == 1
        elif hd == 64 and c["cluster"] and ctas <= 32 and -(-pages // c["nsplit"]) > 2:
            assert c["early"] == 2, (shape, c)
        elif hd == 64 or (not c["cluster"] and group > 2):
            assert c["early"] == 9, (shape, c)
        elif c["cluster"] and ctas > 32 and -(-pages // c["nsplit"]) == 2:
            assert c["early"] == 9, (shape, c)


def test_clusters_of_steps_on_long_caches(cut):
    """Eight (row, KV head) pairs of many 128-wide heads leave the clusters beyond 2560 tokens; fewer pairs and fewer heads do not."""
    for batch, group, kvh, hd, bf16, pages, want in [(4, 6, 2, 128, 1, 160, 1), (4, 6, 2, 128, 1, 161, 0), (2, 8, 4, 128, 1, 250, 0), (1, 2, 8, 128, 1, 250, 1), (4, 7, 2, 64, 0, 250, 1), (1, 8, 4, 128, 1, 250, 1), (1, 2, 8, 128, 0, 81, 0), (1, 2, 8, 128, 0, 80, 1)]:
        assert cut((batch, group, kvh, hd, bf16, pages), batch, True)["cluster"] == want, (batch, group, kvh, hd, bf16, pages)


def test_pages_from_which_a_cluster_streams(cut):
    """(head width, bf16 pages, heads per KV head, rows, CTAs, reads ahead, two CTAs per SM): pages.  Where the streaming kernel was the slower one it waits for more."""
    for args, want in [((64, 0, 7, 1, 32, 1, 1), 5), ((64, 1, 7, 1, 32, 1, 1), 3), ((64, 0, 4, 1, 16, 1, 1), 3), ((64, 0, 8, 4, 128, 1, 1), 3), ((64, 0, 8, 4, 256, 1, 1), 16), ((64, 1, 1, 2, 256, 0, 1), 16),
                       ((64, 0, 8, 8, 320, 1, 1), 5), ((64, 1, 8, 8, 256, 1, 1), 3), ((64, 0, 8, 8, 320, 0, 1), 7), ((64, 0, 7, 40, 320, 0, 1), 10), ((64, 1, 8, 40, 320, 0, 1), 5),
                       ((128, 0, 6, 40, 320, 0, 0), 8), ((128, 1, 6, 40, 320, 0, 1), 3), ((128, 0, 2, 1, 128, 1, 0), 5), ((128, 0, 6, 1, 32, 1, 0), 3), ((128, 1, 6, 4, 128, 1, 0), 5)]:
        assert cut.lib.stream_from(*args) == want, args
