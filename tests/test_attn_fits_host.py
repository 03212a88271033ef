"""Clusters of the attention launches where the device has no room for sixteen CTAs of one, or for any (csrc/attn_plan.h, compiled for the host)."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "attn_plan.h"
using namespace hm;
// room: CTAs of one cluster that the device holds at once
extern "C" void plan(int batch, int group, int kvh, int hd, int bf16, int pages, int most, int room, int* out) {
    int asked = 0;
    auto fits = [&](const AttnPlan& p) {
        ++asked;
        bool all = !p.decode_cluster || p.cut(batch, true).nsplit <= room;
        for (int M = 1; M <= 64; ++M) all = all && (!p.cluster || p.cut(M, false).nsplit <= room);
        return all;
    };
    const AttnPlan p = attn_plan_that_fits(batch, group * kvh, kvh, hd, bf16 != 0, pages, 148, most > 0, most, fits);
    out[0] = p.cluster; out[1] = p.decode_cluster; out[2] = p.by_pages; out[3] = asked;
    out[4] = p.cut(batch, true).nsplit; out[5] = p.scratch_splits();
}
"""
SHAPES = [(1, 6, 2, 128, 1, 63), (1, 7, 2, 64, 0, 250), (2, 2, 8, 128, 0, 5), (4, 8, 4, 128, 1, 64), (1, 8, 4, 128, 0, 157)]


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("fits")
    (d / "fits.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "homura_b200", "csrc"), "-o", str(d / "fits.so"), str(d / "fits.cpp")])
    lib = C.CDLL(str(d / "fits.so"))

    def call(shape, most, room):
        out = (C.c_int * 6)()
        lib.plan(*shape, most, room, out)
        return dict(zip(("cluster", "decode", "by_pages", "asked", "splits", "scratch"), out))

    return call


@pytest.mark.parametrize("shape", SHAPES)
def test_clusters_shrink_to_what_fits(plan, shape):
    whole, eight, none = plan(shape, 16, 16), plan(shape, 16, 8), plan(shape, 16, 7 if shape[-1] > 7 else 4)
    assert whole["decode"] and whole["by_pages"] == min(shape[-1], 16) and whole["asked"] == 1
    assert eight["decode"] and eight["by_pages"] == min(shape[-1], 8) and eight["splits"] <= 8
    assert not none["decode"] and not none["cluster"] and none["asked"] == 2 and none["splits"] <= none["scratch"]


def test_nothing_is_asked_without_clusters(plan):
    assert plan((1, 6, 2, 128, 1, 63), 0, 0)["asked"] == 0
    assert plan((40, 6, 2, 128, 1, 63), 16, 0)["asked"] == 0
