"""The two parts of the LM head that the last projections of a step ask the L2 for follow one another: read from the source, since they change no result."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "homura_b200", "csrc")


def test_the_second_window_starts_where_the_first_one_ends():
    with open(os.path.join(CSRC, "engine.cu")) as f:
        source = f.read()
    assert re.search(r"pf_bytes_ = std::min\(PROJ_PF, w->bytes\(\) - off\);", source)  # the length of every window
    assert re.findall(r"prefetch\(&lm_head_(?:, ([^)]*))?\)", source) == ["", "PROJ_PF"]  # offsets, in the order of the launches
