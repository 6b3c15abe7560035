"""Rules of the kernel sources that no run can be relied on to show broken."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nemo_b200", "csrc")
MESH_TABLES = ("a.nbr", "a.cdel")   # written by no kernel


def functions(text):
    """(header, body) of each function definition at namespace level, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__(?:global|device)__[^;{}]*\([^;{}]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(0), text[m.end():i]


def test_dependent_launches_read_written_data_by_ordinary_loads():
    """A kernel launched by launch_dep starts while the kernel before it may still write the state: its loads
    on the read-only path are of the mesh tables alone, and its parameters promise nothing read-only."""
    files = {f: open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC)}
    deps = {k for t in files.values() for k in re.findall(r"launch_dep\((k_\w+)", t)}
    assert {"k_stage_euler64", "k_stage_mhd64", "k_stage_euler32", "k_stage_mhd", "k_mortar", "k_ctrl_step"} <= deps
    seen = set()
    for text in files.values():
        for head, body in functions(text):
            kernel = re.search(r"\b(k_\w+)\(", head)
            if kernel is None or kernel.group(1) not in deps:
                continue
            seen.add(kernel.group(1))
            assert "__restrict__" not in head, head
            assert "ld.global.nc" not in body, head
            for arg in re.findall(r"__ldg\(\s*&?([\w.\->]+)", body):
                assert arg in MESH_TABLES, (head, arg)
    assert seen == deps


def test_features_are_ordered_before_the_first_layer():
    """The learned indicator's features pass between the lanes of a warp through shared memory: a barrier that
    orders memory (a vote does not) stands between the writes and the reads."""
    text = open(os.path.join(CSRC, "stage_fp64.cu")).read()
    body, = [b for h, b in functions(text) if "epilogue64(" in h]
    between = body[body.index("feat[lane] = "):body.index("feat[i]")]
    assert "__syncwarp();" in between


def test_fallback_flag_is_written_by_its_own_element():
    """FP32 form: the flag of an element is set either way by a thread of that element, not cleared by a thread of
    another warp without a barrier before it is set."""
    text = open(os.path.join(CSRC, "stage_fp32.cu")).read()
    body, = [b for h, b in functions(text) if "epilogue32(" in h]
    assert re.findall(r"s_fb\[(.*?)\] =", body) == ["el"]
