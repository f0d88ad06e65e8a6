"""Kernels launched with programmatic stream serialization are resident while their predecessor still writes their input: none
of them may read step data through read-only loads (__ldg, ld.global.nc, const __restrict__ pointers)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lcdrsimulator_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def function(text, name):
    """Parameter list and body of a function."""
    m = re.search(r"\b" + name + r"\(", text)
    i = text.index("{", m.end())
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
    return text[m.end():i], text[i:j]


def test_no_read_only_loads_behind_a_dependent_launch():
    tiled, kzm, qsr = source("qsr_tiled.cuh"), source("kzm.cu"), source("qsr.cu")
    launched = set(re.findall(r"launch_pdl\(\s*([A-Za-z_0-9<>? :]+?),", tiled + kzm + qsr))
    assert launched == {"k", "k_sweep_tiled<kMode>", "noise ? k_kzm_step_ring<true> : k_kzm_step_ring<false>"}
    for text, name in ((tiled, "process_tile"), (tiled, "k_step_tiled"), (tiled, "k_sweep_tiled"),
                       (tiled, "k_step_ensemble"), (kzm, "k_kzm_step_ring")):
        params, body = function(text, name)
        assert "__ldg" not in body and ".nc." not in body, name
        # what a step writes: fields and low words (the work list, masks and descriptors are made before any step)
        assert not re.search(r"const float\*\s*__restrict__", params), name
    # the accessors of the field
    for name in ("SmemQ", "SmemQRt", "GlobQRt"):
        body = tiled[tiled.index("struct " + name + " {"):]
        assert "__ldg" not in body[:body.index("};")], name
