"""A kernel that may be scheduled while its predecessor still writes (it calls chain_wait) must not read through
the read-only path: no const pointer parameter marked __restrict__ and no __ldg, in the kernel or in the device
functions that the pair kernels share, but for data that no kernel of the chain writes (a build's positions, the
batch's tables, the state that a time step saved before the rebinning).  Read from the sources: the compiler may
move such a load in front of the wait, which no run is sure to show."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "particle-interaction-with-optix_b200",
                    "csrc")
CONSTANT = {"x", "y", "z", "firsts", "sys", "vh", "ids"}
SHARED = ("pair_common.cuh", "pair_pass.cuh", "pair_cluster.cuh", "pair_compat.cu", "bin_common.cuh")


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def functions(text):
    """(head, body) of every function definition at the start of a line or after a template's."""
    for m in re.finditer(r"__global__[^{;]*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(0), text[m.end():i]


def misuse(text):
    bad = [p for p in re.findall(r"const [\w:]+\* __restrict__ (\w+)", text) if p not in CONSTANT]
    return bad + [e for e in re.findall(r"__ldg\(([^()]*)", text)
                  if not re.match(r"&(\w+)\[", e) or re.match(r"&(\w+)\[", e).group(1) not in CONSTANT]


def test_chained_kernels_read_with_ordinary_loads():
    chained = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        for head, body in functions(read(name)):
            if "chain_wait()" in body:
                chained += 1
                assert not misuse(head + body), (name, head.split("(")[-2][-30:], misuse(head + body))
    assert chained >= 18


def test_shared_device_functions_read_with_ordinary_loads():
    for name in SHARED:
        assert not misuse(read(name)), (name, misuse(read(name)))


def test_every_chained_launch_waits():
    kernels = {}
    for name in sorted(os.listdir(CSRC)):
        for head, body in functions(read(name)) if name.endswith((".cu", ".cuh")) else ():
            kernels[re.findall(r"(k_\w+)\s*\(", head)[-1]] = "chain_wait()" in body
    launched = set()
    for name in os.listdir(CSRC):
        if name.endswith(".cu"):
            launched |= set(re.findall(r"chain_launch\((k_\w+)", read(name)))
    assert launched and all(kernels[k] for k in launched), [k for k in launched if not kernels.get(k)]
