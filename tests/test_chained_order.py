"""A pair kernel must find all SMs free when it is scheduled: crowded cells put its work into few neighbouring
blocks, and those pile up on the SMs that come free first.  So the kernels launched directly in front of one let
their successor go (chain_next) only at their end or where all their blocks end at once.  Read from the sources,
since the pile-up shows in the time alone and not in every run."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "particle-interaction-with-optix_b200",
                    "csrc")
NEVER = {"pair_pass.cu": ["k_cellpair_list"], "bin.cu": ["k_descriptors"], "pair.cu": ["k_pair_config"]}
# where a kernel may let its successor go: no large cell to sort, one round of equal work, after the walk
ONLY = {"bin.cu": ("k_large_sort", r"if \(count <= 0\) chain_next\(\);"),
        "step.cu": ("k_verlet_carry", r"if \(\(long long\)gridDim\.x \* blockDim\.x >= n\) chain_next\(\);"),
        "pair_cluster.cu": ("k_pair_cluster", r"\}\s*__syncthreads\(\);\s*chain_next\(\);\s*reduce_totals")}


def body(name, kernel):
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = re.search(r"__global__[^{;]*\b%s\([^{;]*\{" % kernel, text).end()
    depth, i = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[start:i]


def test_kernels_in_front_of_a_pair_kernel_end_before_it_is_scheduled():
    for name, kernels in NEVER.items():
        for kernel in kernels:
            assert "chain_next" not in body(name, kernel), kernel
    for name, (kernel, form) in ONLY.items():
        text = body(name, kernel)
        assert text.count("chain_next") == 1 and re.search(form, text), kernel
