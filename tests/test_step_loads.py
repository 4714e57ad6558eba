"""The step kernels are resident while the kernel before them writes: only what stays constant through a
step may be read through the read-only path, whose loads a wait does not order."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cil_cuda_gb300", "csrc")
# network weights, the colony table (its copy into shared memory and a bin width), uploaded noise
CONSTANT = (r"w \+ kMlp", r"reinterpret_cast<const float4 \*>\(w \+ kMlp", r"src \+ i\b", r"&a\.col\[", r"a\.noise \+")


def _sources():
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(f) as h:
            yield os.path.basename(f), re.sub(r"//[^\n]*", "", h.read())


def test_read_only_loads_are_of_constant_data():
    seen = 0
    for name, text in _sources():
        for m in re.finditer(r"__ldg\(", text):
            arg = text[m.end():m.end() + 80]
            assert any(re.match(c, arg) for c in CONSTANT), "%s: __ldg(%s" % (name, arg[:40])
            seen += 1
    assert seen > 0


def test_step_kernels_have_no_restrict_parameters():
    # but the caller's positions, complete before cil_bin_elements_noalloc's first launch
    for name, text in _sources():
        for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\(([^{;]*?)\)\s*\{\s*enter_step_kernel|"
                             r"__global__[^{;]*?\b(k_\w+)\(([^{;]*?)\)\s*\{\s*cil::enter_step_kernel", text):
            kernel, params = (m.group(1), m.group(2)) if m.group(1) else (m.group(3), m.group(4))
            restrict = re.findall(r"const \w+ \*__restrict__ (\w+)", params)
            assert restrict == (["pos"] if kernel == "k_na_keys" else []), (name, kernel, restrict)
    assert "__restrict__" not in re.search(r"int colony_of_tile\(([^)]*)\)", dict(_sources())["cil_internal.cuh"]).group(1)
