"""Source rules of the kernels that are launched while the previous kernel of the stream still runs (launch_next): they wait before
they touch global memory, and read nothing through the path for data that no one writes during the kernel's lifetime."""
import glob
import os
import re

from conftest import ROOT


def _sources():
    for path in sorted(glob.glob(os.path.join(ROOT, "sapa_b200", "csrc", "*.cu*"))):
        with open(path) as f:
            text = f.read()
        yield os.path.basename(path), re.sub(r"/\*.*?\*/", " ", re.sub(r"//[^\n]*", "", text), flags=re.S)


def _functions(text):
    """(qualifiers and parameters, body) of the __global__ and __device__ functions."""
    for m in re.finditer(r"__(?:global|device)__[^;{}]*\)[^;{}()]*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(0), text[m.end():at]


def test_dependent_kernels_read_through_the_coherent_path():
    ahead, waiting, texts = set(), set(), list(_sources())
    for _, text in texts:
        ahead |= set(re.findall(r"\blaunch_(?:next|next_with_l1|with_smem|persistent)\(\s*(?:mt == 32 \? )?(\w+)", text)) - {"void", "kernel", "Kernel"}
    for name, text in texts:
        for head, body in _functions(text):
            kernel = "__global__" in head and re.findall(r"(\w+)\s*\(\s*(?:const|unsigned|int)\b", head)[-1]
            waits = "begin_after_previous();" in body
            if waits:
                waiting.add(kernel)
            if kernel in ahead:
                assert "__restrict__" not in head, (name, head)
            if kernel in ahead or (not kernel and "begin_after_previous();" in text):      # device functions of these files serve such kernels
                body = body.replace("if constexpr (IN_ORDER) return __ldg(p);", "")
                assert "__ldg" not in body and not re.search(r"Bilinear<\w+, true>|(?:fetch_once|load8)<true", body), (name, head)
                for p in head.split(","):                 # `sm`: shared memory
                    assert not re.search(r"\bconst\b.*__restrict__ (?!sm$)", p.strip()), (name, p)
    assert ahead and ahead <= waiting, ahead - waiting
