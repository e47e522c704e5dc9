"""Rules that the kernels' sources keep and no run can show."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gtr_b200", "csrc")


def _kernels():
    """(name, body) of every __global__ function."""
    for name in sorted(os.listdir(SRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(SRC, name)).read()
        text = re.sub(r"//[^\n]*", "", text)
        for m in re.finditer(r"__global__", text):
            i = text.index("{", text.index(")", text.index("__launch_bounds__", m.start()) if "__launch_bounds__" in text[m.start():m.start() + 80] else m.start()))
            depth, j = 0, i
            while True:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
                if depth == 0:
                    break
            yield f"{name}: {text[m.start():i].strip()[:100]}", text[i:j]


def test_dependents_are_released_after_the_block_has_its_tensor_memory():
    """A kernel launched to overlap may allocate tensor memory before it waits for its predecessor: it must not start while a block of
    that one still has to get its own.  (A block that leaves at once allocates none.)"""
    seen = 0
    for name, body in _kernels():
        if "tmem_alloc" not in body:
            continue
        seen += 1
        have = body.index("__syncthreads()", body.index("tmem_alloc"))       # every thread knows then that the allocation is done
        for m in re.finditer(r"pdl_release\(\);(\s*return)?", body):
            assert m.group(1) or m.start() > have, name
    assert seen >= 5
