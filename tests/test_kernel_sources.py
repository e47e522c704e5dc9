"""Rules that the kernels' sources keep and no run can show."""
import os
import random
import re
import shutil
import subprocess

import pytest

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


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"), reason="needs nvcc")
def test_spans_begin_where_they_should_in_the_longest_sequences(tmp_path):
    """floor(j * chunks / parts) up to 2^30 chunks, at the compiler's evaluation of the kernels' own expression."""
    rng = random.Random(1)
    cases = [(64, 64, j) for j in range(65)] + [(92683, 23171, 23170), (92683, 23171, 23171), (2 ** 30 - 1, 65535, 65534), (2 ** 30 - 1, 65535, 65535),
                                                (65535 + 65534, 65535, 65534), (46341, 46341, 46340)]
    for _ in range(100):
        n = rng.randrange(1, 2 ** rng.randrange(1, 31))
        parts = rng.randint(1, min(n, 65535))
        cases.append((n, parts, rng.randint(0, parts)))
    lines = [f"static_assert(gla::part_begin({j}, {n} / {parts}, {n} % {parts}, {parts}) == {j * n // parts});" for n, parts, j in cases]
    source = tmp_path / "parts.cu"
    source.write_text('#include "gla_tiles.cuh"\n' + "\n".join(lines))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    run = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", SRC, "-c", str(source), "-o", str(tmp_path / "parts.o")],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
    kernel = open(os.path.join(SRC, "gla_kernel.cuh")).read()
    assert "part_begin(j, P.len_, P.longer, P.per)" in kernel
