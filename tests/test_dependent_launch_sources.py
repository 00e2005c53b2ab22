"""Kernels that may start while their predecessor still writes (they call
pdl_wait) read vectors by ordinary loads: through pointers that are not
__restrict__ and without __ldg, which require data that nothing writes while the
kernel lives.  Stated on the sources: no run can show that it holds."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem-rs_b200", "csrc")
FILES = ("vec_kernels.cuh", "pa_kernels.cuh", "chunk_scatter.cuh", "hex_kernels.cuh", "tet_kernels.cuh")
# data written before the first launch: rule tables, a chunk plan's lists, quadrature data, the handle's arguments
CONSTANT = re.compile(r"^(TF|TB|gr|ph|R\.\w+|L\.(cu_|lmap)\w*|A\.L\.lmap|C\.(L\.lmap|G|Sm|sk|sm)|A\.qd)\b")


def functions(text):
    """(signature, body) of every function at namespace level."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"(?:__global__|__device__)[^;{}]*\)\s*\{", text):
        depth, k = 0, m.end() - 1
        while True:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            if depth == 0:
                break
            k += 1
        yield m.group(0), text[m.end():k]


def reached():
    """Functions that wait, and the device functions they call."""
    found = {}
    for f in FILES:
        with open(os.path.join(CSRC, f)) as h:
            for sig, body in functions(h.read()):
                names = re.findall(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", sig))
                if names:
                    found.setdefault(names[0], []).append((f, sig, body))
    live = [n for n, v in found.items() if any("pdl_wait()" in b for _, _, b in v)]
    seen = set()
    while live:
        n = live.pop()
        if n in seen:
            continue
        seen.add(n)
        for _, _, body in found[n]:
            live += [c for c in re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", body) if c in found]
    return {n: found[n] for n in seen}


def test_the_known_kernels_are_seen():
    names = set(reached())
    assert {"k_pcg_update", "k_cheb_step", "fixup_kernel", "fixup_row_t", "fixup_acc", "chunk_load_x", "chunk_sums",
            "chunk_shared_kernel", "hex_apply_kernel", "tet_moment_kernel", "tet_point_kernel", "pa_apply_body"} <= names


@pytest.mark.parametrize("name", sorted(reached()))
def test_no_read_only_loads_of_vectors(name):
    for f, sig, body in reached()[name]:
        for p in re.findall(r"__restrict__\s*(\w+)", sig):
            assert CONSTANT.match(p), f"{f}: {name}: {p} is __restrict__"
        for a in re.findall(r"__ldg\(\s*([\w.]+)", body):
            assert CONSTANT.match(a), f"{f}: {name}: __ldg({a})"


@pytest.mark.parametrize("name", FILES + ("fg_common.cuh", "femgpu.cu"))
def test_no_kernel_releases_its_successor_early(name):
    """CTAs that wait beside a running kernel slow it, and take SMs unevenly: a
    dependent kernel starts when the CTAs ahead of it have exited."""
    with open(os.path.join(CSRC, name)) as h:
        assert "launch_dependents" not in re.sub(r"//[^\n]*", "", h.read())
