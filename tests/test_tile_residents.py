"""The CTAs per SM that the tile rule of the box applies counts with, for every
kind, order, precision, format and lane shape, against the registers that the
build reports for each kernel and the shared memory of its plan."""
import os
import re
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fem-rs_b200")
LOG = os.path.join(PKG, "lib", "ptxas.log")


def up(a, b):
    return -(-a // b) * b


def table():
    with open(os.path.join(PKG, "csrc", "femgpu.cu")) as h:
        text = h.read()
    body = text[text.index("static void choose_tile("):]
    m = re.search(r"resident((?:\[\d\])+) = (\{.*?\});", body, re.S)
    dims = [int(d) for d in re.findall(r"\[(\d)\]", m[1])]
    assert dims == [2, 2, 2, 3, 3], "one entry per lane shape, precision, format, kind and order"
    v = [int(x) for x in re.findall(r"\d+", m[2])]
    assert len(v) == 72
    return lambda lanes8, fp32, affine, kind, p: v[(((lanes8 * 2 + fp32) * 2 + affine) * 3 + kind - 1) * 3 + p - 1]


def kernels():
    """{(order, kind, fp32, affine, lanes): (registers, warps, ring stages)}"""
    with open(LOG) as h:
        log = subprocess.run(["c++filt"], input=h.read(), capture_output=True, text=True, check=True).stdout
    out = {}
    for m in re.finditer(r"pa_apply_kernel<([^>]*)>.*?Used (\d+) registers", log, re.S):
        p, kind, t, wy, st, _, fmt, lx = [a.replace("(int)", "").strip() for a in m[1].split(",")]
        out[int(p), int(kind), int(t == "float"), int(fmt), int(lx)] = (int(m[2]), int(wy), int(st))
    return out


@pytest.mark.skipif(not os.path.exists(LOG), reason="no build log")
def test_residents_match_the_build():
    resident, found = table(), kernels()
    assert len(found) == 72
    for (p, kind, fp32, affine, lx), (regs, wy, st) in found.items():
        size, d = (4 if fp32 else 8), p + 1
        nc = {1: 1, 2: 6, 3: 7}[kind]
        stage = (6 * (kind != 1) + d ** 3 * (2 if kind == 3 else 1)) * 32 if affine else d * nc * 32
        tiles = 1 if p == 3 and not fp32 else 2
        x = up(d * (wy * (32 // lx) * p + 1) * up(lx * p + 1, 16 // size) * size, 128)
        smem = up(tiles * x + wy * st * stage * size + wy * d * d * lx * size + d * d * wy * 32 * size, 8) + (2 + wy * st) * 8
        by_regs = 65536 // (up(regs * 32, 256) * wy)
        by_smem = (228 * 1024) // (up(smem, 128) + 1024)  # 1 KB of each CTA is the system's
        assert resident(lx == 8, fp32, affine, kind, p) == min(by_regs, by_smem), (p, kind, fp32, affine, lx, regs, smem)
