"""The later MOOD passes' cluster kernel gives one result whatever order its
warps run in between two barriers (cluster_order.cpp runs it on the CPU)."""
import os
import re
import shutil
import subprocess

import pytest

import pkg

CSRC = os.path.join(pkg.PKG_DIR, "csrc")
HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = "/usr/local/cuda/include"


def _item(src, start):
    """The definition that begins with `start`, to the end of its braces."""
    a = src.index(start)
    depth, b = 0, src.index("{", a)
    for b in range(b, len(src)):
        depth += {"{": 1, "}": -1}.get(src[b], 0)
        if depth == 0:
            break
    return src[a:b + 1] + (";" if not src[a:b].rstrip().endswith(")") and "(" not in src[a:src.index("{", a)] else "") + "\n"


def _generated():
    with open(os.path.join(CSRC, "kernels.cu")) as f:
        k = f.read()
    with open(os.path.join(CSRC, "mood_cluster.cuh")) as f:
        m = f.read()
    fn = "__device__ __forceinline__ "
    parts = [_item(k, s) for s in (
        "enum : int { DM_SHOCK", fn + "int iabs_c(", fn + "int rec_sel(", fn + "int2* rec_list(", fn + "double flicd_x_at(",
        fn + "double flicd_y_at(", "struct NewState", fn + "bool detect_decide(")]
    m = m.replace("#pragma once", "")
    m, n1 = re.subn(r'asm volatile\("barrier.*?"memory"\);', "emu_cluster_sync();", m, flags=re.S)
    m, n2 = re.subn(r'asm volatile\("mov\.u32.*?\)\);', "n = emu_cluster_nctaid();", m, flags=re.S)
    m, n3 = re.subn(r"__shared__ Mc m;", "Mc& m = emu_shared<Mc>();", m)
    assert n1 and n2 and n3 == 2 and "asm" not in m
    return "namespace hosono {\nnamespace kstrict {\n" + "".join(parts) + m + "}\n}\n"


# 1000: to the end of the MOOD loop; 4: stopped by the pass cap
@pytest.mark.parametrize("cap", [1000, 4])
def test_order_of_warps(cap, tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    (tmp_path / "cluster_order_gen.h").write_text(_generated())
    exe = str(tmp_path / "cluster_order")
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-I", str(tmp_path), "-I", CSRC,
                    "-I", os.path.join(pkg.ROOT, "include"), "-I", CUDA, os.path.join(HERE, "cluster_order.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, str(cap)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
