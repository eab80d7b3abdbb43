"""Host-side geometry of the dense backward's kernels (csrc/dense_bwd_tiles.h), compiled for the CPU: what a kernel lays out has to
fit the memory that its launch gives it."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    gxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not gxx or not os.path.isfile(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("tiles")
    (d / "t.cpp").write_text('#include "dense_bwd_tiles.h"\nextern "C" {\n'
                             'size_t bitmap_bytes(int n) { return l1b::bwd_bitmap_bytes(n); }\n'
                             'size_t zero_mask_bytes(int n) { return l1b::bwd_zero_mask_bytes(n); }\n'
                             'int zeros_apart(int n) { return l1b::bwd_zeros_apart(n); }\n}\n')
    subprocess.run([gxx, "-shared", "-fPIC", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"), "-I", include,
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    lib = ctypes.CDLL(str(d / "t.so"))
    lib.bitmap_bytes.restype = lib.zero_mask_bytes.restype = ctypes.c_size_t
    return lib


def test_zero_masks_fit_the_bitmaps(tiles):
    """Two bytes per token in the memory of the bitmaps, which stop growing at 128 KiB; more tokens than that go without."""
    assert tiles.bitmap_bytes(1 << 23) == tiles.bitmap_bytes(4096) == 4 * (1 << 18) // 8
    for n in [1, 3, 33, 1000, 4096, 32768, 65533, 65535, 65536, 65537, 65540, 100000, (1 << 24) - 1]:
        assert tiles.zero_mask_bytes(n) >= 2 * n
        assert bool(tiles.zeros_apart(n)) == (n <= 65536)
        assert not tiles.zeros_apart(n) or tiles.zero_mask_bytes(n) <= tiles.bitmap_bytes(n)
    source = open(os.path.join(PKG, "csrc", "dense_ties.cu")).read()
    assert "z.apart" in source and "bwd_zeros_apart(n_tok)" in source  # the pass is entered by this rule


@pytest.mark.parametrize("name", ["coo.cu", "dense_ties.cu"])
def test_cluster_barrier_before_remote_shared_memory(name):
    """Shared memory of another CTA of the cluster may be accessed only behind a cluster barrier: before it that CTA need not run yet."""
    source = re.sub(r"//.*", "", open(os.path.join(PKG, "csrc", name)).read())
    bodies = [b for b in re.split(r"\n}\n", source) if "map_shared_rank" in b]
    assert bodies
    for body in bodies:
        assert "cluster.sync()" in body[:body.index("map_shared_rank")], body[:300]


def test_barriers_of_the_fused_kernels_are_unconditional():
    """A barrier of several warps stands only under conditions that no wait that ran out can make different for some of them (which warp
    it is, the tile's number): under any other -- a word of shared memory, say -- some warps could wait for others that never come."""
    source = re.sub(r"//.*", "", open(os.path.join(PKG, "csrc", "dense_softmax_v.cu")).read())
    uniform = [r"if \(warp < NW\)", r"for \(int m = 0; m < n[st]; m\+\+\)"]
    found = 0
    for kernel in re.findall(r"^softmax_v\w*_kernel\(.*?^}", source, re.S | re.M):
        stack, start, depth = [], 0, 0
        for i, c in enumerate(kernel):
            depth += (c == "(") - (c == ")")
            if c in "{;}" and depth == 0:
                head = kernel[start:i].strip()
                if re.match(r"(named_barrier|__syncthreads|if\s*\(.*\)\s*(named_barrier|__syncthreads))\b", head, re.S):
                    found += 1
                    assert re.match("named_barrier|__syncthreads", head), head  # not the statement of an `if` without braces
                    for h in stack[1:]:
                        assert any(re.fullmatch(u, h) for u in uniform), (h, head)
                if c == "{":
                    stack.append(head)
                elif c == "}":
                    stack.pop()
                start = i + 1
    assert found >= 10


def test_kernels_that_move_registers_are_asked_what_they_were_built_with():
    """setmaxnreg.inc waits without a limit when the block was launched with fewer registers than its warps ask for in all, and a
    launch has as many as the compiler gave the kernel: whoever launches such a kernel asks for them first."""
    for name in os.listdir(os.path.join(PKG, "csrc")):
        source = re.sub(r"//.*", "", open(os.path.join(PKG, "csrc", name), errors="replace").read()) if name.endswith((".cu", ".cuh")) else ""
        kernels = [re.search(r"(\w+_kernel)\(", b).group(1) for b in source.split("__global__")[1:] if "setmaxnreg.inc" in b]
        for kernel in kernels:
            launches = re.findall(r"auto kern = %s<.*?<<<" % kernel, source, re.S)
            assert launches and all("L1B_REGISTERS(kern, TC_REGS_LAUNCH)" in x for x in launches), (name, kernel)
        assert not kernels or "4 * TC_REGS + TC_REGS_REST <= 5 * TC_REGS_LAUNCH" in source
