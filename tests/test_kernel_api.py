"""The kernel library's C header (csrc/kernels/api.h) declares every exported launcher, so a
C or C++ host can call them without copying prototypes out of the sources."""
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_header_declares_every_exported_launcher():
    libs = glob.glob(os.path.join(ROOT, "vllm_cpp_b200", "_kernels*.so"))
    assert libs, "kernel library not built"
    out = subprocess.run(["nm", "-D", "--defined-only", libs[0]], capture_output=True, text=True).stdout
    exported = {l.split()[-1] for l in out.splitlines() if " T b200_" in l}
    header = open(os.path.join(ROOT, "csrc", "kernels", "api.h")).read()
    declared = set(re.findall(r"\b(b200_[a-z0-9_]+)\(", header))
    assert exported - declared == set(), f"not declared in api.h: {sorted(exported - declared)}"
    assert declared - exported == set(), f"declared but not exported: {sorted(declared - exported)}"


@pytest.mark.parametrize("cols", [64, 128, 256, 512])
def test_shared_memory_keeps_out_ctas_without_tensor_memory(cols):
    """Of a kernel whose CTAs meet in clusters no more may be resident on an SM than find their columns among its 512, whatever
    the registers let in; a launch that they bound already asks for no more than it needs."""
    from vllm_cpp_b200.ops import _lib
    if not _lib.available():
        pytest.skip("kernel library not built")
    bound, sm = _lib.lib().b200_tmem_bound_smem, 228 * 1024
    regs = _lib.lib().b200_ctas_by_registers                 # 352 threads: the third CTA comes in at 56 registers
    assert [regs(r, 352) for r in (32, 56, 57, 60, 64, 80, 88)] == [5, 3, 2, 2, 2, 2, 1] and regs(168, 192) == 2 and regs(255, 192) == 1
    for smem in (0, 45 * 1024, 70 * 1024, 81 * 1024, 120 * 1024):
        for fit in range(1, 11):
            got = bound(smem, fit, cols)
            if fit * cols <= 512:
                assert got == smem
            else:
                assert got >= smem and (512 // cols + 1) * got > sm
                assert got == smem or 512 // cols * (got + 2048) <= sm          # (with a CTA's static part: the others still fit)


def test_clusters_of_short_products_find_their_tensor_memory():
    """Of the products whose CTAs meet in clusters, those of one or two k-blocks ask for little shared memory: no more CTAs an SM than
    have columns, by shared memory alone."""
    from vllm_cpp_b200.ops import _lib
    if not _lib.available():
        pytest.skip("kernel library not built")
    L, sm = _lib.lib(), 228 * 1024
    for kblocks in range(1, 20):
        for bn in (128, 256):
            assert sm // L.b200_gemm_pair_smem(bn, kblocks) * 2 * bn <= 512
        for mp in range(16, 129, 16):
            cols = max(32, 1 << (mp - 1).bit_length())
            assert sm // L.b200_gemm_cluster_smem(mp, kblocks, 2) * cols <= 512


def test_successors_start_once_tensor_memory_is_taken():
    """A kernel lets its successor in when one thread of every CTA says so. Where the columns of tensor memory are still to be taken then, by
    another warp, the successor can take them first and wait for the kernel's end, which waits for the columns. So a barrier of
    the CTA lies between the two."""
    seen = 0
    for name in sorted(os.listdir(os.path.join(ROOT, "csrc", "kernels"))):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "csrc", "kernels", name)).read())
        for kernel in text.split("__global__")[1:]:
            taken = re.search(r"\btmem_alloc(_pair)?\(", kernel)
            let_in = re.search(r"\bpdl_launch_dependents\(", kernel)
            if taken and let_in:
                seen += 1
                assert "__syncthreads();" in kernel[taken.end():let_in.start()], (name, kernel[:100])
    assert seen >= 8
