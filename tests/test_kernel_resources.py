"""Registers and shared memory of the element kernels, as ptxas reports them at
the build: they decide how many warps an SM holds, which bounds these kernels."""
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LOG = os.path.join(ROOT, "efem_b200", "_build", "residual.cu.o.ptxas")
SM_REGISTERS = 65536


@pytest.fixture(scope="module")
def kernels():
    """mangled name -> (registers, static shared memory) of residual.cu's kernels"""
    if not os.path.exists(LOG):
        pytest.skip("built without the ptxas report")
    with open(LOG) as f:
        text = f.read()
    found = re.findall(r"Compiling entry function '(\S+)'.*?Used (\d+) registers([^\n]*)", text, re.S)
    smem = [re.search(r"(\d+) bytes smem", rest) for _, _, rest in found]
    return {name: (int(regs), int(s.group(1)) if s else 0) for (name, regs, _), s in zip(found, smem)}


def element_kernels(kernels):
    """(nen, ngp, type, threads, law, faces) -> registers"""
    out = {}
    for name, (regs, _) in kernels.items():
        m = re.search(r"k_elem_residualILi(\d+)ELi(\d+)E([df])Li(\d+)ELi(n?\d+)ELb([01])E", name)
        if m:
            out[int(m[1]), int(m[2]), m[3], int(m[4]), int(m[5].replace("n", "-")), m[6] == "1"] = regs
    return out


def test_blocks_without_faces_do_not_pay_for_them(kernels):
    """The kernel without pressure faces has the element's registers alone: with
    128 threads and the neo-Hookean law at least six CTAs (24 warps) in FP64
    and nine (36) in FP32; with the faces' the FP64 ones hold five."""
    elem = element_kernels(kernels)
    assert len(elem) == 7 * 2 * 3 * 4 * 2  # element kinds, precisions, CTA sizes, laws, faces or not
    for (nen, ngp, t, threads, law, faces), regs in elem.items():
        if not faces and threads == 128 and law == 0:
            assert SM_REGISTERS // (128 * regs) >= (6 if t == "d" else 9), (nen, ngp, t, regs)


def test_register_summing_kernel_fits_eight_times(kernels):
    """k_elem_thread: 128 registers and the shared memory for eight CTAs of 64
    threads (16 warps) on an SM of 228 KB, 1 KB of which each CTA takes besides."""
    found = [v for k, v in kernels.items() if "k_elem_thread" in k]
    assert len(found) == 4
    for regs, smem in found:
        assert SM_REGISTERS // (64 * regs) >= 8 and 233472 // (smem + 1024) >= 8, (regs, smem)
