"""The prepare kernels' register and shared-memory budgets, from ptxas, as
the occupancy they are designed for needs them (CPU: nvcc cross-compiles).

On an SM of 64K registers and 228 KB of shared memory (1 KB reserved per
CTA), eight 128-thread YUV CTAs need at most 64 registers and 28,160 bytes
each, and ten 128-thread table CTAs at most 48 registers; a kernel that
grows past these silently loses a CTA per SM (the YUV kernel once held the
8-bit table it does not use and ran seven). Curve CTAs run eight to an SM as
YUV ones do. A batch's kernels and the one-pair kernels (PrepareOneKernel) are
held to the same. Registers spilled past the limits below go unnoticed as
well: they cost the table prepare 6 % once."""

import os
import re
import shutil
import subprocess

import pytest

from vqm_b200 import build

SM_SHARED = 233472
CTA_RESERVED = 1024


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    """(group, half, threads) of every batch kernel and ("one", group, half,
    threads) of every one-pair kernel: registers, shared memory and spills."""
    tmp_path = tmp_path_factory.mktemp("ptxas")
    nvcc = build.NVCC if os.path.exists(build.NVCC) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("nvcc not found")
    src = os.path.join(build.ROOT, "vqm_b200", "csrc", "ss2_prepare.cu")
    inc = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    r = subprocess.run([nvcc, *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-Xptxas=-v",
                        "-I" + inc, "-c", src, "-o", str(tmp_path / "prepare.o")],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    kernels, name = {}, None
    for line in r.stderr.splitlines():
        m = re.search(r"Compiling entry function '\S*Prepare(One)?KernelILi(\d)ELb(\d)ELi(\d+)E",
                      line)
        if m:
            name = tuple(int(g) for g in m.groups()[1:])
            if m.group(1):
                name = ("one",) + name
            continue
        if name is None:
            continue
        m = re.search(r"(\d+) bytes spill stores", line)
        if m:
            kernels.setdefault(name, {})["spill"] = int(m.group(1))
        m = re.search(r"Used (\d+) registers.*?(\d+) bytes smem", line)
        if m:
            kernels.setdefault(name, {}).update(regs=int(m.group(1)), smem=int(m.group(2)))
            name = None
    return kernels


def test_prepare_kernels_fit_their_occupancy(kernels):
    k = kernels
    for half in (0, 1):
        yuv = k[(1, half, 128)]
        assert yuv["regs"] * 128 * 8 <= 65536 and yuv["spill"] == 0, yuv
        assert 8 * (yuv["smem"] + CTA_RESERVED) <= SM_SHARED, yuv
        table = k[(0, half, 128)]
        assert table["regs"] * 128 * 10 <= 65536, table
        assert 10 * (table["smem"] + CTA_RESERVED) <= SM_SHARED, table


@pytest.mark.parametrize("half", [0, 1])
def test_one_pair_and_curve_kernels_fit_their_occupancy(kernels, half):
    for form in ((), ("one",)):
        for group in (1, 3):
            k = kernels[form + (group, half, 128)]
            assert k["regs"] * 128 * 8 <= 65536, (form, group, k)
            assert 8 * (k["smem"] + CTA_RESERVED) <= SM_SHARED, (form, group, k)
        table = kernels[form + (0, half, 128)]
        assert table["regs"] * 128 * 10 <= 65536, (form, table)
        assert 10 * (table["smem"] + CTA_RESERVED) <= SM_SHARED, (form, table)


@pytest.mark.parametrize("half", [0, 1])
def test_spills_stay_within_their_limits(kernels, half):
    """Bytes of spill stores: the table kernels of a batch, those of one pair
    and the 128-thread YUV kernels."""
    for threads in (128, 256):
        assert kernels[(0, half, threads)]["spill"] <= 40
        assert kernels[("one", 0, half, threads)]["spill"] <= 96
    for form in ((), ("one",)):
        assert kernels[form + (1, half, 128)]["spill"] == 0
