"""Register counts of the built kernels, from the compiler's own report beside the library (CPU only): those whose launch
shapes were chosen for a number of resident blocks keep to it."""

import os
import re
import subprocess

import pytest

from conftest import ROOT

PKG = os.path.join(ROOT, "cpp-spo-dvr_b200")


@pytest.fixture(scope="module")
def kernels():
    """Mangled name -> (registers, bytes of spill stores)."""
    log = os.path.join(PKG, "lib", "ptxas.log")
    if not os.path.exists(log):
        subprocess.run(["make", "-C", PKG, "-j4"], check=True, stdout=subprocess.DEVNULL)
    out, name, spill = {}, None, 0
    for line in open(log):
        if m := re.search(r"Compiling entry function '(\S+)'", line):
            name = m.group(1)
        elif m := re.search(r"(\d+) bytes spill stores", line):
            spill = int(m.group(1))
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            out[name] = (int(m.group(1)), spill)
    return out


@pytest.mark.parametrize("kernel", ["axis_pass_kernel", "xy_pass_kernel"])
def test_general_kernels_leave_room_for_two_blocks_of_256_threads(kernels, kernel):
    forms = {n: r for n, r in kernels.items() if f"{len(kernel)}{kernel}I" in n}
    assert len(forms) == 2, forms  # float and double
    assert all(r <= 65536 // (2 * 256) for r, _ in forms.values()), forms


@pytest.mark.parametrize("kernel,most", [("xy2_kernelIfLi8ELi8ELi32E", 40),
                                         ("xy2p_kernelIfLi12ELi12ELi16E", 80), ("xy2p_kernelIdLi12ELi12ELi8E", 128)])
def test_xy_kernels_keep_their_resident_blocks(kernels, kernel, most):
    """256, 192 and 96 threads: 6, 4 and 5 blocks per SM."""
    (registers, _), = [r for n, r in kernels.items() if kernel in n]
    assert registers <= most, registers


def test_block_density_kernel_leaves_room_for_eight_blocks(kernels):
    forms = {n: r for n, r in kernels.items() if "20block_density_kernelI" in n}
    assert forms and all(r <= 32 and spill == 0 for r, spill in forms.values()), forms
