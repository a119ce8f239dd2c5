"""Registers of kernels whose speed rests on them, as the compiler reports them (-Xptxas -v): a kernel of one block a row that
asks for more keeps its own further blocks off an SM (many rows) or the next product's block (few rows), and one that spills
waits for its own loads twice.  No run's result shows that."""
import functools
import os
import re
import subprocess

import pytest

from odin_infer_b200.csrc import build

CSRC = os.path.dirname(os.path.abspath(build.__file__))


@functools.lru_cache(maxsize=None)
def resources(source):
    """kernel (mangled) -> (registers, bytes of spill stores) of a source."""
    nvcc = build._nvcc()
    if nvcc is None:
        pytest.skip("no nvcc here")
    flags = [f for f in build.NVCC_FLAGS if f != "-shared"]
    out = subprocess.run([nvcc, *flags, "-Xptxas", "-v", "-I", CSRC, "-c", "-o", os.devnull, os.path.join(CSRC, source)],
                         stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, check=True).stdout
    return {name: (int(registers), int(spilled)) for name, spilled, registers in re.findall(
        r"Compiling entry function '(\w+)'.*?(\d+) bytes spill stores.*?Used (\d+) registers", out, flags=re.S)}


LIMITS = [   # source, kernel (mangled), registers, bytes spilled
    # a block of 1,024 threads a token: 64 registers are all there are
    ("moe.cu", "moe_router_kernel", 64, 0),
    # prompts: five blocks of 256 threads an SM
    ("rowwise.cu", "row_update_kernel", 48, 4),
    ("rowwise.cu", "17activation_kernel", 40, 0),
    ("rowwise.cu", "sigmoid_gate_vec_kernel", 40, 0),
    ("latent.cu", "latent_prep_kernelI.*Lb0E", 40, 0),   # one part
    ("head_prep.cu", "head_prep_kernelI.*Lb0E", 40, 0),
    ("elementwise.cu", "add_rmsnorm_wide_kernel", 64, 0),
    # a decode step's rows, a block of 512 threads each: beside it the next product's block wants 14 k of the SM's 64 k registers
    ("streams.cu", r"mix_streams_fast_kernelILi\dELi\dELi1E", 80, 0),
]


@pytest.mark.parametrize("source,kernel,registers,spilled", LIMITS, ids=[limit[1] for limit in LIMITS])
def test_registers(source, kernel, registers, spilled):
    found = {name: r for name, r in resources(source).items() if re.search(kernel, name)}
    assert found
    for name, used in found.items():
        assert used[0] <= registers and used[1] <= spilled, (name, used)
