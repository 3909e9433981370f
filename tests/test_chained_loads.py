"""Kernels launched with programmatic serialisation start while the kernel before them still writes, so
only data that no kernel of the chain writes may take the read-only path (csrc/bk_launch.cuh). The
sources of the chained kernels: the arguments of __ldg and the const __restrict__ parameters of
__global__ functions are those constants and nothing else."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "baking_b200" / "csrc"
FILES = ("bk_device.cuh", "bk_scatter.cuh", "bk_substep.cu", "bk_adjoint.cu", "bk_adjoint_transport.cu",
         "bk_measure.cu")
# per-particle constants, shared parameters, the batch's tables (written by host copies before any launch)
CONSTANTS = re.compile(r"cst\.\w+|eta_param\b|dry \+ i|mass \+ i|b\.owner\b|f \+ k\b|f \+ k \+ 1|src \+ w")
PARAMETERS = {("k_adj_g2p_return", "eta_param"), ("k_adj_p2g", "volume"), ("k_step_summary", "mass"),
              ("k_step_summary", "dry")}
PLAIN = {"k_surface_accumulate", "k_measure", "k_measure_finish"}  # launched without overlap


@pytest.mark.parametrize("name", FILES)
def test_read_only_loads_are_of_constants(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for argument in re.findall(r"__ldg\(([^()]*(?:\([^()]*\))?[^()]*)\)", text):
        assert CONSTANTS.fullmatch(argument.strip()) or CONSTANTS.match(argument.strip()), argument
    for kernel, parameters in re.findall(r"__global__[^{;]*?\b(k[b]?_\w+)\(([^{;]*?)\)\s*\{", text):
        if kernel in PLAIN:
            continue
        for parameter in re.findall(r"const \w+\*\s*__restrict__\s*(\w+)", parameters):
            assert (kernel, parameter) in PARAMETERS
