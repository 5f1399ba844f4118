"""Sources of the chained kernels (launch.cuh): a kernel that may start while the
one before still runs must not promise the compiler that a state, tendency or
pass buffer is its own.  __restrict__ stands on tables only."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "climatemachine.jl_gb300", "csrc")
# geometry, column factors, and an ensemble's launch parameters and tiles: no kernel writes them during a step
TABLES = {"geo", "ge", "F", "params", "tiles"}


def test_only_tables_are_restrict_qualified_in_chained_kernels():
    chained, found = [], {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        if not re.search(r"\b(launch_chained|chain_wait)\s*\(", code):
            continue
        chained.append(os.path.basename(path))
        names = set(re.findall(r"__restrict__\s+(\w+)", code))
        assert code.count("__restrict__") == len(re.findall(r"__restrict__\s+\w+", code))
        if names - TABLES:
            found[chained[-1]] = sorted(names - TABLES)
    assert {"stage.cu", "shell.cu", "arrays.cu", "viscous.cu", "viscous_common.cuh", "hyper.cu", "hyper_shell.cu",
            "hevi.cu"} <= set(chained)
    assert not found, found
