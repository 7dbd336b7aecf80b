"""Kernels that may be placed while their predecessor in the stream still runs (programmatic dependents) read its output through
ordinary loads.  `const T* __restrict__` and __ldg promise the compiler data that nobody writes while the kernel lives: such a load may
take the non-coherent path and may be moved above griddepcontrol.wait.  The promise holds for weights and tables alone."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llama_rust_b200", "csrc")
LASTING = {"w", "table", "pos_table", "maps", "bias", "q_norm", "k_norm", "entries", "phases", "peers"}  # written before any launch of the stream
WAITS = ("pdl_enter()", "griddepcontrol.wait", "stream_body<", "gemm_tc_tile<")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^{;]*)\)\s*\{")


def _body(text, at):
    depth, i = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at:i]


def _kernels():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in KERNEL.finditer(text):
            body = _body(text, m.end())
            if any(w in body for w in WAITS) and m.group(1) != "gemm_tc_grouped_kernel":  # launched in stream order
                out[m.group(1)] = (m.group(2), body)
    return out


def test_the_sources_are_read():
    found = _kernels()
    assert len(found) > 40 and {"gemm_tc_kernel", "to_f16_rows_kernel", "digit_records_kernel", "add_units_kernel", "rmsnorm_kernel"} <= set(found)


@pytest.mark.parametrize("name", sorted(_kernels()))
def test_dependents_read_through_ordinary_loads(name):
    params, _ = _kernels()[name]
    promised = set(re.findall(r"const\s+\w+\*\s*__restrict__\s+(\w+)", params))
    assert promised <= LASTING, (name, promised - LASTING)


def test_non_coherent_loads_are_of_weights_and_tables():
    """__ldg in the files of dependents: the norm weights of the stream kernel's element-wise step, the attention's distance table."""
    seen = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        if any(w in text for w in WAITS):
            seen[os.path.basename(path)] = re.findall(r"__ldg\(\s*(.{0,40})", text)
    assert {f for f, calls in seen.items() if calls} <= {"llr_mma_common.cuh", "llr_mixers.cu", "llr_moe.cu"}, seen
    assert all("src.x2" in c for c in seen.get("llr_mma_common.cuh", []))
    assert all(c.startswith(("b0 +", "b1 +")) for c in seen["llr_mixers.cu"])
