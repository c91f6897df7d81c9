"""Kernels launched programmatically start while the kernel before them still
writes their inputs, so none of them reads memory through the read-only path
(ld.global.nc is for memory that nothing writes while the kernel runs)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "ppopp27-brdc-ae_b200", "csrc")


def _source():
    return {f: open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))}


def _programmatic():
    """Kernels that launch_pdl, or cudaLaunchKernelEx with pdl_attr's
    attribute, launches."""
    text = _source()["brdc_capi.cu"]
    names = set(re.findall(r"launch_pdl\(\s*(k_\w+)", text))
    names |= set(re.findall(r"cudaLaunchKernelEx\(&\w+,\s*(k_norm|k_level|k_plan|k_vec_gemm)\b", text))
    return sorted(names)


@pytest.mark.parametrize("kernel", _programmatic())
def test_no_read_only_loads(kernel):
    bodies = [m.group(0) for s in _source().values()
              for m in re.finditer(r"__global__[^{;]*?\b%s\(.*?\n}\n" % kernel, s, re.S)]
    assert len(bodies) == 1
    assert "__ldg(" not in bodies[0] and "__restrict__" not in bodies[0]
