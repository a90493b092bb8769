"""Registers of the FP64 kernels, from ptxas's own report (no GPU needed): the right-hand side by lines at five blocks of
128 threads per SM (102 registers), the integer sums at three of 256 (80), both without spilled registers.
"""
import re

import pytest

from test_kernel_resources import _ptxas_report


def _resources(report, fragment):
    out = []
    for part in report.split("Compiling entry function '")[1:]:
        if fragment in part.split("'")[0]:
            out.append((int(re.search(r"Used (\d+) registers", part).group(1)),
                        int(re.search(r"(\d+) bytes spill stores", part).group(1))))
    return out


@pytest.mark.parametrize("src,fragment,count,budget", [("nyles_line.cu", "k_line", 1, 102), ("nyles_mg.cu", "k_mg_fx", 3, 80)])
def test_fp64_register_budgets(src, fragment, count, budget, tmp_path):
    try:
        from nyles_gb300 import build
        build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    found = _resources(_ptxas_report(src, str(tmp_path)), fragment)
    assert len(found) == count, found
    for regs, spilled in found:
        assert regs <= budget and spilled == 0, found
