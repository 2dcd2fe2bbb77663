"""Register allocation of the compiled kernels, from what ptxas reported when they were built."""
import re

import pytest


def _reports(stem):
    """{mangled kernel name: (bytes of spill stores, bytes of spill loads)} of one source file"""
    from lightly_trian_quant_b200 import build

    build.build()
    (path,) = (build.CSRC / "build").glob(f"{stem}.*.ptxas")
    kernel, out = None, {}
    for line in path.read_text().splitlines():
        if m := re.search(r"Compiling entry function '(\w+)'", line):
            kernel = m.group(1)
        elif m := re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line):
            out[kernel] = (int(m.group(1)), int(m.group(2)))
    return out


@pytest.mark.parametrize("stem,kernels", [("kf_gemm", 80), ("kf_gemm_pair", 40), ("kf_attn", 8)])
def test_kernels_do_not_spill(stem, kernels):
    """every instantiation of the GEMM and attention kernels keeps its values in registers: no form, format or output type is left out of the look."""
    reports = _reports(stem)
    assert len(reports) == kernels
    assert not {k: v for k, v in reports.items() if v != (0, 0)}
