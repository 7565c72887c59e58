"""Kernels launched as programmatic dependents read what the kernel before them writes after their wait
only.  A __restrict__ parameter would let a compiler read it ahead: none of theirs has one."""
import pathlib
import re

SRC = pathlib.Path(__file__).resolve().parents[1] / "typhon_gb300" / "csrc"


def test_no_restrict_parameters():
    text = (SRC / "kernels.cuh").read_text()
    names = set(re.findall(r"launch_pdl\((k_\w+)", text)) | {"k_rk_update"}  # the last by a pointer
    assert len(names) >= 12
    for name in sorted(names):
        heads = re.findall(r"__global__ void[^;{]*?\b" + name + r"\(([^{;]*?)\)\s*\{", text)
        assert heads, name
        for params in heads:
            assert "__restrict__" not in params, name
