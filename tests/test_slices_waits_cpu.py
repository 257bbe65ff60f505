"""Whole warps wait as one in the pair GEMM with K split over a cluster, as in the kernels beside it."""
import importlib.util
import pathlib

from vllm_gcu_b200.csrc import build


def test_whole_warps_wait_as_one():
    spec = importlib.util.spec_from_file_location(
        "kernel_waits", pathlib.Path(__file__).with_name("test_kernel_waits_cpu.py"))
    other = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(other)
    text = (build.CSRC / "gemm_pair_slices.cu").read_text()
    waits = other._waits(text)
    assert waits and "mbar_wait_warp(" in text
    assert not [line for line, blocks in waits if not any("elect_one()" in b for b in blocks)]
