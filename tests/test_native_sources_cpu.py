"""A library of one family's kernels has every entry point that a plain GEMM may call."""
import inspect
import re

import pytest

from vllm_gcu_b200.csrc import build
from vllm_gcu_b200.models import get_model_class
from vllm_gcu_b200.ops import cuda as C


@pytest.mark.parametrize("arch", ["SapapelForCausalLM", "FizunexForCausalLM", "FepopelForCausalLM",
                                  "VadelixForCausalLM"])
def test_gemm_entry_points(arch):
    model = get_model_class(arch)
    calls = inspect.getsource(C._gemm_bf16)
    if "moe" in model.native_sources:
        calls += inspect.getsource(C.gemm_bf16_grouped)
    names = set(re.findall(r"\bb200_gemm_\w+", calls))
    assert names
    text = "".join((build.CSRC / f"{s}.cu").read_text() for s in model.native_sources)
    defined = set(re.findall(r"B200_API int (b200_\w+)\(", text))
    assert names <= defined, names - defined
