"""Flags are read from the environment that is in place when they are asked for."""
import os

from vllm_gcu_b200 import envs


def test_an_environment_put_in_place_of_the_first(monkeypatch):
    for name in ("VLLM_B200_ORACLE", "VLLM_GCU_ORACLE"):
        monkeypatch.delenv(name, raising=False)
    monkeypatch.setattr(os, "environ", {"VLLM_B200_ORACLE": "norm"})
    assert envs.ORACLE == ["norm"]
    monkeypatch.setattr(os, "environ", {})
    assert envs.ORACLE is None
