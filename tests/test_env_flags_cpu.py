"""Flags are read when they are asked for, under both prefixes, however they were set or removed."""
import os

from vllm_gcu_b200 import envs


def test_flags_follow_the_environment(monkeypatch):
    for name in ("VLLM_B200_ORACLE", "VLLM_GCU_ORACLE"):
        monkeypatch.delenv(name, raising=False)
    assert envs.ORACLE is None
    monkeypatch.setenv("VLLM_GCU_ORACLE", "norm")
    assert envs.ORACLE == ["norm"]
    monkeypatch.setenv("VLLM_B200_ORACLE", "all,gemm_bf16")       # the first prefix goes first
    assert envs.ORACLE == ["all", "gemm_bf16"]
    os.environ.pop("VLLM_B200_ORACLE")
    os.environ.update(VLLM_GCU_ORACLE="rope")
    assert envs.ORACLE == ["rope"]
    del os.environ["VLLM_GCU_ORACLE"]
    assert envs.ORACLE is None


def test_without_the_mapping_behind(monkeypatch):
    monkeypatch.setattr(envs, "_RAW", None)
    monkeypatch.setenv("VLLM_B200_ORACLE", "x")
    assert envs.ORACLE == ["x"]
    monkeypatch.delenv("VLLM_B200_ORACLE")
    assert envs.ORACLE is None
