"""Leaf-height knobs without a GPU: 0 (the choice by the panel's height) is a value
like any other, the autotuner times it, and it is what an untuned batch gets."""
import pytest


@pytest.fixture(scope="module")
def lib():
    from candmc_gb300 import _abi, build
    build.build()
    return _abi.load()


@pytest.mark.parametrize("knob", [b"leaf_rows", b"pipe_leaf_rows"])
def test_default_height_can_be_set_back(lib, knob):
    try:
        for v in (32, 0, 256, 0):
            assert lib.candmc_set_tuning(knob, v) == 0
        for v in (-1, 1, 31, 257):
            assert lib.candmc_set_tuning(knob, v) == 1
    finally:
        lib.candmc_set_tuning(knob, 0)


def test_autotuner_knows_the_default(tmp_path, monkeypatch):
    from candmc_gb300 import autotune
    monkeypatch.setenv("CANDMC_TUNING_DB", str(tmp_path / "db.json"))
    assert autotune.lookup([1000], [32]) == {"nstreams": 16, "leaf_rows": 0}
    assert 0 in autotune.GRID["leaf_rows"]
