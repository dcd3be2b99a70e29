"""The build's list of sources is the sources there are: a lost one is reported
by the build, not by an undefined symbol when the library is loaded."""
import os

import pytest


def test_listed_sources_are_the_sources():
    from bgk3d_gpu_b200 import build as B
    have = {f for f in os.listdir(B.CSRC) if f.endswith(".cu")}
    assert len(B.LIB_SOURCES) == len(set(B.LIB_SOURCES))
    assert set(B.LIB_SOURCES) | {"dropin.cu"} == have


def test_a_missing_source_stops_the_build(monkeypatch):
    from bgk3d_gpu_b200 import build as B
    monkeypatch.setattr(B, "LIB_SOURCES", ["no_such_source.cu"])
    with pytest.raises(RuntimeError, match="no_such_source"):
        B.build()
