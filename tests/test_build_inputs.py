"""The build rebuilds when any file it compiles changes: its lists name every source and header
of csrc."""
import os

from axisymmetricjet_b200 import build


def test_every_source_and_header_is_a_dependency():
    files = os.listdir(build.CSRC)
    assert sorted(f for f in files if f.endswith(".cu")) == sorted(build.SOURCES)
    assert sorted(f for f in files if f.endswith(".cuh")) == sorted(build.HEADERS)
