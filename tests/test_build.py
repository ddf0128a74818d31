"""build.py rebuilds the library when any file that goes into it is newer."""

import importlib.util

from conftest import PKG_DIR


def test_library_depends_on_every_source_and_header(monkeypatch):
    spec = importlib.util.spec_from_file_location("tvs_build", PKG_DIR / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    asked = {}
    monkeypatch.setattr(build, "_stale", lambda target, deps: asked.update({target: set(deps)}))
    build.build()
    assert asked[build.LIB] >= {p for p in build.CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".hpp")}
