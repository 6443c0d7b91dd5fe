"""When the build makes the torch extension again."""
import importlib.metadata
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_torch_extension_follows_its_sources_and_its_torch(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("tt_build_under_test", os.path.join(ROOT, "pku-aiprogramming_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    made = []

    def run(cmd, verbose):
        made.append(cmd)
        (tmp_path / "_ttorch.so").write_bytes(b"")

    monkeypatch.setattr(build, "_run", run)
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(build, "OBJ", str(tmp_path))
    build.build_torch_binding()
    assert len(made) == 1
    build.build_torch_binding()
    assert len(made) == 1                                  # nothing changed
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "0.0.1")
    build.build_torch_binding()
    assert len(made) == 2                                  # another torch
    build.build_torch_binding()
    assert len(made) == 2
    os.utime(tmp_path / "_ttorch.so", (0, 0))              # older than its source
    build.build_torch_binding()
    assert len(made) == 3
