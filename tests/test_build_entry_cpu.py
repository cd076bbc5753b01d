"""build() with and without the reference's sources beside the repository: the
harness made from them is left out when the folder is missing or empty."""
import importlib
import types

import pytest


@pytest.mark.parametrize("sources, harness", [(None, False), ([], False), (["BPTree.cu"], True)])
def test_reference_harness_only_from_sources(tmp_path, monkeypatch, sources, harness):
    entry = importlib.import_module("__graft_entry__")
    src = tmp_path / "reference"
    if sources is not None:
        src.mkdir()
        for name in sources:
            (src / name).write_text("")
    made = []
    monkeypatch.setattr(entry, "REFERENCE_SRC", str(src))
    monkeypatch.setattr(entry, "_pkg_build_module",
                        lambda: types.SimpleNamespace(build=lambda verbose: None))
    monkeypatch.setattr(entry.subprocess, "run", lambda cmd, check: made.append(cmd))
    # only what is built matters here, not what is loaded after it
    monkeypatch.setattr(entry.importlib, "import_module",
                        lambda name: types.SimpleNamespace(lib=lambda: None))
    entry.build()
    assert ["all" in cmd for cmd in made] == [True, False][: len(made)]
    assert any("ref" in cmd for cmd in made) == harness
