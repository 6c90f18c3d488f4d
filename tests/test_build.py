"""When the build script takes its results as current."""

from bionemo_inference_runtime_b200.csrc import build


def test_host_path_is_built_again_for_another_pytorch(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path)
    monkeypatch.setattr(build, "_stale", lambda target, sources: False)
    assert build._host_stale()  # nothing says what it was made for
    (tmp_path / build.HOST_MADE_FOR).write_text(build._host_made_for())
    assert not build._host_stale()
    version = build.importlib.metadata.version
    monkeypatch.setattr(build.importlib.metadata, "version", lambda name: version(name) + ".post1")
    assert build._host_stale()
