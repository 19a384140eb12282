"""What the build looks at before it keeps a module that is there."""
import torch


def test_the_cpp_module_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    from torch_ggml_ops_b200 import _build

    runs = []
    monkeypatch.setattr(_build, "_run", runs.append)
    monkeypatch.setattr(_build, "BUILD", tmp_path)
    monkeypatch.setattr(_build, "_newer", lambda out, deps: True)   # as far as the sources go, it is up to date
    _build.build_ext()
    _build.build_ext()
    assert len(runs) == 1
    monkeypatch.setattr(torch, "__version__", "99.0")
    _build.build_ext()
    _build.build_ext()
    assert len(runs) == 2
    _build.build_ext(force=True)
    assert len(runs) == 3
