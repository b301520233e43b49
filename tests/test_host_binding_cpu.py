"""Finding and building the short way into the library (host_binding.cpp), without a GPU."""
import os
import subprocess
import sysconfig
import warnings

import pytest
import torch

from litetopk_b200 import _lib, api, build


@pytest.mark.parametrize("library", ["none", "not a library"])
def test_wrong_arguments_are_named_without_the_library(monkeypatch, tmp_path, library):
    path = tmp_path / "liblitedsa_b200.so"
    if library != "none":
        path.write_bytes(b"text")
    monkeypatch.setattr(_lib, "LIB_PATH", path)
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_host", False)
    f, b, i, u = (torch.zeros((4, 64, 576), dtype=t) for t in (torch.float32, torch.bfloat16, torch.int32, torch.uint8))
    for call, error in ((lambda: api.sparse_prefill(f, u[0], i[0], 1.0), TypeError), (lambda: api.sparse_prefill(u, u[0], i[0], 1.0), ValueError),
                        (lambda: api.sparse_prefill(b, u[0], i[0], 1.0, job_tokens=2), ValueError),
                        (lambda: api.lite_topk(u, u[0], f[0], None, 1, 0), TypeError), (lambda: api.dsv4_c128a_bf16(f, None, b[0], 0, 1.0), TypeError),
                        (lambda: api.dsv4_masked_mla_bf16_out(f, b[0], i[0], i, i, i, i, 1.0, 64, b, f, None), TypeError)):
        with pytest.raises(error):
            call()
    with pytest.raises((ImportError, OSError)):
        _lib.lib()


def test_the_module_is_one_interpreters_and_one_torchs(monkeypatch, tmp_path, built_lib):
    """Another torch or interpreter: the module that is there is not loaded, which is said once, and build() makes another."""
    lib = tmp_path / _lib.LIB_PATH.name
    lib.write_bytes(b"")
    monkeypatch.setattr(build, "OUT_DIR", tmp_path)
    monkeypatch.setattr(build, "LIB", lib)
    monkeypatch.setattr(build, "is_stale", lambda: False)
    monkeypatch.setattr(_lib, "LIB_PATH", lib)
    made = []

    def compiler(cmd, **kwargs):
        made.append(cmd[cmd.index("-o") + 1])
        with open(made[-1], "wb") as f:
            f.write(b"no module")
        return subprocess.CompletedProcess(cmd, 0, "")
    monkeypatch.setattr(build.subprocess, "run", compiler)

    def found():
        monkeypatch.setattr(_lib, "_host", False)
        return [_lib.host(), _lib.host()]
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert found() == [None, None]                  # none was ever built
    paths = set()
    for change in (lambda: None, lambda: monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other"),
                   lambda: monkeypatch.setattr(sysconfig, "get_config_var", lambda name: ".cpython-399-other.so")):
        change()
        if paths:
            with pytest.warns(UserWarning, match="another Python or torch") as w:
                assert found() == [None, None]
            assert len(w) == 1
        build.build()
        build.build()
        paths.add(_lib.host_path())
        assert _lib.host_path().exists() and len(made) == len(paths)
    assert set(tmp_path.glob("litedsa_host*.so")) == paths and len(paths) == 3
    os.utime(lib, (lib.stat().st_mtime + 1000,) * 2)      # a newer library
    build.build()
    assert set(tmp_path.glob("litedsa_host*.so")) == {_lib.host_path()} and len(made) == 4
