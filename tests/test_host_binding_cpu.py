"""Finding and building the short way into the library (host_binding.cpp), without a GPU."""
import pytest
import torch

from litetopk_b200 import _lib, api


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
