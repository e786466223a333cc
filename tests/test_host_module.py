"""CPU: the torch-facing module of the hot entry points -- it loads beside the library, refuses (returns None) whatever is
not a plain CUDA tensor so that the general path runs, and gets the same format bytes as the structure."""
import pytest

torch = pytest.importorskip("torch")


def _quantizers():
    import hbq_b200 as H

    class Sub(H.HBQQuantizer):
        def _format(self):
            f = super()._format()
            f.block_size = 64
            return f

    return [H.HBQQuantizer(128, 2, 1, 5, 3, l2_block_size=32, l2_sc_bit=2, l2_scheme="Mix", use_ceil=True), H.HBQQuantizer(),
            H.MXFPQuantizer(16, 2, 1, 5, 3, per_tensor_scale=True, scale_allow_subnormal=True), H.MXFPQuantizer(32, 4, 3, 8, 0, use_round=True),
            H.MXINTQuantizer(8, 5, 0, 32), H.MXExQuantizer(), H.VSQQuantizer(4), Sub(128, 2, 2, 5, 3, l2_block_size=8)]


def test_format_bytes_follow_the_fields():
    for q in _quantizers():
        assert q._fmt_bytes() == bytes(q._format())
        if hasattr(q, "sc_mbit"):
            q.block_size = 256
            q.sc_mbit = 2
            assert q._fmt_bytes() == bytes(q._format())


def test_module_refuses_what_is_not_a_plain_cuda_tensor():
    from hbq_b200 import _lib
    from hbq_b200.build import build_library
    build_library()
    m = _lib.host()
    fmt = _quantizers()[0]._fmt_bytes()
    x = torch.zeros((2, 128), dtype=torch.float16)
    for t in (x, None, 3, x.float(), x.t()):
        assert m.quantize(t, fmt, -1) is None
        assert m.gemm(t, x, 0, 0, 0, None, True) is None
        assert m.gemm_w4(t, x, 128, 128, fmt, 4, None, x) is None
    with pytest.raises(TypeError):
        m.quantize(x, b"short", -1)
    with pytest.raises(TypeError):
        m.quantize(x, fmt)


def test_module_is_rebuilt_for_another_torch_or_python(monkeypatch, tmp_path):
    from hbq_b200 import _lib, build
    build.build_library()
    assert build.host_matches() and not build.host_is_stale()
    other = str(tmp_path / "hbq_host.so")
    tag = build.host_tag().encode()
    assert tag.count(torch.__version__.encode()) == 1
    with open(build.HOST_PATH, "rb") as f, open(other, "wb") as g:
        g.write(f.read().replace(tag, tag.replace(torch.__version__.encode(), b"0" * len(torch.__version__))))
    assert not build.host_matches(other)
    monkeypatch.setattr(build, "HOST_PATH", other)
    assert build.host_is_stale()
    monkeypatch.setattr(_lib, "HOST_PATH", other)
    monkeypatch.setattr(_lib, "_host", None)
    with pytest.raises(_lib.HbqError):
        _lib.host()
    monkeypatch.setattr(build, "is_stale", lambda: False)                # the module alone
    build.build_library()
    assert build.host_matches(other) and not build.host_is_stale()
    assert [p.name for p in tmp_path.iterdir()] == ["hbq_host.so"]


def test_torch_without_cuda_builds_the_library_alone(monkeypatch, tmp_path):
    import hbq_b200 as H
    from hbq_b200 import _lib, build
    build.build_library()
    built = []
    monkeypatch.setattr(torch.version, "cuda", None)
    monkeypatch.setattr(build, "HOST_PATH", str(tmp_path / "hbq_host.so"))
    monkeypatch.setattr(build, "_build_cuda", lambda verbose: built.append(1))
    monkeypatch.setattr(_lib, "_host", None)
    assert build.build_library(force=True) == build.LIB_PATH and built == [1] and not list(tmp_path.iterdir())
    x = torch.zeros((2, 128), dtype=torch.float16)
    with pytest.raises(_lib.HbqError):
        H.HBQQuantizer(128, 2, 2, 5, 3, l2_block_size=8).q(x)            # a CPU tensor, as with any torch
