"""The C-ABI library loads and exports every symbol declared in include/clt_b200.h (no GPU needed)."""
import ctypes

from crosslayer_transcoder_b200 import _lib


def test_header_parses():
    protos = _lib.parse_header()
    assert "clt_encoder_fwd_act" in protos and "clt_adam_step" in protos
    assert len(protos) >= 18
    ret, args = protos["clt_adam_step"]
    assert ret is ctypes.c_int and len(args) == 14


def test_library_exports_every_declared_symbol():
    L = _lib.lib()                      # raises if a declared symbol is missing
    assert L.cdll.clt_version() >= 1
    for name in L.protos:
        assert hasattr(L.cdll, name)


def test_argument_errors_do_not_launch():
    L = _lib.lib()
    # bad dims are rejected before anything touches a device
    rc = L.cdll.clt_encoder_fwd_store(None, None, None, 0, 1, 1, 1, 0, None, None)
    assert rc != 0 and "bad dims" in L.last_error()


def test_fused_outputs_that_are_not_aligned_are_refused():
    """Epilogues store whole vectors of a row: an output that does not start on one is an argument error, not an access."""
    L, one = _lib.lib(), 1 << 20        # (addresses that nothing looks at)
    rc = L.cdll.clt_encoder_layer_fwd(one, 0, one, one, one, one + 4, 8, 64, 256, one, None)
    assert rc != 0 and "aligned" in L.last_error()
    rc = L.cdll.clt_select_topk_export(one, one, one, one, one, one + 16, 8, 2, 256, 4, 1, None)
    assert rc != 0 and "aligned" in L.last_error()


def _calls_in(path):
    """(entry point, number of arguments, line) of every ``_call("clt_...", ...)`` / ``lib().call("clt_...", ...)``
    in a Python source file, with the arguments counted at nesting depth 0."""
    import re

    text = path.read_text()
    out = []
    for m in re.finditer(r'(?:_call|\.call)\(\s*"(clt_\w+)"', text):
        i, depth, n, seen = m.end(), 0, 0, False
        while i < len(text):
            c = text[i]
            if c in "([{":
                depth += 1
            elif c in ")]}":
                if depth == 0:
                    break
                depth -= 1
            elif c == "," and depth == 0:
                n += 1
                seen = False
                i += 1
                continue
            elif c == "=" and depth == 0 and text[i + 1] != "=" and text[i - 1] not in "<>!=":
                n -= 1                      # a keyword argument of the wrapper (tag=...), not of the entry point
            if not c.isspace():
                seen = True
            i += 1
        import re as _re
        if _re.search(r",\s*\*\w", text[m.end():i]):
            continue                        # (arguments forwarded with *args cannot be counted)
        out.append((m.group(1), n if seen else n - 1, text.count("\n", 0, m.start()) + 1))
    return out


def test_host_code_calls_match_the_declared_abi():
    """Every kernel call in the host code names a declared entry point and passes as many arguments as the
    header declares (paths that only run on a GPU cannot drift from the ABI unnoticed)."""
    from pathlib import Path

    protos = _lib.parse_header()
    pkg = Path(_lib.__file__).resolve().parent
    files = [pkg / "engine.py", pkg / "data.py", pkg / "parallel.py", pkg / "model" / "clt_lightning.py"]
    n_calls = 0
    for f in files:
        for name, nargs, line in _calls_in(f):
            assert name in protos, f"{f.name}:{line}: {name} is not declared in the header"
            want = len(protos[name][1])
            assert nargs == want, f"{f.name}:{line}: {name} called with {nargs} arguments, the header declares {want}"
            n_calls += 1
    assert n_calls > 60


def test_bench_work_model_names_are_entry_points():
    """Every kernel the benchmark has a work model for is a declared entry point (a renamed or removed one would
    silently lose its roofline fraction)."""
    import importlib.util
    from pathlib import Path

    from crosslayer_transcoder_b200 import synthetic

    spec_ = importlib.util.spec_from_file_location("bench", Path(_lib.__file__).resolve().parents[1] / "bench.py")
    bench = importlib.util.module_from_spec(spec_)
    spec_.loader.exec_module(bench)
    protos = _lib.parse_header()
    for name, spec in synthetic.WORKLOADS.items():
        work = bench.algorithmic_work(bench.bench_spec(spec), 2, spec.d_features // 2, 10 ** 6, 2, nd_pad=256,
                                      fused_exchange=True)
        for k, v in work.items():
            assert k.split("[")[0] in protos, k
            assert v[0] in ("tensor", "hbm") and v[1] > 0, (name, k, v)


def test_native_call_path_converts_like_ctypes():
    """The compiled wrappers pass None, addresses, tensors, integers (masked like C) and floats as ctypes does, reject
    what they cannot convert before calling, and leave ctypes' own pointer objects to ctypes."""
    import pytest
    import torch

    from crosslayer_transcoder_b200 import build

    L = _lib.lib()
    if not L._native and None in build._binding_tools():
        pytest.skip("no Python headers or C compiler: calls go through ctypes")
    assert set(L._native) == {n for n, (r, a) in L.protos.items() if r is ctypes.c_int and a}
    name, types = "clt_adam_step", [t for _, t in L.protos["clt_adam_step"][1]]
    seen = []

    @ctypes.CFUNCTYPE(ctypes.c_int, *types)
    def probe(*args):
        seen.append(args)
        return 7

    t = torch.zeros(4)
    values = {ctypes.c_void_p: [t, None, 4096, torch.nn.Parameter(t)], ctypes.c_int: [3, -1, True, 2 ** 40 + 5],
              ctypes.c_int64: [2 ** 40, -2], ctypes.c_float: [0.1, 2]}
    args = [values[ty][i % len(values[ty])] for i, ty in enumerate(types)]
    mod = __import__("sys").modules[type(L).__module__]
    loaded = L._native[name].__self__
    try:
        assert loaded.bind(name, ctypes.cast(probe, ctypes.c_void_p).value)
        assert L._native[name](*args) == 7
        assert probe(*[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args]) == 7
        assert seen[0] == seen[1]
        for bad in (args[:-1], [object()] + args[1:], ["x"] * len(args)):
            with pytest.raises(TypeError):
                L._native[name](*bad)
        assert len(seen) == 2
    finally:
        loaded.bind(name, ctypes.cast(L._fn[name], ctypes.c_void_p).value)
    with pytest.raises(mod.CltError, match="bad dims"):
        L.call("clt_encoder_fwd_store", None, None, None, 0, 1, 1, 1, 0, None, None)
    dev = ctypes.c_void_p()
    with pytest.raises((mod.CltError, ctypes.ArgumentError)):
        L.call("clt_host_register", 0, 0, ctypes.byref(dev))


def test_call_path_that_cannot_load_leaves_ctypes(tmp_path, monkeypatch):
    """An extension of another Python has another name; one that does not load, or is some other module, is passed over."""
    import sysconfig

    import pytest

    # the suffix names this interpreter, so a tree that another one built has no such file
    assert _lib.BINDING_PATH.name == "_clt_call" + sysconfig.get_config_var("EXT_SUFFIX")
    for content in (b"", b"not an object file"):
        path = tmp_path / "_clt_call.so"
        path.write_bytes(content)
        monkeypatch.setattr(_lib, "BINDING_PATH", path)
        L = _lib._Lib()
        assert L._native == {}
        with pytest.raises(_lib.CltError, match="bad dims"):
            L.call("clt_encoder_fwd_store", None, None, None, 0, 1, 1, 1, 0, None, None)
    monkeypatch.setattr(_lib, "BINDING_PATH", tmp_path / "absent.so")
    assert _lib._Lib()._native == {}


def test_call_path_of_another_source_is_passed_over(tmp_path, monkeypatch):
    """A compiled call path is used only if it was made from today's conversions, not just from today's prototypes."""
    import shutil

    import pytest

    from crosslayer_transcoder_b200 import build

    if not _lib._Lib()._native:
        pytest.skip("no Python headers or C compiler: calls go through ctypes")
    path = tmp_path / _lib.BINDING_PATH.name
    shutil.copy(_lib.BINDING_PATH, path)        # a copy: a module that was loaded from a file is loaded once
    monkeypatch.setattr(_lib, "BINDING_PATH", path)
    assert _lib._Lib()._native
    monkeypatch.setattr(build, "_C_PRELUDE", build._C_PRELUDE + "/* converts otherwise */")
    assert _lib._Lib()._native == {}


def test_decoder_splits_where_that_was_measured_to_be_faster():
    """The rule for the parts of the decoder's contraction axis, at sizes that lost 19 to 50 % as parts and at sizes that
    gained (both forms timed on 148 SMs)."""
    parts = lambda L, B, D, F, cross, bf16, sms=148: _lib.lib().query("clt_decoder_dense_parts", B, L, D, F, cross, bf16, sms)
    for size in [(3, 1137, 952, 720, 1, 1), (8, 528, 512, 2208, 0, 1), (8, 346, 792, 2160, 0, 1), (3, 466, 1744, 3760, 0, 1),
                 (8, 134, 1480, 3296, 0, 1), (12, 1056, 248, 264, 1, 1), (12, 811, 144, 5080, 0, 1),
                 (4, 512, 1024, 640, 1, 1), (8, 43, 2296, 9456, 0, 0), (8, 5, 1992, 30664, 0, 0), (12, 36, 1232, 2584, 0, 0)]:
        assert parts(*size) == 0, size
    for size in [(1, 257, 768, 10000, 0, 1), (1, 257, 768, 120000, 0, 1), (1, 5, 64, 4096, 0, 1), (12, 300, 768, 10000, 1, 1),
                 (8, 342, 216, 720, 1, 1), (12, 512, 768, 1024, 1, 0), (1, 27, 216, 119168, 0, 0), (6, 781, 368, 1304, 0, 0),
                 (8, 119, 1584, 5616, 0, 0)]:
        n = parts(*size)
        assert 1 < n <= 2 * 296 + size[0], size
        assert parts(*size, 160) > 1                            # another chip's count is another plan, not a refusal
    # whole chains where the tiles fill the chip, are no longer than a few blocks, or where there is nothing to do
    for size in [(12, 4000, 768, 10000, 1, 1), (12, 333, 768, 24576, 0, 1), (2, 64, 64, 256, 1, 1), (1, 0, 64, 4096, 0, 1)]:
        assert parts(*size) == 0, size
