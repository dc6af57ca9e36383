"""The native module that calls the launchers with tensors: what it takes gives the bits of the Python path, and what
it does not take is answered NotImplemented, so that the Python path decides as before."""
import re
from pathlib import Path

import pytest
import torch

from shadowspill_b200 import build

from shadowspill_b200.ops import _lib, attention, functional as F


CSRC = Path(build.KERNEL_DIR)


def test_the_launchers_are_declared_once():
    """One header gives the parameters to the sources that define the launchers and to the module that calls them; the
    ctypes table has the same."""
    kinds = {"int": _lib.c_int, "long long": _lib.c_ll, "float": _lib.c_f}
    text = re.sub(r"//.*", "", (CSRC / "launchers.h").read_text())
    found = {}
    for name, params in re.findall(r"\bint (ss_\w+)\(([^)]*)\);", text):
        found[name] = [_lib.c_p if "*" in p else kinds[" ".join(p.split()[:-1])] for p in params.split(",")]
    called = set(re.findall(r"\bss_[a-z]\w+(?=,)", (CSRC / "host_calls.cpp").read_text().split("namespace {")[1]))
    assert called and called <= set(found)
    for name, types in found.items():
        if name in _lib._SIGNATURES:
            assert _lib._SIGNATURES[name] == types, name
        defining = [f for f in CSRC.glob("*.cu") if re.search(rf"\bint {name}\([^;{{]*\{{", f.read_text())]
        assert len(defining) == 1 and '#include "launchers.h"' in defining[0].read_text(), name
    assert called <= set(_lib._SIGNATURES)
    assert not re.search(r"\bint ss_\w+\(", (CSRC / "host_calls.cpp").read_text())


def test_the_module_is_built_again_for_another_torch(monkeypatch, tmp_path):
    csrc = tmp_path / "csrc"
    csrc.mkdir()
    for name in ("host_calls.cpp", "launchers.h"):
        (csrc / name).write_text("")
    for name in ("libss_kernels.so", "_host_calls.so"):
        (tmp_path / name).write_text("")
    runs = []

    def run(cmd, verbose):
        runs.append(cmd)
        Path(cmd[cmd.index("-o") + 1]).write_text("")
    monkeypatch.setattr(build, "KERNEL_DIR", csrc)
    monkeypatch.setattr(build, "KERNEL_LIB", tmp_path / "libss_kernels.so")
    monkeypatch.setattr(build, "HOST_CALLS", tmp_path / "_host_calls.so")
    monkeypatch.setattr(build, "_run", run)
    if build._cuda_home() is None:
        pytest.skip("no CUDA headers here")
    import os
    build.build_host_calls()
    build.build_host_calls()
    assert len(runs) == 1                                  # a module of unknown origin is built once
    monkeypatch.setattr(torch, "__version__", "0.0")
    build.build_host_calls()
    assert len(runs) == 2
    later = (tmp_path / "_host_calls.so").stat().st_mtime + 10
    os.utime(csrc / "launchers.h", (later, later))
    build.build_host_calls()
    assert len(runs) == 3


def _operands(device, rows=72, dh=64):
    g = torch.Generator().manual_seed(rows)
    bf = lambda *s: (torch.randn(*s, generator=g) * 0.5).bfloat16().to(device)
    cu = torch.tensor([0, rows // 3, rows], dtype=torch.int32, device=device)
    pos = torch.arange(rows, dtype=torch.int32, device=device)
    return dict(x=bf(rows, 128), w=bf(192, 128), res=bf(rows, 192), w13=bf(256, 128), gu=bf(rows, 256), w2=bf(64, 128),
                dy=bf(rows, 64), scale=bf(128), rstd=torch.rand(rows, generator=g).to(device), q=bf(rows, 4, dh),
                k=bf(rows, 2, dh), v=bf(rows, 2, dh), lse=torch.zeros(4, rows, device=device), cu=cu, pos=pos)


def _calls(o):
    h = _lib.host()
    return [h.gemm(o["x"], o["w"], False, False, None, False, 1.0), h.linear_residual(o["x"], o["w"], o["res"], None),
            h.swiglu_linear(o["x"], o["w13"], None, None, True), h.swiglu_linear_dgrad(o["dy"], o["w2"], o["gu"]),
            h.rmsnorm_fwd(o["x"], o["scale"], 1e-5, False, None, None, None),
            h.rmsnorm_bwd(o["x"], o["scale"], o["x"], o["rstd"], None, False, None, False),
            h.rope(o["x"].clone(), o["pos"], 0, 2, 64, 64, 1e4, False),
            h.attention_fwd(o["q"], o["k"], o["v"], o["cu"], None, None, None),
            h.attention_bwd(o["q"], o["k"], o["v"], o["q"], o["lse"], o["q"], o["cu"], None, None, None, None)]


@pytest.mark.skipif(not _lib._HOST_PATH.exists(), reason="the extension is not built")
def test_cpu_tensors_and_other_objects_are_left_to_python():
    assert all(r is NotImplemented for r in _calls(_operands("cpu")))
    h = _lib.host()
    assert h.gemm(None, [1], False, False, None, False, 1.0) is NotImplemented
    with pytest.raises(TypeError):
        h.gemm(None)


def _functional(o, dw):
    dgrad = F.swiglu_linear_dgrad(o["dy"], o["w2"], o["gu"])
    out, lse = attention.forward(o["q"], o["k"], o["v"], o["cu"], 0)
    flat = [F.linear_fwd(o["x"], o["w"]), F.linear_residual(o["x"], o["w"], o["res"]), dgrad,
            *F.swiglu_linear(o["x"], o["w13"]), *F.rmsnorm_fwd(o["x"], o["scale"]),
            F.rmsnorm_bwd(o["x"], o["scale"], o["x"], o["rstd"], dw), dw,
            F.rope_(o["x"].clone(), o["pos"], col0=0, heads=2, dh=64), out, lse]
    return flat + list(attention.backward(o["q"], o["k"], o["v"], out, lse, o["q"], o["cu"], 0))


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 72, 257])
def test_the_bits_of_the_python_path(rows, monkeypatch):
    """The same launchers get the same arguments, so everything is equal. `dw` sums over blocks in no fixed order: a bound on its rounding instead, 32-bit
    sums of `rows` terms of at most 8."""
    o = _operands("cuda", rows)
    got = _functional(o, torch.zeros(128, device="cuda"))
    assert not any(r is NotImplemented for r in _calls(o))

    class Refuses:
        def __getattr__(self, name):
            return lambda *a: NotImplemented
    with monkeypatch.context() as m:
        m.setattr(_lib, "_host", Refuses())
        want = _functional(o, torch.zeros(128, device="cuda"))
    for i, (a, b) in enumerate(zip(got, want)):
        if a.dtype == torch.float32 and a.shape == (128,):
            assert float((a - b).abs().max()) <= rows * 8 * 2.0 ** -23 * 4
        else:
            assert torch.equal(a, b), i
    h = _lib.host()
    wide = torch.zeros(rows, 132, dtype=torch.bfloat16, device="cuda")
    odd = wide[:, :128].copy_(o["x"])                                   # a pitch of 264 bytes
    off = torch.zeros(rows * 128 + 4, dtype=torch.bfloat16, device="cuda")[4:].view(rows, 128).copy_(o["x"])
    for t in (odd, off):                                               # both were refused, and are, by the Python path
        assert h.gemm(t, o["w"], False, False, None, False, 1.0) is NotImplemented
        with pytest.raises((ValueError, RuntimeError)):
            F.linear_fwd(t, o["w"])
    view = o["q"].view(rows, 256)[:, :128]                             # a pitch of 512 bytes: taken as it is
    assert torch.equal(F.linear_fwd(view, o["w"]), F.linear_fwd(view.contiguous(), o["w"]))
    torch.cuda.synchronize()
    _lib.check_status()
