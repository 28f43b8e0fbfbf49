"""The CPython form of the contiguous call (csrc/binding.cpp): what it does not take goes the general way, with that way's errors, and
what it takes gives the general way's results."""
import os
import subprocess
import sys
import types

import pytest
import torch

from conftest import ROOT

import nvfp4_gemm
from nvfp4_cutlass_b200 import _C
from nvfp4_cutlass_b200.csrc import build


def operands(device, m=128, n=256, k=256, e=2):
    g = torch.Generator().manual_seed(m + n + k)
    w = (torch.randn(e, n, k, generator=g) * 0.05).to(torch.bfloat16)
    b, sfb, gw = nvfp4_gemm.quantize_weight_nvfp4(w.to(device))
    sizes = [m] + [0] * (e - 1) if m < 256 else [m // 2] * e
    return dict(a=torch.randn(m, k, generator=g).to(torch.bfloat16).to(device), b=b, sfb=sfb, gw=gw,
                d=torch.zeros(m, n, dtype=torch.bfloat16, device=device), m_indices=nvfp4_gemm.make_m_indices(sizes, device=device, alignment=16))


WRONG = {
    "a": lambda t: t.float(), "b": lambda t: t.to(torch.uint8), "sfb": lambda t: t[:-1], "gw": lambda t: t.double(), "d": lambda t: t[:-1],
    "m_indices": lambda t: t.long(),
}


@pytest.mark.parametrize("name", WRONG)
def test_it_answers_none_to_what_does_not_fit(name):
    _C.lib()
    t = operands("cpu")
    t[name] = WRONG[name](t[name])
    assert _C._contiguous_call(*t.values(), 0, 1, 0, 0) is None
    with pytest.raises(RuntimeError, match="assertion failed"):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**t)


def test_it_answers_none_to_host_tensors_subclasses_and_odd_options():
    _C.lib()

    class Sub(torch.Tensor):
        pass

    t = list(operands("cpu").values())
    assert _C._contiguous_call(*t, 0, 1, 0, 0) is None
    assert _C._contiguous_call(t[0].as_subclass(Sub), *t[1:], 0, 1, 0, 0) is None
    assert _C._contiguous_call(*t, 0, 1, 0, -16) is None and _C._contiguous_call(*t, 0, 1, 0, "16") is None
    assert _C._contiguous_call(*t, 0, 1, 0, 1 << 80) is None and _C._contiguous_call(None, *t[1:], 0, 1, 0, 0) is None
    with pytest.raises(TypeError):
        _C._contiguous_call(*t)


FIRST_USE = """
import sys
from nvfp4_cutlass_b200 import _C
seen = 0
def step(frame, event, arg):
    global seen
    seen += event == "opcode"
    if _C._lib is not None:
        assert callable(_C._contiguous_call), "the library is there, the call is not"
    return step
def enter(frame, event, arg):
    if frame.f_code is _C.lib.__code__:
        frame.f_trace_opcodes = True
        return step
sys._getframe().f_trace_opcodes = True               # Python 3.12 has opcode events only if a frame asked for them before
sys.settrace(enter)
_C.lib()
sys.settrace(None)
assert seen > 100
assert _C._lib is not None and _C._contiguous_call(*range(10)) is None
"""


def test_a_thread_that_finds_the_library_loaded_can_call():
    """At no instruction of the first use is the library visible to another thread and the call that comes with it not."""
    r = subprocess.run([sys.executable, "-c", FIRST_USE], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("found", ["nothing", "something else"])
def test_without_the_binding_everything_goes_the_general_way(monkeypatch, tmp_path, found):
    path = tmp_path / "_binding.so"
    if found != "nothing":
        path.write_bytes(b"not a module")
    for name, value in (("_BINDING_PATH", str(path)), ("_lib", None), ("_contiguous_call", _C._no_binding)):
        monkeypatch.setattr(_C, name, value)
    with pytest.warns(RuntimeWarning, match="does not load"):
        assert _C.lib() is not None
    t = operands("cpu")
    assert _C._contiguous_call(*t.values(), 0, 1, 0, 0) is None
    with pytest.raises(RuntimeError, match="a is a CUDA tensor"):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**t)


@pytest.fixture
def compiled(monkeypatch):
    """Command lines that the build would run; nothing is run."""
    commands = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: commands.append(cmd) or types.SimpleNamespace(returncode=0, stdout="", stderr=""))
    return commands


def binding_commands(commands):
    return [cmd for cmd in commands if any(arg.endswith("binding.cpp") for arg in cmd)]


def test_another_torch_gets_a_module_of_its_own(compiled, monkeypatch, tmp_path):
    assert build.binding_path() == _C._BINDING_PATH and os.path.exists(_C._BINDING_PATH)
    monkeypatch.setattr(build, "OUT_DIR", str(tmp_path))
    with open(build.binding_path(), "w"):
        pass
    build.build()
    assert binding_commands(compiled) == []                              # this torch has its module
    monkeypatch.setattr(torch, "__version__", "99.0")
    build.build()
    (cmd,) = binding_commands(compiled)
    assert cmd[cmd.index("-o") + 1] == build.binding_path() and "torch99.0" in build.binding_path()
    assert f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}" in cmd


@pytest.mark.parametrize("torch_is", ["missing", "without CUDA", "there, its headers do not compile"])
def test_the_library_builds_without_the_binding(compiled, monkeypatch, tmp_path, capsys, torch_is):
    """The C ABI's consumers need the CUDA toolkit alone."""
    monkeypatch.setattr(build, "OUT_DIR", str(tmp_path))
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path))
    if torch_is == "missing":
        monkeypatch.setitem(sys.modules, "torch", None)
    elif torch_is == "without CUDA":
        monkeypatch.setattr(torch.version, "cuda", None)
    else:
        with open(build.binding_path(), "w"):                            # of an older header
            pass
        record = build.subprocess.run
        monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: types.SimpleNamespace(
            returncode=int(bool(binding_commands([cmd])) and record(cmd) is not None), stdout="", stderr="no such header"))
    build.build(force=True)
    assert "without binding.cpp's module" in capsys.readouterr().err
    assert len(binding_commands(compiled)) == (torch_is not in ("missing", "without CUDA")) and os.listdir(tmp_path) == []


def test_a_kernel_that_does_not_compile_fails_the_build(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path))
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: types.SimpleNamespace(returncode=1, stdout="", stderr="bad"))
    with pytest.raises(RuntimeError, match="failed on"):
        build.build()


class OnDevice:
    """A host tensor that says of itself that it is on CUDA device 0."""
    is_cuda = True

    def __init__(self, t):
        self._t = t

    def get_device(self):
        return 0

    def __getattr__(self, name):
        return getattr(self._t, name)


def test_a_tuned_call_that_fits_is_judged_by_one_expression(monkeypatch):
    """Calls with tune arguments do not go through the binding; their conditions are not taken one by one either, which took half
    as long again as the whole call."""
    t = {name: OnDevice(x) for name, x in operands("cpu").items()}
    one_by_one = []
    monkeypatch.setattr(_C, "_require", lambda cond, what: one_by_one.append((bool(cond), what)))
    assert _C._contiguous_device(**t, device_status=None) == 0 and one_by_one == []
    monkeypatch.setattr(_C, "_one_device", lambda *tensors: torch.device("cuda", 0))
    t["sfb"] = OnDevice(t["sfb"]._t[:-1])
    _C._contiguous_device(**t, device_status=None)
    assert [what for cond, what in one_by_one if not cond] == ["sfb.size(0) == num_groups * (k / 64)"]


@pytest.mark.gpu
@pytest.mark.parametrize("swap,align,m", [(0, 128, 256), (1, 16, 16), (1, 32, 96)])
@pytest.mark.parametrize("residual", [True, False])
def test_both_ways_give_the_same(swap, align, m, residual):
    t = operands("cuda", m=m)
    calls = []
    fast = _C._contiguous_call
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    wide = torch.full((m, 384), 7.0, dtype=torch.bfloat16, device="cuda")
    for kw in ({}, dict(device_status=status)):                 # a status word is not an ordinary call
        for d in (t["d"], wide[:, :256]):
            d.zero_()
            _C.lib()
            _C._contiguous_call = lambda *a: calls.append(fast(*a)) or calls[-1]
            try:
                nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**{**t, "d": d}, enable_residual_pass=residual, m_alignment=align,
                                                                     tune_swap_ab=swap, **kw)
            finally:
                _C._contiguous_call = fast
            calls.append(d.clone())
    assert calls[0] == 0 and calls[2] == 0 and len(calls) == 6          # the first two went through the binding, the others did not
    assert float(calls[1].float().norm()) > 0
    for other in (calls[3], calls[4], calls[5]):
        assert torch.equal(calls[1], other)
    assert bool((wide[:, 256:] == 7.0).all())


@pytest.mark.gpu
def test_errors_and_streams_are_those_of_the_general_way():
    t = operands("cuda", m=256)
    with pytest.raises(RuntimeError, match="m_alignment 128 or 256"):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**t, m_alignment=64)
    with pytest.raises(RuntimeError, match="multiples of 8 elements"):
        odd = torch.zeros(256, 257, dtype=torch.bfloat16, device="cuda")[:, :256]
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**{**t, "d": odd})
    with pytest.raises(RuntimeError, match="operand is a CUDA tensor|is a CUDA tensor"):
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**{**t, "gw": t["gw"].cpu()})
    want = t["d"].clone()
    nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**{**t, "d": want})
    torch.cuda.synchronize()
    side, got = torch.cuda.Stream(), torch.zeros_like(want)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):              # captured on the stream that is current
            nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(**{**t, "d": got})
    assert float(got.float().norm()) == 0
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
