"""The CPython form of the contiguous call (csrc/binding.cpp): what it does not take goes the general way, with that way's errors, and
what it takes gives the general way's results."""
import ctypes
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
    """Host tensors: none of them is an ordinary call's, and the general way names what does not fit.  The binding's own
    conditions are tried below, where the tensors could be taken."""
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


@pytest.fixture
def entry():
    """What the binding hands to the C entry, which is not called: nothing is launched, whatever the binding takes."""
    _C.lib()
    module, handed = _C._contiguous_call.__self__, []
    vp, i32, i64 = ctypes.c_void_p, ctypes.c_int, ctypes.c_int64
    fake = ctypes.CFUNCTYPE(i32, vp, i64, vp, vp, vp, vp, i64, vp, *[i32] * 8, vp, vp, vp)(lambda *args: handed.append(args) or 0)
    module.bind(ctypes.cast(fake, vp).value)
    yield handed
    module.bind(ctypes.cast(_C.lib().nvfp4_grouped_gemm_contiguous, vp).value)


def across(t):
    """The same values, the first dimension the contiguous one."""
    return t.t().contiguous().t()


class Subclass(torch.Tensor):
    pass


NOT_ORDINARY = {
    "a": [lambda t: t.float(), lambda t: t.half(), lambda t: t[None], lambda t: t[0], lambda t: t[:-1], lambda t: t[:, :-64].contiguous(), across],
    "b": [lambda t: t.to(torch.uint8), lambda t: t.int(), lambda t: t[None], lambda t: t.flatten(), lambda t: t[:-1], lambda t: t[:, :-1].contiguous(),
          lambda t: torch.cat((t, t)), across, lambda t: torch.cat((t, t), 1)[:, :t.shape[1]]],
    "sfb": [lambda t: t.long(), lambda t: t.float(), lambda t: t[None], lambda t: t.flatten(), lambda t: t[:-1], lambda t: t[:, :-1].contiguous(),
            lambda t: torch.cat((t, t)), across],
    "gw": [lambda t: t.double(), lambda t: t.bfloat16(), lambda t: t[:-1], lambda t: torch.cat((t, t)), lambda t: torch.stack((t, t), 1)[:, 0]],
    "d": [lambda t: t.float(), lambda t: t.half(), lambda t: t[None], lambda t: t[0], lambda t: t[:-1], lambda t: t[:, :-8], across],
    "m_indices": [lambda t: t.long(), lambda t: t.float(), lambda t: t[None], lambda t: t[:-1], lambda t: torch.cat((t, t)),
                  lambda t: t.repeat_interleave(2)[::2]],
}
NOT_PLAIN = [lambda t: t.cpu(), lambda t: t.to("meta"), lambda t: t.as_subclass(Subclass), lambda t: t.data_ptr(), lambda t: None]


@pytest.mark.gpu
@pytest.mark.parametrize("name", NOT_ORDINARY)
def test_it_takes_no_tensor_that_does_not_fit(entry, name):
    """Nothing behind the binding knows the sizes of the buffers: each of its conditions, by a call that fails that one."""
    t = operands("cuda", m=256)
    assert _C._contiguous_call(*t.values(), 0, 1, 0, 0) == 0 and len(entry) == 1
    for i, change in enumerate(NOT_ORDINARY[name] + NOT_PLAIN):
        assert _C._contiguous_call(*{**t, name: change(t[name])}.values(), 0, 1, 0, 0) is None, i
    if t[name].dim() == 2:
        assert _C._contiguous_call(*{**t, name: t[name].to_sparse()}.values(), 0, 1, 0, 0) is None
    batched = []
    torch.vmap(lambda x: batched.append(_C._contiguous_call(*{**t, name: x}.values(), 0, 1, 0, 0)) or x)(torch.stack((t[name], t[name])))
    assert batched == [None] and len(entry) == 1


@pytest.mark.gpu
def test_what_it_hands_on(entry):
    t = operands("cuda", m=256)
    pointers = {name: x.data_ptr() for name, x in t.items()}
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert _C._contiguous_call(*t.values(), 3, 0, 1, 16) == 0
    want = (pointers["a"], 256, pointers["b"], pointers["sfb"], pointers["gw"], pointers["d"], 256, pointers["m_indices"], 256, 256, 256, 2, 3, 0, 1, 16,
            None, None, side.cuda_stream)
    assert entry.pop() == want
    for option in range(4):
        for value in (-1, 1 << 31, 1 << 80, 1.0, "1", None):
            options = [0, 1, 0, 0]
            options[option] = value
            assert _C._contiguous_call(*t.values(), *options) is None
    wide = torch.zeros(256, 384, dtype=torch.bfloat16, device="cuda")
    for name, at in (("a", 0), ("d", 5)):                               # a parameter whose rows are further apart
        assert _C._contiguous_call(*{**t, name: torch.nn.Parameter(wide[:, 128:], requires_grad=False)}.values(), 0, 1, 0, 0) == 0
        assert entry.pop()[at:at + 2] == (wide.data_ptr() + 256, 384)
    # the stride of a single row is not one
    one = {**t, "a": t["a"].as_strided((1, 256), (8, 1)), "d": t["d"][:1], "m_indices": t["m_indices"][:1]}
    assert _C._contiguous_call(*one.values(), 0, 1, 0, 0) == 0 and entry.pop()[1] == 256


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
