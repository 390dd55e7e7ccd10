"""Calls through the C extension (csrc/py/fastcall.c) against the general path in Python: the same results over what it takes, and everything
else still answered by the general path, errors among it."""
import pathlib
import subprocess
import sysconfig

import pytest
import torch

from maco_b200 import _build, _native as N, ops
from maco_b200.ops import attention as A, elementwise as E


def test_builds_and_leaves_cpu_tensors_to_the_general_path():
    if _build.build_fastcall() is None:
        pytest.skip("no compiler or no Python header")
    quick = N.fastcall("elementwise")
    x = torch.ones(2, 8)
    assert quick(E.T_GELU, x, None, None, None, 0.0, 0.0) is None
    assert quick(E.T_ADD, [1.0], None, None, None, 0.0, 0.0) is None              # not a tensor
    with pytest.raises(TypeError):
        quick(E.T_GELU, x)
    q, k = torch.ones(1, 4, 128), torch.ones(1, 2, 16, 128)
    assert N.fastcall("attention")(q, k, k, None, 0.1) is None
    with pytest.raises(ValueError):
        ops.gelu(x)
    with pytest.raises(AttributeError):
        ops.add([1.0], x)


@pytest.fixture
def empty_build(monkeypatch, tmp_path):
    """The extension's build with folders of its own, nothing built yet."""
    if _build.build_fastcall() is None:
        pytest.skip("no compiler or no Python header")
    monkeypatch.setattr(_build, "LIB_DIR", tmp_path)
    return tmp_path


@pytest.mark.parametrize("cc", ["gcc -pthread", "env gcc", "", " "])
def test_compiler_with_arguments(empty_build, monkeypatch, cc):
    monkeypatch.setenv("CC", cc)
    path = _build.build_fastcall()
    assert path.parent == empty_build and path.exists()


@pytest.mark.parametrize("cc", ["false", "/nonexistent/cc", "gcc -no-such-option", "gcc 'unbalanced"])
def test_the_build_survives_without_it(empty_build, monkeypatch, cc):
    from types import SimpleNamespace
    done = empty_build / "done.o"
    done.touch()
    monkeypatch.setattr(_build, "_compile_one", lambda src, verbose: done)
    monkeypatch.setattr(_build, "subprocess", SimpleNamespace(run=lambda cmd, **kw: (
        SimpleNamespace(returncode=0) if cmd[1] == "-shared" else subprocess.run(cmd, **kw))))        # (the link)
    monkeypatch.setattr(_build, "_nvcc", lambda: "nvcc")
    monkeypatch.setenv("CC", cc)
    with pytest.warns(UserWarning, match="not built"):
        assert _build.build() == _build.LIB_PATH
    assert not list(empty_build.glob("maco_fastcall*"))


def _loaded_from():
    mod = N._load_fastcall(N.lib())
    return mod and pathlib.Path(mod.__file__)


def test_only_this_sources_and_interpreters_build_is_loaded(empty_build, monkeypatch):
    others = [empty_build / n for n in ("maco_fastcall.so", "maco_fastcall-0123456789ab.cpython-37m-x86_64-linux-gnu.so")]
    for o in others:
        o.write_bytes(b"another interpreter's")
    first = _loaded_from()
    assert first.parent == empty_build and first.name.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    assert others[1].exists()
    # an edited source is another file, built when it is asked for, and what it replaces goes
    edited = empty_build / "fastcall.c"
    edited.write_text(_build.FASTCALL_SRC.read_text().replace("elementwise: seven arguments", "elementwise: 7 arguments"))
    monkeypatch.setattr(_build, "FASTCALL_SRC", edited)
    second = _loaded_from()
    assert second != first and second.exists() and not first.exists() and b"elementwise: 7 arguments" in second.read_bytes()


def test_the_package_without_its_sources(empty_build, monkeypatch):
    built = _loaded_from()
    (empty_build / "maco_fastcall-0123456789ab.cpython-37m-x86_64-linux-gnu.so").write_bytes(b"another interpreter's")
    monkeypatch.setattr(_build, "FASTCALL_SRC", empty_build / "fastcall.c")
    assert _loaded_from() == built
    built.unlink()
    assert _loaded_from() is None


def test_nothing_is_built_where_that_is_switched_off(empty_build, monkeypatch):
    monkeypatch.setenv("MACO_NO_AUTOBUILD", "1")
    assert _loaded_from() is None and not list(empty_build.iterdir())
    monkeypatch.setattr(N, "_fastcall", None)
    assert N.fastcall("elementwise")(E.T_GELU, None, None, None, None, 0.0, 0.0) is None       # the general path
    monkeypatch.delenv("MACO_NO_AUTOBUILD")
    built = _loaded_from()
    monkeypatch.setenv("MACO_NO_AUTOBUILD", "1")
    assert _loaded_from() == built                           # what is there is loaded


def _general(monkeypatch, module):
    monkeypatch.setattr(module, "_quick", lambda *a: None)


def _taken(name, args, out=None):
    """The C call itself: it takes the call, and writes where it is told to."""
    if _build.build_fastcall() is None:
        pytest.skip("no compiler or no Python header")
    res = N.fastcall(name)(*args)
    assert type(res) is torch.Tensor and (out is None or res is out)
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1,), (4, 512), (3, 7, 33)])
def test_ordinary_calls_are_taken(monkeypatch, dtype, shape):
    x, y = (torch.randn(*shape, device="cuda").to(dtype) for _ in range(2))
    w, b = (torch.randn(shape[-1], device="cuda").to(dtype) for _ in range(2))
    calls = [(E.T_GELU, x, None, None, 0.0, 0.0, lambda: ops.gelu(x)), (E.T_SOFTMAX, x, None, None, 0.0, 0.0, lambda: ops.softmax(x)),
             (E.T_ADD, x, y, None, 0.0, 0.0, lambda: ops.add(x, y)), (E.T_AXPBY, x, y, None, 2, -1.5, lambda: ops.axpby(x, y, 2, -1.5)),
             (E.T_RMSNORM, x, w, None, 1e-6, 0.0, lambda: ops.rmsnorm(x, w)), (E.T_LAYERNORM, x, w, b, 1e-5, 0.0, lambda: ops.layernorm(x, w, b)),
             (E.T_GELU, torch.nn.Parameter(x, requires_grad=False), None, None, 0.0, 0.0, lambda: ops.gelu(x))]
    got = []
    for kind, a, in1, in2, f0, f1, _ in calls:
        out = torch.empty(shape, device="cuda", dtype=dtype)
        _taken("elementwise", (kind, a, in1, in2, out, f0, f1), out)
        got.append((out, _taken("elementwise", (kind, a, in1, in2, None, f0, f1))))
    _general(monkeypatch, E)
    for (out, new), call in zip(got, calls):
        want = call[-1]()
        assert torch.equal(out, want) and torch.equal(new, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "view", "one_head_view", "scale", "more_batch"])
def test_ordinary_attention_is_taken(monkeypatch, dtype, form):
    B, H, G, S = (3, 1, 4, 300) if form == "one_head_view" else (3, 2, 4, 300)
    q = torch.randn(B, H * G, 128, device="cuda").to(dtype)
    k, v = (torch.randn(B + (form == "more_batch"), H, S + 77 * (form != "plain"), 128, device="cuda").to(dtype)[:, :, :S] for _ in range(2))
    scale, out = (0.05 if form == "scale" else 128 ** -0.5), torch.empty_like(q)
    A._lib()
    _taken("attention", (q, k, v, out, scale), out)
    new = _taken("attention", (q, k, v, None, scale))
    _general(monkeypatch, A)
    want = ops.attention_decode(q, k, v, scale=scale)
    assert torch.equal(out, want) and torch.equal(new, want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1,), (5,), (4, 512), (3, 7, 33), (2, 0, 8), ()])
@pytest.mark.parametrize("form", ["plain", "out", "strided", "parameter"])
def test_elementwise_same_as_general(monkeypatch, dtype, shape, form):
    g = torch.Generator(device="cuda").manual_seed(1)
    mk = lambda: torch.randn(*shape, device="cuda", generator=g).to(dtype) if shape else torch.randn((), device="cuda", generator=g).to(dtype)
    x, y = mk(), mk()
    if form == "strided" and len(shape) > 1:
        x = torch.cat([x, x], -1)[..., :shape[-1]]
    if form == "parameter":
        x = torch.nn.Parameter(x, requires_grad=False)
    cols = shape[-1] if shape else 1
    w, b = torch.randn(cols, device="cuda", generator=g).to(dtype), torch.randn(cols, device="cuda", generator=g).to(dtype)

    def all_of():
        o = (lambda: torch.empty(shape, device="cuda", dtype=dtype)) if form == "out" else (lambda: None)
        calls = [lambda: ops.gelu(x, out=o()), lambda: ops.silu(x, out=o()), lambda: ops.softmax(x, out=o()), lambda: ops.scale(x, 3, out=o()),
                 lambda: ops.add(x, y, out=o()), lambda: ops.silu_gate(x, y, out=o()), lambda: ops.gelu_bwd(x, y, out=o()),
                 lambda: ops.axpby(x, y, 2.0, -1, out=o()), lambda: ops.rmsnorm(x, w, out=o()), lambda: ops.layernorm(x, w, b, out=o())]
        res = []
        for c in calls:
            try:
                res.append(c())
            except (IndexError, ValueError, RuntimeError) as e:
                res.append(type(e))
        return res

    got = all_of()
    _general(monkeypatch, E)
    for a, b_ in zip(got, all_of()):
        assert (a == b_) if isinstance(b_, type) else (a.shape == b_.shape and a.dtype == b_.dtype and torch.equal(a, b_))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["plain", "out", "view", "one_head_view", "scale", "more_batch", "strided_q"])
def test_attention_same_as_general(monkeypatch, dtype, form):
    g = torch.Generator(device="cuda").manual_seed(2)
    B, H, G, S = (3, 1, 4, 300) if form == "one_head_view" else (3, 2, 4, 300)
    q = torch.randn(B, H * G, 128, device="cuda", generator=g).to(dtype)
    k = torch.randn(B + (form == "more_batch"), H, S + 77, 128, device="cuda", generator=g).to(dtype)
    v = torch.randn_like(k)
    if form in ("view", "one_head_view", "more_batch"):
        k, v = k[:, :, :S], v[:, :, :S]
    if form == "strided_q":
        q = torch.cat([q, q], 1)[:, :H * G]
    kw = {"scale": 0.05} if form == "scale" else {}
    run = lambda: ops.attention_decode(q, k, v, out=torch.empty(B, H * G, 128, device="cuda", dtype=dtype) if form == "out" else None, **kw)
    got = run()
    _general(monkeypatch, A)
    assert torch.equal(got, run())


@pytest.mark.gpu
def test_refusals_stay():
    q = torch.randn(2, 8, 128, device="cuda").bfloat16()
    k = torch.randn(2, 2, 64, 128, device="cuda").bfloat16()
    for bad_k, bad_v in ((k, k[:, :, :32]), (k.transpose(1, 2), k.transpose(1, 2)), (k[:1], k[:1])):
        with pytest.raises(ValueError):
            ops.attention_decode(q, bad_k, bad_v)
    with pytest.raises(ValueError):
        ops.gelu(torch.randn(4, 8, device="cuda"), out=torch.empty(8, 4, device="cuda").t())
    with pytest.raises(ValueError):
        ops.gelu(torch.ones(4, 8, device="cuda", dtype=torch.int32))


@pytest.mark.gpu
def test_factors_that_only_float_takes():
    x = torch.randn(4, 8, device="cuda")
    assert torch.equal(ops.scale(x, "2.5"), ops.scale(x, 2.5))
    assert torch.equal(ops.softmax(ops.axpby(x, x, torch.tensor(2.0), "-1")), ops.softmax(ops.axpby(x, x, 2.0, -1.0)))
    for factor, error in (("two", ValueError), (None, TypeError), (torch.ones(2), (RuntimeError, ValueError))):
        with pytest.raises(error):
            ops.scale(x, factor)
    q, k = torch.randn(1, 4, 128, device="cuda").half(), torch.randn(1, 2, 16, 128, device="cuda").half()
    assert torch.equal(ops.attention_decode(q, k, k, scale="0.1"), ops.attention_decode(q, k, k, scale=0.1))
