"""The native call modules (i_b200/csrc/python) and the general route beside them: what the modules do not
handle has to reach the general route, which words the errors, and nothing torch throws may end the process."""
import importlib.machinery
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

from conftest import ROOT


def rand(shape, seed):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


FAKE = """
    import torch
    from torch._subclasses.fake_tensor import FakeTensorMode
    from i_b200 import ilang
    f = ilang.i("^ij~ij")
    two = ilang.i("^ij~ij") & ilang.i("-ij~ij")
    ilang._load_calls()
    assert ilang._cuda_call, "the native module is not in use"
    mode = FakeTensorMode()
    with mode:
        x = torch.empty(3, 4, 5, device="cuda")
        coo = torch.sparse_coo_tensor(torch.zeros(2, 3, dtype=torch.long, device="cuda"), torch.ones(3, device="cuda"), (4, 5))
"""

WRAPPERS = {
    "vmap": "with mode: torch.func.vmap(f.exec_torch)(x)",
    "vmap_into": "with mode: torch.func.vmap(lambda t: f.into(t, t))(x)",
    "vmap_output_list": "with mode: torch.func.vmap(lambda t: two.into([t, t], t))(x)",
    "grad": "with mode: torch.func.grad(lambda t: f.exec_torch(t).sum())(x[0])",
    "fake": "f.exec_torch(x[0])",
    "fake_into": "f.into(x[0], x[1])",
    "sparse": "f.exec_torch(coo)",
    "sparse_into": "f.into(coo, x[0])",
}


def test_tensors_without_memory_raise(ilang):
    # Wrappers, fake and sparse tensors: a Python exception from the general route, never an abort.  In a
    # child process with fake CUDA tensors, so that no GPU is needed and an abort is a return code.
    pytest.importorskip("torch")
    code = textwrap.dedent(FAKE)
    for name, call in WRAPPERS.items():
        code += "try:\n    %s\nexcept (RuntimeError, TypeError) as e:\n    print(%r, 'raised', flush=True)\n" % (call, name)
    run = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=600)
    raised = [line.split()[0] for line in run.stdout.splitlines() if line.endswith(" raised")]
    assert run.returncode == 0 and raised == list(WRAPPERS), run.stdout[-500:] + run.stderr[-2000:]


def test_modules_are_those_of_this_python_and_torch(ilang, monkeypatch, tmp_path):
    # A module of another torch is not found; a file that does not load leaves the ctypes route.
    from i_b200 import build
    torch = pytest.importorskip("torch")
    assert torch.__version__ in build.call_module("cuda", torch.__version__)
    assert os.path.exists(build.call_module("cuda", torch.__version__))
    assert ilang._load_call("cuda", "torch") and ilang._load_call("host", "numpy")
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.1")
        assert ilang._load_call("cuda", "torch") is False
    broken = tmp_path / "broken.so"
    broken.write_bytes(b"no library")
    monkeypatch.setattr(build, "call_module", lambda *given: str(broken))
    assert ilang._load_call("cuda", "torch") is False and ilang._load_call("host", "numpy") is False


def test_the_build_does_without_what_the_modules_need(monkeypatch, tmp_path):
    from i_b200 import build
    no_cuda = tmp_path / "torch"
    (no_cuda / "lib").mkdir(parents=True)
    spec = importlib.machinery.ModuleSpec("torch", None, is_package=True)
    spec.submodule_search_locations = [str(no_cuda)]
    with monkeypatch.context() as m:
        m.setattr(build.importlib.util, "find_spec", lambda name: spec)
        m.setattr(build.subprocess, "run", lambda cmd, **_: subprocess.CompletedProcess(cmd, "cuda_call" in " ".join(cmd), "", ""))
        build._build_call_modules(str(tmp_path))
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    build._build_call_modules(str(tmp_path))


@pytest.fixture
def torch():
    return pytest.importorskip("torch")


@pytest.mark.gpu
def test_both_routes_give_the_same(ilang, torch, monkeypatch):
    i = ilang.i
    f, two = i("ik*kj~ijk") >> i("+ijk~ij"), i("^ij~ij") & i("-ij~ij")
    a, b = rand((7, 9), 1), rand((9, 5), 2)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()

    def calls():
        out, host = torch.empty(7, 5, device="cuda"), np.empty((7, 5), np.float32)
        got = [f.exec_torch(da, db), f.into(out, da, db), f.into([out], da, db), *two.exec_torch(da),
               *two.into((torch.empty_like(da), torch.empty_like(da)), da)]
        return [x.cpu().numpy() for x in got] + [f.exec_numpy(a, b), f.into(host, a, b), *two.exec_numpy(a)]
    native = calls()
    monkeypatch.setattr(ilang, "_cuda_call", False)      # the general route from here on
    monkeypatch.setattr(ilang, "_host_call", False)
    for x, y in zip(native, calls(), strict=True):
        assert x.shape == y.shape and x.dtype == y.dtype and np.array_equal(x, y)


@pytest.mark.gpu
def test_what_the_native_route_refuses(ilang, torch):
    f = ilang.i("-ij~ij")
    x = torch.randn(6, 10, device="cuda")
    want = 0.0 - x.cpu().numpy()
    assert np.array_equal(f.exec_torch(x.t()).cpu().numpy(), want.T)                    # strides: copied
    assert np.array_equal(f.into(torch.empty(5, 6, device="cuda"), x[:, ::2].t()).cpu().numpy(), want[:, ::2].T)
    assert np.array_equal(f.into(np.empty((6, 10), np.float32), x), want)               # device to host
    assert np.array_equal(f.into(torch.empty(6, 10, device="cuda"), x.cpu().numpy()).cpu().numpy(), want)
    assert np.array_equal(f.exec_torch(torch.nn.Parameter(x)).cpu().numpy(), want)
    with pytest.raises(TypeError, match="float32"):
        f.exec_torch(x.double())
    with pytest.raises(TypeError, match="contiguous"):
        f.into(torch.empty(10, 6, device="cuda").t(), x)
    with pytest.raises(TypeError, match="float32"):
        f.into(torch.empty(6, 10, device="cuda", dtype=torch.float16), x)
    with pytest.raises(RuntimeError):
        f.exec_torch(x, x)
    for sparse in (x.to_sparse(), x.to_sparse_csr()):
        with pytest.raises(RuntimeError):
            f.exec_torch(sparse)
    with pytest.raises(RuntimeError):
        torch.func.vmap(f.exec_torch)(torch.randn(3, 6, 10, device="cuda"))
    with pytest.raises(torch.OutOfMemoryError):                                         # 1.4 TB of output
        ilang.i("i*j~ij").exec_torch(torch.zeros(600000, device="cuda"), torch.zeros(600000, device="cuda"))
    for given in (want.astype(">f4"), np.asfortranarray(want), want.astype(np.float64)):
        assert np.array_equal(f.exec_numpy(given), 0.0 - want)
    with pytest.raises(TypeError, match="float32"):
        f.into(np.empty((6, 10), np.float64), want)


@pytest.mark.gpu
def test_an_output_that_shares_memory_until_written(ilang, torch):
    # A lazy clone shares its source's memory; writing it as an output must not write the source.
    f = ilang.i("-ij~ij")
    x, source = torch.randn(6, 10, device="cuda"), torch.zeros(6, 10, device="cuda")
    for outputs in (torch._lazy_clone(source), [torch._lazy_clone(source)]):
        assert torch.equal(f.into(outputs, x), 0.0 - x) and not source.any()
    lazy = torch._lazy_clone(x)
    assert torch.equal(f.exec_torch(lazy), 0.0 - x)
