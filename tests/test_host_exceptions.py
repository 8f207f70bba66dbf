"""C++ exceptions of the launchers' native side arrive as Python exceptions.  Each case runs in a process of
its own: an exception that reached the interpreter's C frames would end it."""

import subprocess
import sys
import textwrap

import pytest

from helpers import GOLDEN

_PRELUDE = """
import torch
from rotorquant_vllm import _lib
from rotorquant_vllm import cuda as rq
def refused(call):
    try:
        call()
    except Exception as exc:
        print("refused", type(exc).__name__)
    else:
        raise SystemExit("accepted")
"""


def _run(body: str) -> subprocess.CompletedProcess:
    import os

    root = os.path.dirname(os.path.dirname(GOLDEN))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.join(root, "rotorquant-vllm_b200"), root]))
    return subprocess.run([sys.executable, "-c", _PRELUDE + textwrap.dedent(body)], capture_output=True, text=True,
                          env=env, timeout=300)


@pytest.mark.parametrize("body", [
    # a tensor without a version counter
    """
    with torch.inference_mode():
        r = torch.eye(128)
    refused(lambda: _lib.host().mark_valid(r))
    refused(lambda: rq.validate_rotation(r))
    """,
    # tensors without memory
    """
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        rows, norms, cents = (torch.empty(*s, dtype=t, device="cuda") for s, t in
                              (((2, 3, 64), torch.uint8), ((2, 3, 1), torch.float32), ((8,), torch.float32)))
        refused(lambda: rq.iso_decompress(rows, norms, cents, torch.bfloat16))
    """,
])
def test_exceptions_are_python_exceptions(body):
    done = _run(body)
    assert done.returncode == 0 and "refused" in done.stdout, (done.returncode, done.stdout, done.stderr[-2000:])


def test_a_rotation_that_outlives_the_modules_is_silent():
    """A validated matrix that dies at interpreter exit, after the native module was cleared."""
    done = _run("""
        import functools
        @functools.lru_cache(None)
        def layer():
            r = torch.eye(128)
            rq.validate_rotation(r)
            return {"rotation": r}
        layer()
    """)
    assert done.returncode == 0 and "_forget" not in done.stderr, done.stderr[-2000:]


def test_another_torch_wants_another_module(monkeypatch):
    """The native side is built against one torch: with another installed it is missing, and the build makes it."""
    import importlib.util
    import os

    import torch

    from rotorquant_vllm import _lib

    path = os.path.join(os.path.dirname(os.path.dirname(GOLDEN)), "rotorquant-vllm_b200", "csrc", "build.py")
    spec = importlib.util.spec_from_file_location("rq_build", path)
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert _lib.host_path() == build.host_library() and os.path.exists(_lib.host_path())
    monkeypatch.setattr(torch, "__version__", "0.1.0")
    monkeypatch.setattr(_lib, "_HOST", None)
    assert _lib.host_path() == build.host_library() and build._stale(build.host_library())
    with pytest.raises(RuntimeError, match="build it with"):
        _lib.host()


@pytest.mark.gpu
def test_no_memory_for_the_result():
    done = _run("""
        packed = torch.zeros(1 << 14, 32, 64, dtype=torch.uint8, device="cuda")
        norms = torch.zeros(1 << 14, 32, 1, device="cuda")
        cents = torch.arange(8.0, device="cuda")
        torch.cuda.set_per_process_memory_fraction(0.0)
        try:
            rq.iso_decompress(packed, norms, cents, torch.float32)
        except torch.cuda.OutOfMemoryError:
            print("refused")
    """)
    assert done.returncode == 0 and "refused" in done.stdout, (done.returncode, done.stdout, done.stderr[-2000:])
