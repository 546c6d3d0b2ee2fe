"""The native call path without a GPU: what it makes of inputs it cannot serve."""

from __future__ import annotations

import copy
import gc
import os
import subprocess
import sys
import weakref

import pytest

from conftest import ROOT

_SCRIPT = r'''
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.symbolic_shapes import ShapeEnv
from xqt_b200 import native

bound = native.host().Bound(((2, 2, (), (), 0, 0),), lambda *args: "slow", None, torch.bfloat16, torch.bfloat16, 0, 2, 16, 8, takes_residual=True)
assert bound(torch.zeros(2, 16)) == "slow" and bound(torch.zeros(2, 16), None) == "slow"
with FakeTensorMode() as mode:
    fixed = torch.empty(2, 16, dtype=torch.bfloat16, device="cuda:0")
    out = torch.empty(2, 8, dtype=torch.bfloat16, device="cuda:0")
dynamic = FakeTensorMode(shape_env=ShapeEnv())
with dynamic:
    rows = dynamic.shape_env.create_unbacked_symint()
    symbolic = torch.empty(rows, 16, dtype=torch.bfloat16, device="cuda:0")
for args in ((fixed,), (fixed, out), (fixed, None, out), (symbolic,), (fixed, symbolic), (fixed, None, symbolic)):
    try:
        got = bound(*args)
    except Exception as error:
        assert type(error).__module__.startswith(("builtins", "torch")), error
    else:
        assert got == "slow"
print("survived")
'''


def test_fake_tensors_raise_in_python():
    """A tensor without data or with symbolic sizes makes torch's C++ queries throw; a C function must not let that out (it
    ended the process, so the calls are made in a child)."""

    pytest.importorskip("xqt_b200._host")
    child = subprocess.run([sys.executable, "-c", _SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300,
                           env={**os.environ, "PYTHONPATH": str(ROOT)})
    assert child.returncode == 0 and "survived" in child.stdout, child.stderr[-2000:]


def test_bound_objects_behave_like_closures():
    host = pytest.importorskip("xqt_b200._host")
    import torch

    run = host.Bound(((1, 1, (), (), 0, 0),), lambda *args: args, None, torch.bfloat16, torch.bfloat16, 0, 1, 8, 8, keep=("kept",))
    run.label = "x"
    assert copy.copy(run) is run and copy.deepcopy(run) is run and run.label == "x" and run.__dict__ == {"label": "x"}
    for wrong in (lambda: delattr(run, "slow"), lambda: setattr(run, "slow", None), lambda: delattr(run, "keep"), lambda: setattr(run, "keep", ())):
        with pytest.raises((TypeError, AttributeError)):
            wrong()
    run.slow = lambda *args: "replaced"
    assert run(1) == "replaced"
    gone, cycle = weakref.ref(run), [run]
    run.cycle = cycle
    del run, cycle
    gc.collect()
    assert gone() is None
