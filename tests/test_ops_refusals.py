"""Arguments that the front end has to refuse before the library sees them.  Runs on CPU: the library is replaced by one
that must not be reached, and the tensors pass for CUDA tensors."""
import subprocess
import sys

import pytest
import torch
from conftest import ROOT

from tilelang_moe_b200 import ops


class _Unreached:
    def __getattr__(self, name):
        raise AssertionError(f"{name} was reached")


@pytest.fixture()
def no_library(monkeypatch):
    monkeypatch.setattr(ops, "_need_cuda", lambda *ts: None)
    monkeypatch.setattr(ops._lib, "load", _Unreached)


@pytest.mark.parametrize("ids,k", [(torch.zeros(7, dtype=torch.int64), 1), (torch.zeros(8, dtype=torch.int64), 2),
                                   (torch.zeros(8, 2, dtype=torch.int32), 1), (torch.zeros(0, dtype=torch.int32), 1),
                                   (torch.zeros(8, dtype=torch.int64), -1)])
def test_routed_gemm_counts_its_ids(no_library, ids, k):
    """The library reads T * k ids from a raw pointer: another number of them would be a read past the tensor."""
    X, W = torch.zeros(8, 64, dtype=torch.bfloat16), torch.zeros(4, 8, 64, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="expert ids"):
        ops.grouped_gemm_routed(X, W, ids, k)


def test_routed_gemm_wants_one_device(no_library):
    X, W = torch.zeros(8, 64, dtype=torch.bfloat16), torch.zeros(4, 8, 64, dtype=torch.bfloat16)
    ids = torch.zeros(8, dtype=torch.int64)
    for args in ((X, W.to("meta"), ids), (X, W, ids.to("meta"))):
        with pytest.raises(ValueError, match="one device"):
            ops.grouped_gemm_routed(*args, 1)


def test_import_under_a_torch_without_cuda():
    """The private functions behind the current device and stream are missing there: the module loads all the same and
    refuses CPU tensors with its message."""
    code = ("import torch\n"
            "for name in ('_cuda_getDevice', '_cuda_getCurrentRawStream'):\n"
            "    if hasattr(torch._C, name): delattr(torch._C, name)\n"
            "from tilelang_moe_b200 import ops\n"
            "try: ops.topk_softmax(torch.zeros(2, 8), 2)\n"
            "except ValueError as e: print(e)\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "CUDA tensors only" in r.stdout, r.stderr
