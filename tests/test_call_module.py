"""The call module (`velox_b200/csrc/calls`) where it cannot be had, and calls that it is not asked about.  Needs no GPU."""
import types

import pytest
import torch

from velox_b200.csrc import build, ops


@pytest.fixture
def fresh(monkeypatch):
    monkeypatch.setattr(ops, "_CALLS", None)
    monkeypatch.setattr(ops, "_LIB", types.SimpleNamespace(_name="no library"))
    return monkeypatch


def _raises(error):
    def f(*args, **kwargs):
        raise error
    return f


@pytest.mark.parametrize("error", [build.BuildError("no compiler"), ImportError("no headers"), OSError("no such file")])
def test_operations_are_left_to_the_wrappers_without_the_module(fresh, error):
    """A module that does not compile, or whose build lacks something, costs a warning, once; every operation then says None."""
    fresh.setattr(build, "build_calls", _raises(error))
    with pytest.warns(RuntimeWarning, match=str(error)):
        calls = ops._calls()
    assert calls.gemm_bf16(1, 2, 3) is None and calls.add_rmsnorm() is None
    assert ops._calls() is calls


def test_operations_are_left_to_the_wrappers_when_the_module_does_not_load(fresh, tmp_path):
    (tmp_path / "broken.so").write_bytes(b"no library")
    fresh.setattr(build, "build_calls", lambda *a, **k: str(tmp_path / "broken.so"))
    with pytest.warns(RuntimeWarning, match="cannot be had"):
        assert ops._calls().gated_act() is None


def test_tensors_of_the_host_are_refused_before_anything_is_built(fresh):
    fresh.setattr(ops, "_LIB", None)
    fresh.setattr(build, "build", _raises(AssertionError("built")))
    fresh.setattr(build, "build_calls", _raises(AssertionError("built")))
    fresh.setattr(ops, "_MATMUL_SET", True)
    x, w, ids = torch.zeros(4, 64), torch.ones(64), torch.zeros(4, dtype=torch.int32)
    for call in (lambda: ops.add_rmsnorm(x, None, w, 1e-6, torch.bfloat16), lambda: ops.gated_act(x, "silu"), lambda: ops.gemm_bf16(x.bfloat16(), x.bfloat16()),
                 lambda: ops.qk_norm_rope_kv(x, None, None, 1e-6, None, 0, ids, None, None, None, 2, 1, 16),
                 lambda: ops.gemm_tcgen05(x.bfloat16(), x.bfloat16()),
                 lambda: ops.paged_decode_attention(x.bfloat16(), 64, x, x, ids, ids, ids, 1.0, 0, 1, 1, 64, 4, 4),
                 lambda: ops.paged_prefill_attention_tc(x.bfloat16(), 64, x, x, ids, ids, ids, 1.0, 0, 1, 1, 64, 1, 4, 4)):
        with pytest.raises(ops.KernelError, match="CUDA tensors"):
            call()
