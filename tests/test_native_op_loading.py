"""Loading and building the native operator (CPU): a build for another torch is refused in words and built again, and what
needs no operator does without it."""
import importlib.util
import os

import pytest
import torch

from flash_attention_v100.kernels import _cabi
from flash_attention_v100.ops import attention as ops

CSRC = os.path.join(os.path.dirname(_cabi._PKG_DIR), "csrc")


@pytest.fixture
def unloaded(monkeypatch):
    monkeypatch.setattr(_cabi, "_op", None)
    monkeypatch.setattr(_cabi, "_status_words", {}, raising=False)
    monkeypatch.setattr(ops, "_status_words", {})
    return monkeypatch


def test_an_operator_built_for_another_torch_is_refused(unloaded):
    unloaded.setattr(torch, "__version__", "1.0.0+other")
    with pytest.raises(_cabi.FlashAttentionLibraryError, match=r"built for torch .*, this is 1\.0\.0\+other.*build\.py"):
        _cabi.load_op()
    assert _cabi._op is None


def test_a_file_that_is_no_operator_is_refused(unloaded, tmp_path):
    path = tmp_path / "fa_b200_torch.so"
    path.write_bytes(b"not a library")
    unloaded.setattr(_cabi, "OP_PATH", str(path))
    with pytest.raises(_cabi.FlashAttentionLibraryError, match="does not fit torch"):
        _cabi.load_op()


def test_an_operator_from_before_the_check_is_refused(unloaded):
    unloaded.setattr(_cabi, "OP_PATH", _cabi.LIB_PATH)              # loads, and does not say which torch it is for
    with pytest.raises(_cabi.FlashAttentionLibraryError, match="does not fit torch"):
        _cabi.load_op()


def test_status_words_need_no_operator_and_reach_it_when_it_is_loaded(unloaded, tmp_path):
    unloaded.setattr(torch.Tensor, "pin_memory", lambda t: t)       # (no GPU here)
    real = _cabi.OP_PATH
    unloaded.setattr(_cabi, "OP_PATH", str(tmp_path / "missing.so"))
    first = ops._status_word(torch.device("cuda", 0))
    with pytest.raises(_cabi.FlashAttentionLibraryError, match="not found"):
        ops.native_call(first, first, first, None, False, False, None, False)

    told = {}

    class Op:
        @staticmethod
        def set_status_word(device, address):
            told[device] = address
    unloaded.setattr(_cabi, "OP_PATH", real)
    unloaded.setattr("importlib.util.module_from_spec", lambda spec: Op)
    unloaded.setattr("importlib.machinery.ExtensionFileLoader.exec_module", lambda self, module: None)
    assert _cabi.load_op() is Op
    second = ops._status_word(torch.device("cuda", 3))
    assert told == {0: first.data_ptr(), 3: second.data_ptr()}


def test_the_operator_is_built_again_for_another_torch(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("fa_b200_build", os.path.join(CSRC, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    out = tmp_path / "fa_b200_torch.so"
    monkeypatch.setattr(build, "OP_OUT", str(out))
    commands = []

    class Done:
        returncode, stdout = 0, ""

    def run(cmd, **kw):
        commands.append(cmd)
        out.write_bytes(b"")
        return Done
    monkeypatch.setattr(build.subprocess, "run", run)
    folder, version = build._installed_torch()
    assert version == str(torch.__version__)
    build.build_op()
    build.build_op()
    assert len(commands) == 1                                       # nothing changed
    monkeypatch.setattr(build, "_installed_torch", lambda: (folder, "9.9.9"))
    build.build_op()
    build.build_op()
    assert len(commands) == 2 and '-DFA_TORCH_VERSION="9.9.9"' in commands[1]
