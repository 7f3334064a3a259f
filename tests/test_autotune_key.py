"""The autotuner's choices belong to the kernels they were timed on (no GPU): the
key changes with the library's contents and with nothing else."""

import os
import subprocess
import sys

from finitevolx_b200 import _lib, autotune


def test_key_follows_the_library(tmp_path, monkeypatch):
    so = tmp_path / "libfvx.so"
    so.write_bytes(b"one")
    monkeypatch.setattr(_lib, "LIB_PATH", so)
    monkeypatch.setattr(autotune, "_device_key", lambda: "B200")
    first = autotune._key("qg_stage", "weno5", "2048x2048")
    assert first == autotune._key("qg_stage", "weno5", "2048x2048") != autotune._key("qg_stage", "weno5", "258x258")
    os.utime(so, ns=(1, 1))  # the same build, copied
    assert autotune._key("qg_stage", "weno5", "2048x2048") == first
    so.write_bytes(b"two")
    os.utime(so, ns=(2, 2))
    assert autotune._key("qg_stage", "weno5", "2048x2048") != first


def test_ensemble_key_is_the_same_in_every_process():
    # a key from str's randomised hash never matched in a later run
    code = ("from types import SimpleNamespace as N; from finitevolx_b200 import autotune as a; "
            "a._device_key = a._build_key = lambda: 'x'; "
            "print(a._ensemble_key(N(members=[(128, 2), (256, 3)], method='weno5')))")
    keys = [subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, check=True,
                           env=dict(os.environ, PYTHONHASHSEED=seed)).stdout for seed in ("1", "2")]
    assert keys[0] == keys[1] != ""
