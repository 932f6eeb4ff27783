"""The extension with the per-step calls of Python hosts: bound by load() whatever was imported before it, and taking what
the calls took.  No GPU: the calls get as far as the library's argument checks."""
import os
import subprocess
import sys
import sysconfig

import pytest

from slang_b200 import lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_api_imported_before_the_extension_exists():
    code = """
import sys
sys.modules["slang_b200._fastcall"] = None      # an import of it fails, as before the first build
from slang_b200 import api, lib
del sys.modules["slang_b200._fastcall"]
lib.load()
buffer = api.Buffer.__new__(api.Buffer)
buffer.device, buffer._h, buffer.size = api.Device.__new__(api.Device), 0, 4
buffer.device._h = 0
try:
    buffer.clear()
except lib.MlpError as e:
    print("refused:", e)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "refused: mlp error" in r.stdout, r.stderr


def test_the_extension_is_named_for_its_python():
    lib.load()
    assert lib.fastcall.__file__.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


@pytest.mark.parametrize("input_grads", [None, 0])
def test_no_input_gradients_may_be_none(input_grads):
    from slang_b200 import api
    lib.load()

    class Handle:
        _h = address = 0

    trainer = api.Trainer.__new__(api.Trainer)
    trainer.device = trainer.k_learn = trainer.network = trainer.loss = Handle()
    with pytest.raises(lib.MlpError):
        trainer.learn_gradient(0, 0, 16, clear_loss=False, input_grads_address=input_grads)
