"""A wait of the tile queue that runs out, and who learns of it (native/queue_wait.cu)."""
import os
import subprocess

import pytest

from antelope_b200 import build, cfgtext
from cases import variant

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_wait_that_runs_out_is_seen(tmp_path):
    exe, cfg = tmp_path / "queue_wait", tmp_path / "inputParam.cfg"
    cfg.write_text(cfgtext.dumps(variant(calc__shotNumber=10)))
    lib = os.path.dirname(build.LIB)
    subprocess.check_call([build.NVCC] + build.ARCH + ["-std=c++17", "-I", build.CSRC, "-o", str(exe),
                          os.path.join(HERE, "native", "queue_wait.cu"), "-L", lib, "-lsbe_b200", "-Xlinker",
                          "-rpath," + lib])
    out = subprocess.run([str(exe), str(cfg)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
