"""A wait of the tensor-core training kernels that ran out is reported by the call that meets it, once,
and no gradient of that call reaches the parameters (cnn_wait_flag.cu, compiled here)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_wait_flag_is_reported_once_and_training_stops(tmp_path):
    import optimizec_b200 as P

    P.lib()
    exe = str(tmp_path / "cnn_wait_flag")
    lib = os.path.dirname(P.LIB_PATH)
    subprocess.check_call([P.NVCC, *P.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-o", exe,
                           os.path.join(HERE, "cnn_wait_flag.cu"), "-L" + lib, "-ldns2d", "-Xlinker", "-rpath," + lib])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
