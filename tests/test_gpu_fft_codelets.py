"""The packed register transforms round as the scalar ones do (fft_codelets.cu, compiled here with the library's
flags): which product of a rotation an FMA keeps exact is written out in fft.cuh to match what this compiler does
with the scalar expressions, and the cluster kernels and large-grid diagnostics still have those.  Every radix of
the plans that run on packed values, both directions."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_packed_codelets_equal_scalar_ones(tmp_path):
    import optimizec_b200 as P

    exe = str(tmp_path / "fft_codelets")
    subprocess.check_call([P.NVCC, *P.ARCH, *P.CUFLAGS, "-o", exe, os.path.join(HERE, "fft_codelets.cu")])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
