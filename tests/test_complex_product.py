"""The complex products of the line passes (cmul and cmul_conj of fft_line.cuh, compiled
for the host): each part is one fused multiply-add by b.x onto a rounded product by b.y,
so its error is at most u |part| + u |product by b.y| (1 + u), u = 2^-24.  With multipliers
near 1, as a slice's transmission and the propagator's low frequencies are, that is one
rounding at full size.  No GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="needs nvcc")
def test_products_round_once_at_full_size(tmp_path):
    from utr_public_gb300 import _build
    exe = str(tmp_path / "complex_product_host")
    subprocess.run([_build.nvcc()] + _build.ARCH + ["-O3", "-std=c++17",
                    "-I" + os.path.join(ROOT, "utr_public_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "complex_product_host.cu"), "-o", exe], check=True)
    rng = np.random.default_rng(5)
    n = 20000
    a = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    b = np.exp(1j * np.concatenate([rng.normal(0, 0.05, n // 2), rng.uniform(-np.pi, np.pi, n // 2)]))
    b = b.astype(np.complex64)
    inp, out = tmp_path / "in.bin", tmp_path / "out.bin"
    np.stack([a, b], 1).tofile(inp)
    subprocess.run([exe, str(inp), str(out)], check=True)
    got = np.fromfile(out, np.complex64).reshape(n, 2).astype(np.complex128)
    # the products of two 24-bit numbers are exact in double
    ar, ai, br, bi = (q.astype(np.float64) for q in (a.real, a.imag, b.real, b.imag))
    u = 2.0**-24
    for k, sign in ((0, 1.0), (1, -1.0)):
        re, im = ar * br - sign * ai * bi, ai * br + sign * ar * bi
        small_re, small_im = np.abs(ai * bi), np.abs(ar * bi)
        for part, exact, small in ((got[:, k].real, re, small_re), (got[:, k].imag, im, small_im)):
            bound = u * np.abs(exact) + u * small * (1 + u)
            assert (np.abs(part - exact) <= bound * (1 + 2.0**-20)).all()
