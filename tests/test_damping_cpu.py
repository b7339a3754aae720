"""The absorbing layers' coefficients a and b on the host, against 64 bits at every depth of a layer."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

SOURCE = r"""
#include "damping.hpp"
extern "C" void damping(int n, const float *vp, const float *K, const float *alpha, float dt, float *a, float *b) {
    for (int i = 0; i < n; i++) jv::damping_ab(vp[i], K[i], alpha[i], dt, a[i], b[i]);
}
"""


@pytest.fixture(scope="module")
def damping(tmp_path_factory):
    d = tmp_path_factory.mktemp("damping")
    (d / "d.cpp").write_text(SOURCE)
    so = str(d / "d.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, PKG, "csrc"), str(d / "d.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(vp, K, alpha, dt):
        out = [np.empty_like(vp) for _ in range(2)]
        lib.damping(vp.size, *(x.ctypes.data_as(ctypes.c_void_p) for x in (vp, K, alpha)), ctypes.c_float(dt),
                    *(x.ctypes.data_as(ctypes.c_void_p) for x in out))
        return out
    return run


@pytest.mark.parametrize("pml,h,fm,dt", [(4, 5.0, 20.0, 4e-4), (16, 5.0, 20.0, 4e-4), (20, 10.0, 40.0, 8e-4),
                                         (60, 2.5, 60.0, 1e-4), (200, 5.0, 25.0, 1e-3)])
def test_coefficients_at_every_depth(damping, pml, h, fm, dt):
    """With u = 2^-24: d and e = d + alpha round to u and 2u relative, so b is off by 4u for expf (2 ulp) and by 3u
    e dt for its argument; b - 1 rounds once more; then a product and a quotient.  a must be that close relative to
    itself, also where d << alpha and a << 1 - b."""
    n = 2 * (pml - 2)
    q = np.tile((np.arange(n) + 1) / (n + 1.0) if pml == 4 else (np.arange(n) + 0.5) / n, 3)
    vp = np.repeat(np.array([1500.0, 2731.0, 5200.0], np.float32), n)
    K = (21.0 / (2.0 * (pml - 2) * h) * q * q).astype(np.float32)
    alpha = (np.pi * fm * (1.0 - q)).astype(np.float32)
    a, b = damping(vp, K, alpha, dt)
    d = vp.astype(np.float64) * K
    e, dt64 = d + alpha, float(np.float32(dt))
    B, w = np.exp(-e * dt64), np.expm1(-e * dt64)
    A = d * w / e
    u = 2.0 ** -24
    db = B * (4 + 3 * e * dt64) * u
    assert np.all(np.abs(b - B) <= db)
    assert np.all(np.abs(a - A) <= d / e * db + 8 * u * np.abs(A)), (np.abs(a / A - 1).max())


def test_a_cell_that_does_not_absorb(damping):
    z = np.zeros(2, np.float32)
    a, b = damping(np.array([0.0, 3000.0], np.float32), z, z, 1e-3)
    assert np.all(a == 0) and np.all(b == 1)
