"""Device functions by themselves, compiled from the library's headers (tests/device_functions.cu)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from kerrsplat_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    src, out = os.path.join(os.path.dirname(os.path.abspath(__file__)), "device_functions.cu"), tmp_path_factory.mktemp("probe") / "probe.so"
    subprocess.run(build.nvcc_flags() + ["-I", build.CSRC, "-shared", "-o", str(out), src], check=True)
    return ctypes.CDLL(str(out))


def ptr(x):
    return ctypes.c_void_p(x.ctypes.data)


def test_fp64_sincos(probe):
    """Absolute error under 2e-16 up to 1e5, and 2e-16 beyond, where the library's function answers; on either side of
    the switch, next to multiples of pi/2, at zero, infinite and undefined arguments. numpy's extended precision is the
    reference (5e-20)."""
    rng = np.random.Generator(np.random.PCG64(40))
    near = np.round(rng.uniform(-63000, 63000, 20000)) * (np.pi / 2)
    x = np.concatenate([rng.uniform(-1e5, 1e5, 400000), rng.uniform(-4, 4, 100000), near, np.nextafter(near, 1e9), near + rng.uniform(-1e-6, 1e-6, near.size),
                        np.nextafter([1e5, 1e5, -1e5], [0, 2e5, 0]), [0.0, -0.0, 5e-324, 1e-8, 1e5, -1e5], 10.0 ** rng.uniform(5, 12, 1000)])
    x = np.ascontiguousarray(np.concatenate([x, [np.inf, -np.inf, np.nan]]))
    got = np.empty((2, x.size))
    assert probe.probe_sincos(ctypes.c_longlong(x.size), ptr(x), ptr(got)) == 0
    assert np.all(np.isnan(got[:, -3:]))
    xl = x[:-3].astype(np.longdouble)
    assert np.max(np.abs(got[0, :-3] - np.sin(xl))) < 2e-16
    assert np.max(np.abs(got[1, :-3] - np.cos(xl))) < 2e-16


@pytest.mark.parametrize("strength", [1e-8, 1e-5, 1e-3, 1e-2, 0.0625, 0.1249, 0.1251, 0.5, 4.0, 100.0])
@pytest.mark.parametrize("depth", [1e-3, 0.5, 3.0])
def test_fp32_step_adjoint(probe, strength, depth):
    """The FP32 step adjoint on both sides of its switch at |K|^2 D^2 = 1/8 (power series below, FP64 partials above), row
    by row of c-bar against FP64 duals through the step operator, over random steps: a few tens of FP32 roundings (6e-8)
    a row and moderate cancellation between them, 1e-5."""
    rng = np.random.Generator(np.random.PCG64(41))
    n = 4096
    v = rng.standard_normal((n, 6)) * np.array([1.0, 1.0, 0.3, 1.0, 1.0, 3.0])
    D = np.exp(rng.uniform(-3.0, 3.0, n))
    v *= (np.sqrt(strength) / (np.linalg.norm(v, axis=1) * D))[:, None]
    cs = np.empty((n, 11))
    cs[:, 0] = rng.uniform(0.5, 2.0, n)
    cs[:, 1:4] = 0.3 * rng.standard_normal((n, 3))
    cs[:, 5:] = v
    # alpha_I exceeds the polarized absorption, as the cap leaves it
    cs[:, 4] = np.maximum(depth * rng.uniform(0.5, 1.5, n) / D, np.linalg.norm(v[:, :3], axis=1) / 0.99)
    w, R = rng.standard_normal((n, 4)), rng.standard_normal((n, 4))
    # what the kernel rounds its arguments to
    cs, D, w, R = [np.ascontiguousarray(np.float32(x).astype(float)) for x in (cs, D, w, R)]
    kd2 = np.sum(cs[:, 5:] ** 2, axis=1) * D * D
    assert np.all(kd2 < 0.125) if strength < 0.125 else np.all(kd2 > 0.125)
    out = [np.empty((n, 11)) for _ in range(2)]
    for method in (0, 1):
        assert probe.probe_step_adjoint(ctypes.c_longlong(n), ptr(cs), ptr(D), ptr(w), ptr(R), method, ptr(out[method])) == 0
    # in units that do not weigh long steps over short ones: everything times 1 / D
    got, want = [x / D[:, None] for x in out]
    err = np.linalg.norm(got - want, axis=0) / np.linalg.norm(want, axis=0)
    assert np.all(err < 1e-5), err
