"""The transport, reverse, thin and J v kernels at the edges of their tiles and dispatches.

Sizes: fewer rays than a warp and a ragged last group of 32, sample counts around the re-anchoring interval and
the kernels' runs of 16 to 64 samples, splat counts around the 32-bit mask words, more frequencies than a unit
takes, the half-orbit cutoff over several segments, tables too large for shared memory, FP64 renders and
gradients in several pieces of rays.

Tolerances: FP64 against the oracle 1e-9 (the two order their operations differently, which moves the azimuth of
ill-conditioned rays by up to 7e-9 rad; with a few coarse samples on a few rays such a ray can carry the image); the
anchor residuals 1e-8 between two ways to march a ray (they are differences of sums of order 1e3); the FP32 transport against FP64 1e-4 (its budget); the FP32 gradient and J v against FP64 1e-3
(the adjoint tests' criterion); two FP64 runs of the same rays in other groupings 1e-12.
"""
import numpy as np
import pytest

import kerrsplat_b200 as ks
from kerrsplat_b200 import scenes

pytestmark = pytest.mark.gpu

A, THO = 0.5, np.deg2rad(60.0)
L = ks.gravitational_radius(4.0e6)


def rel(x, y):
    """The 2-norm of x - y over y's; of x alone where y is zero (a screen whose rays meet no splat)."""
    n = np.linalg.norm(y)
    return np.linalg.norm(np.asarray(x) - np.asarray(y)) / (n if n > 0 else 1.0)


def wide_splats(n, seed):
    """Splats large and close enough for a screen of a few pixels to see each."""
    rng = np.random.Generator(np.random.PCG64(seed))
    p = scenes.thermal_params(rng, n, A, rlo=3.0, rhi=8.0)
    p[3:6] = np.log(rng.uniform(0.8, 2.0, (3, n)))
    return p


def cache_of(cam, N, uneven=None):
    c = ks.GeodesicCache(cam, N)
    return ks.regenerate(c, A, THO, uneven=uneven)


@pytest.mark.parametrize("na,nb,N,ns,nf,nmax", [(1, 2, 5, 1, 1, -1), (7, 5, 17, 3, 2, -1), (33, 1, 64, 33, 1, 0), (11, 9, 130, 97, 3, -1),
                                                (8, 8, 70, 5, 5, 1), (16, 7, 257, 64, 1, -1), (6, 6, 96, 300, 1, -1)])
def test_transport_edges(oracle, na, nb, N, ns, nf, nmax):
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (na, nb))
    cache, p = cache_of(cam, N), wide_splats(ns, 5)
    nus = np.geomspace(86e9, 690e9, 5)[:nf]
    m = ks.PolarizedSplats(p)
    kw = dict(nmax=nmax, slab=0.3)
    plain = np.asarray(ks.render(cache, m, [0.0, 4.0], nus, L, **kw))
    mixed = np.asarray(ks.render(cache, m, [0.0, 4.0], nus, L, precision=ks.KS_MIXED, **kw))
    for v in range(nf):
        ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, N, 64, [("thermal", p, None)], 4.0, nus[v], L, nmax=nmax, slab=0.3)
        assert rel(plain[v, 1], ref) < 1e-9, v
    assert rel(mixed, plain) < 1e-4
    ds = np.random.Generator(np.random.PCG64(6)).standard_normal(plain.shape)
    g64 = ks.adjoint(cache, m, [0.0, 4.0], nus, L, ds, **kw)
    g32 = ks.adjoint(cache, m, [0.0, 4.0], nus, L, ds, precision=ks.KS_MIXED, **kw)
    assert rel(g32, g64) < 1e-3
    # the gradient along a direction is dstokes . J v
    d = np.random.Generator(np.random.PCG64(7)).standard_normal((3, 21, ns)) * np.maximum(np.abs(p), 0.1)
    j64 = ks.jvp(cache, m, [0.0, 4.0], nus, L, d[:1], **kw)
    dual, back = np.sum(ds * j64[0]), np.sum(g64 * d[0])
    assert abs(dual - back) <= 1e-9 * np.sum(np.abs(ds * j64[0]))
    for nd in (1, 2, 3):
        j32 = ks.jvp(cache, m, [0.0, 4.0], nus, L, d[:nd], precision=ks.KS_MIXED, **kw)
        assert rel(j32[0], j64[0]) < 1e-3, nd
    cache.close()


@pytest.mark.parametrize("shift", [-12.0, -4.0, 0.0, 2.0])
def test_step_adjoint_strengths(shift):
    """The FP32 gradient over electron densities e^shift apart, thin to thick. (test_gpu_device_functions.py runs the step
    adjoint by itself on both sides of its switch.)"""
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (17, 15))
    cache, p = cache_of(cam, 96), wide_splats(12, 8)
    p[12] += shift
    nus, m = [86e9, 230e9], ks.PolarizedSplats(p)
    ds = np.random.Generator(np.random.PCG64(9)).standard_normal(np.shape(ks.render(cache, m, [2.0], nus, L)))
    g64 = ks.adjoint(cache, m, [2.0], nus, L, ds)
    assert rel(ks.adjoint(cache, m, [2.0], nus, L, ds, precision=ks.KS_MIXED), g64) < 1e-3
    cache.close()


@pytest.mark.parametrize("N,uneven", [(1, None), (63, None), (65, None), (129, None), (1000, None), (640, (300.0, 64))])
def test_thin_pieces(oracle, N, uneven):
    cam = ks.Camera((-11.9, 12.3), (-12.1, 11.7), (13, 11))
    cache = cache_of(cam, N, uneven)
    p = scenes.config1(res=4, N=8)["params"]
    img = np.asarray(ks.thin_image(cache, p, 3.0)).T.ravel()
    thin_residuals = cache.residuals()
    cache.samples()   # the whole march of every ray in one thread: the same anchors are checked
    for x, y in zip(thin_residuals, cache.residuals()):
        assert np.all(np.abs(x - y) <= 1e-8)
    nper = np.empty(cam.npix, dtype=int)
    nper[cache.perm] = cache.nsamples_per_ray
    ref = np.zeros(cam.npix)
    for Nj in np.unique(nper):
        q = nper == Nj
        ref[q] = oracle.thin_image(A, THO, cam.alpha[q], cam.beta[q], int(Nj), 64, p, 3.0)
    assert rel(img, ref) < 1e-9
    cache.close()


def test_tables_past_shared_memory(oracle):
    rng = np.random.Generator(np.random.PCG64(8))
    p = scenes.powerlaw_params(rng, 546, A)
    p[3:6] = np.log(rng.uniform(0.3, 0.8, (3, 546)))
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (5, 4))
    cache = cache_of(cam, 32)
    img = np.asarray(ks.render(cache, ks.PowerLawSplats(p), [0.0], [230e9], L))[0, 0]
    ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, 32, 64, [("powerlaw", p, None)], 0.0, 230e9, L)
    assert rel(img, ref) < 1e-10
    cache.close()


@pytest.mark.parametrize("nf", [1, 4])
def test_population_fits(oracle, nf):
    """Power-law and kappa fits from their splats' constants: indices around 2 and in each interval of the kappa
    rotativity fits, the intervals' ends and beyond them, narrow and wide kappa distributions."""
    rng = np.random.Generator(np.random.PCG64(12))
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (9, 7))
    cache = cache_of(cam, 70)
    pp, pk = scenes.powerlaw_params(rng, 4, A), scenes.kappa_params(rng, 9, A)
    for q in (pp, pk):
        q[3:6] = np.log(rng.uniform(0.8, 2.0, q[3:6].shape))
    pp[13] = [1.9, 2.1, 2.5, 3.5]
    pk[13] = [3.05, 3.5, 3.75, 4.0, 4.25, 4.5, 4.75, 5.0, 6.5]
    pk[14] = np.log([0.3, 1.0, 3.0, 50.0, 20.0, 10.0, 5.0, 2.0, 1.0])
    kap = ks.KappaSplats(pk)
    m, nus = ks.CompositeModel(ks.PowerLawSplats(pp), kap), np.geomspace(43e9, 690e9, 4)[:nf]
    plain = np.asarray(ks.render(cache, m, [3.0], nus, L))
    for v in range(nf):
        ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, 70, 64, [("powerlaw", pp, None), ("kappa", pk, kap.hyp)], 3.0, nus[v], L)
        assert rel(plain[v, 0], ref) < 1e-9, v
    assert rel(np.asarray(ks.render(cache, m, [3.0], nus, L, precision=ks.KS_MIXED)), plain) < 1e-4
    cache.close()


def test_fp32_rows_in_global_memory(oracle):
    # 500 knot splats with ten knots each: within the largest FP32 table, past a block's shared memory with its rows
    p = wide_splats(500, 13)
    p[3:6] -= 1.5
    times = np.linspace(-60.0, 40.0, 10)
    knots = scenes.trajectory_knots(p, A, times)
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (9, 7))
    cache = cache_of(cam, 40)
    ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, 40, 64, [("knot", p, None, knots, times)], 3.0, 230e9, L)
    img = np.asarray(ks.render(cache, ks.KnotSplats(p, knots, times), [3.0], [230e9], L, precision=ks.KS_MIXED))
    assert rel(img[0, 0], ref) < 1e-4
    cache.close()


def test_fp64_pieces_of_rays():
    # 52900 rays x 2048 samples: two pieces of the FP64 stream and two of the adjoint's state
    p, N = wide_splats(4, 9), 2048
    m = ks.PolarizedSplats(p)
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), 230)
    ds = np.random.Generator(np.random.PCG64(10)).standard_normal((1, 1, cam.npix, 4))
    cache = cache_of(cam, N)
    img = np.asarray(ks.render(cache, m, [0.0], [230e9], L))[0, 0]
    g = ks.adjoint(cache, m, [0.0], [230e9], L, ds)
    cache.close()
    parts, total = np.empty_like(img), np.zeros_like(g)
    for q in np.array_split(np.arange(cam.npix), 3):
        c = cache_of(ks.Camera(cam.alpha[q], cam.beta[q]), N)
        parts[q] = np.asarray(ks.render(c, m, [0.0], [230e9], L))[0, 0]
        total += ks.adjoint(c, m, [0.0], [230e9], L, ds[:, :, q])
        c.close()
    assert rel(img, parts) < 1e-12 and rel(g, total) < 1e-12
