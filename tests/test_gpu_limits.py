"""Calls at the limits of what the library takes: waits that run out, times far from zero, splats that hardly emit,
tables and states at the edges of memory, graph replays between other calls."""
import numpy as np
import pytest

import kerrsplat_b200 as ks
from kerrsplat_b200 import scenes

pytestmark = pytest.mark.gpu

A, THO = 0.5, np.deg2rad(60.0)
L = ks.gravitational_radius(4.0e6)


def rel(x, y):
    """The 2-norm of x - y over y's."""
    return np.linalg.norm(np.asarray(x) - np.asarray(y)) / np.linalg.norm(y)


def wide_splats(n, seed):
    """Splats large and close enough for a screen of a few pixels to see each."""
    rng = np.random.Generator(np.random.PCG64(seed))
    p = scenes.thermal_params(rng, n, A, rlo=3.0, rhi=8.0)
    p[3:6] = np.log(rng.uniform(0.8, 2.0, (3, n)))
    return p


def orbit_knots(p, times):
    """The centres of `p` on their pattern circles at `times`, (3, times, splats)."""
    ang = np.arctan2(p[1], p[0]) + p[20] * np.asarray(times)[:, None]
    rho = np.hypot(p[0], p[1])
    return np.stack([rho * np.cos(ang), rho * np.sin(ang), np.broadcast_to(p[2], ang.shape)])


def cache_of(na, nb, N):
    return ks.regenerate(ks.GeodesicCache(ks.Camera((-8.9, 9.3), (-9.1, 8.7), (na, nb)), N), A, THO)


@pytest.mark.parametrize("call", ["render", "adjoint", "chi2_gradient", "adjoint_on_device"])
@pytest.mark.parametrize("precision", [ks.KS_FP64, ks.KS_MIXED])
def test_a_staging_wait_that_runs_out_is_reported(call, precision):
    """Every call whose kernels stage a splat table fails with KS_ERR_TIMEOUT when the copy does not land, leaves a
    gradient that it was to add to alone, and leaves no flag behind for the call after it."""
    import torch
    cache, m = cache_of(9, 7, 64), ks.PolarizedSplats(wide_splats(5, 3))
    ds = np.random.Generator(np.random.PCG64(4)).standard_normal((1, 1, cache.npix, 4))
    held = np.asfortranarray(np.full((21, 5), 3.0))
    dev = torch.full((21 * 5,), 3.0, dtype=torch.float64, device="cuda")
    run = {
        "render": lambda: ks.render(cache, m, [0.0], [230e9], L, precision=precision),
        "adjoint": lambda: ks.adjoint(cache, m, [0.0], [230e9], L, ds, precision=precision, dparams=held),
        "chi2_gradient": lambda: ks.chi2_gradient(cache, m, [0.0], [230e9], L, ds, 1.0, precision=precision, dparams=held),
        "adjoint_on_device": lambda: ks.adjoint(cache, m, [0.0], [230e9], L, ds, precision=precision, dparams=dev),
    }[call]
    cache.set_stage_test(True)
    with pytest.raises(ks.KsError) as err:
        run()
    assert err.value.status == ks._lib.KS_ERR_TIMEOUT
    cache.set_stage_test(False)
    assert np.all(held == 3.0) and bool((dev == 3.0).all())
    ks.thin_image(cache, scenes.config1(res=4, N=8)["params"], 0.0)
    assert np.abs(np.asarray(ks.render(cache, m, [0.0], [230e9], L, precision=precision))).max() > 0
    run()
    if call != "render":
        assert not (np.all(held == 3.0) and bool((dev == 3.0).all()))
    cache.close()


@pytest.mark.parametrize("shift", [1e6, 1e8])
def test_fp64_times_far_from_zero(shift):
    """The same scene at times `shift` later: an FP64 time there is rounded by 1e-16 of it, some 1e-8 M, which moves a
    centre by 1e-8 M and a weight by 1e-7 at most; 1e-6 is allowed."""
    rng = np.random.Generator(np.random.PCG64(21))
    p = scenes.thermal_params(rng, 40, A, rlo=3.0, rhi=8.0)
    p[3:6] = np.log(rng.uniform(0.2, 0.4, (3, 40)))
    p[10], p[11] = rng.uniform(-20.0, 20.0, 40), np.log(1e9)
    later = p.copy(order="F")
    later[10] += shift
    cache = cache_of(24, 22, 128)
    img = np.asarray(ks.render(cache, ks.PolarizedSplats(p), [4.0], [230e9], L))
    assert np.abs(img).max() > 0
    assert rel(ks.render(cache, ks.PolarizedSplats(later), [4.0 + shift], [230e9], L), img) < 1e-6
    ds = rng.standard_normal(img.shape)
    g = ks.adjoint(cache, ks.PolarizedSplats(p), [4.0], [230e9], L, ds)
    h = ks.adjoint(cache, ks.PolarizedSplats(later), [4.0 + shift], [230e9], L, ds)
    for row in range(21):
        assert np.linalg.norm(h[row] - g[row]) <= 1e-6 * max(np.linalg.norm(g[row]), 1e-6 * np.linalg.norm(g)), row
    cache.close()


def test_fp64_samples_at_the_edge_of_a_support(oracle):
    """A narrow splat above the outermost sample of one ray, that sample a little inside the weight cutoff (1e-6), where
    the FP32 rounding of a height of some 1000 M (1e-4 M) is more than the distance to the edge: it shows in FP64 on
    every ray. An oracle sample lies up to 1e-9 M from the library's, 5e-7 of a weight: 1e-5 is allowed."""
    q = np.sqrt(1.0 - A * A)
    for beta in np.linspace(3.1, 9.7, 12):
        cam = ks.Camera(np.array([1.3]), np.array([beta]))
        cache = ks.regenerate(ks.GeodesicCache(cam, 256), A, THO)
        s = cache.samples()
        assert s["flags"][0, 0] & 1
        r, th, ph = s["r"][0, 0], s["theta"][0, 0], s["phi"][0, 0]
        ph = ph + A / (2 * q) * np.log((r - 1 - q) / (r - 1 + q)) - np.arctan2(A, r)   # the azimuth of the splats' frame
        p = wide_splats(1, 23)
        p[3:6] = np.log(0.01)
        p[20], p[11], p[12] = 0.0, np.log(1e9), np.log(1e12)
        p[0:3, 0] = r * np.array([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)])
        p[2] += 0.01 * np.sqrt(2 * 13.8149)   # the weight's exponent at the sample; the cutoff's is 13.8155
        img = np.asarray(ks.render(cache, ks.PolarizedSplats(p), [0.0], [230e9], L))[0, 0]
        ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, 256, 64, [("thermal", p, None)], 0.0, 230e9, L)
        assert np.linalg.norm(ref) > 0
        assert rel(img, ref) < 1e-5, beta
        cache.close()


def test_graph_replays_keep_their_own_call():
    """A captured graph renders the frames, frequencies and knots of its capture whatever calls came between, of the
    same sizes (nothing is reallocated) and of other layouts (J v)."""
    import torch
    cache, cuda = cache_of(16, 14, 96), lambda p: torch.tensor(p, device="cuda")
    p, kt = wide_splats(6, 24), np.linspace(-40.0, 60.0, 5)
    knots = orbit_knots(p, kt)
    other = np.asarray(knots) * 1.2
    thermal = ks.PolarizedSplats(cuda(p))
    data = cuda(np.random.Generator(np.random.PCG64(25)).standard_normal((2, 1, cache.npix, 4)) * 1e-6)
    def between(knots, t, nus):
        img = ks.render(cache, ks.KnotSplats(cuda(p), knots, kt), [t], nus, L, precision=ks.KS_MIXED).cpu().numpy()
        ks.jvp(cache, thermal, [t], nus, L, np.ones((1, 21, 6)), precision=ks.KS_MIXED)
        ks.chi2_gradient(cache, thermal, [t], nus, L, data, 1e-7, precision=ks.KS_MIXED)
        return img

    between(knots, 0.0, [230e9, 86e9])   # the buffers have their sizes
    gc = ks.capture_chi2_gradient(cache, thermal, [0.0], [230e9, 86e9], L, data, 1e-7)
    g = ks.capture_render(cache, ks.KnotSplats(cuda(p), knots, kt), [0.0], [230e9, 86e9], L)
    first = g.replay().cpu().numpy().copy()
    chi2, grad = [x.cpu().numpy().copy() for x in gc.replay()]
    assert np.abs(first).max() > 0 and np.abs(grad).max() > 0
    assert not np.array_equal(between(other, 50.0, [345e9, 43e9]), first)
    assert np.array_equal(g.replay().cpu().numpy(), first)
    again = [x.cpu().numpy() for x in gc.replay()]
    assert np.array_equal(again[0], chi2) and np.array_equal(again[1], grad)
    cache.close()


@pytest.mark.parametrize("nf,values", [(1, 48168), (2, 44072), (3, 39976), (4, 44072), (5, 44072)])
def test_largest_tables_by_frequencies(nf, values):
    """The largest FP32 table (51 values a splat and four a knot) at each number of frequencies is taken, one knot more
    is refused. Four frequencies take what two do. The image is that of the frequencies by themselves: 1e-4 is the FP32
    transport's budget."""
    n = 256
    nk = (values // n - 51) // 4
    p = wide_splats(n, 26)
    p[3:6] -= 1.0
    cache, nus = cache_of(7, 6, 40), np.geomspace(86e9, 690e9, 5)[:nf]

    def model(nk):
        t = np.linspace(-60.0, 40.0, nk)
        return ks.KnotSplats(p, orbit_knots(p, t), t)

    with pytest.raises(ValueError, match="too many splats"):
        ks.render(cache, model(nk + 1), [3.0], nus, L, precision=ks.KS_MIXED)
    m = model(nk)
    img = np.asarray(ks.render(cache, m, [3.0], nus, L, precision=ks.KS_MIXED))
    assert np.abs(img).max() > 0
    for v in range(nf):
        assert rel(img[v], np.asarray(ks.render(cache, m, [3.0], nus[v:v + 1], L, precision=ks.KS_MIXED))[0]) < 1e-4
    cache.close()


@pytest.mark.parametrize("ln_te", [-21.0, -22.0, -24.0, -25.5, -28.0, -32.0])
def test_splats_too_cold_to_emit(oracle, ln_te):
    """Beside ordinary splats, cold ones, where exp(h nu / k T) overflows in FP32 or FP64, only rotate the polarization,
    in the limit T = 0 the same whatever T is: 6 T, 5e-9 of a rotativity at the warmest, so FP64 agrees with the
    oracle's image at the warmest (the others are 0 / 0 to it) to 1e-8; FP32 with FP64 as elsewhere, 1e-4 and 1e-3."""
    p = wide_splats(6, 27)
    p[13, ::2] = ln_te
    warm = p.copy(order="F")
    warm[13, ::2] = -21.0
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), (9, 7))
    cache, m = cache_of(9, 7, 70), ks.PolarizedSplats(p)
    img = np.asarray(ks.render(cache, m, [0.0], [230e9], L))
    ref = oracle.polarized_image(A, THO, cam.alpha, cam.beta, 70, 64, [("thermal", warm, None)], 0.0, 230e9, L)
    assert rel(img[0, 0], ref) < 1e-8
    ds = np.random.Generator(np.random.PCG64(28)).standard_normal(img.shape)
    g = ks.adjoint(cache, m, [0.0], [230e9], L, ds)
    assert np.all(np.isfinite(g))
    assert rel(ks.render(cache, m, [0.0], [230e9], L, precision=ks.KS_MIXED), img) < 1e-4
    assert rel(ks.adjoint(cache, m, [0.0], [230e9], L, ds, precision=ks.KS_MIXED), g) < 1e-3
    cache.close()


@pytest.mark.parametrize("ln_ne", [0.0, -20.0, -28.0, -36.0])
def test_fp32_thin_plasma(ln_ne):
    """The FP32 image of a plasma so thin that e^2 n_e / c underflows in FP32 is as accurate as any: 1e-4, its budget
    (measured 8e-7); its gradient 1e-3."""
    p = wide_splats(6, 27)
    p[12] = ln_ne
    cache, m = cache_of(9, 7, 70), ks.PolarizedSplats(p)
    img = np.asarray(ks.render(cache, m, [0.0], [230e9], L))
    assert rel(ks.render(cache, m, [0.0], [230e9], L, precision=ks.KS_MIXED), img) < 1e-4
    ds = np.random.Generator(np.random.PCG64(28)).standard_normal(img.shape)
    g = ks.adjoint(cache, m, [0.0], [230e9], L, ds)
    assert rel(ks.adjoint(cache, m, [0.0], [230e9], L, ds, precision=ks.KS_MIXED), g) < 1e-3
    cache.close()


@pytest.mark.parametrize("precision", [ks.KS_FP64, ks.KS_MIXED])
def test_gradients_and_renders_in_little_memory(precision):
    """With 600 MB of the device free, less than the state of every ray (1.9 GB in FP64, 0.95 GB in FP32), the gradient,
    its captured graph and the FP64 stream (0.54 GB beside other buffers) go over the screen in pieces. The sums are the
    same but for their grouping: 1e-11 in FP64, 1e-5 in FP32."""
    import torch
    rng = np.random.Generator(np.random.PCG64(30))
    m = ks.PolarizedSplats(torch.tensor(scenes.thermal_params(rng, 10, A, rlo=3.0, rhi=8.0), device="cuda"))
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), 128)
    data = torch.tensor(rng.standard_normal((1, 1, cam.npix, 4)) * 1e-6, device="cuda")

    def calls():
        cache = ks.regenerate(ks.GeodesicCache(cam, 512), A, THO)
        chi2, g, img = ks.chi2_gradient(cache, m, [0.0], [230e9], L, data, 1e-7, precision=precision, return_image=True)
        out = [chi2, np.asarray(g), np.asarray(img.cpu()), np.asarray(ks.render(cache, m, [0.0], [230e9], L, precision=precision).cpu())]
        if precision == ks.KS_MIXED:
            graph = ks.capture_chi2_gradient(cache, m, [0.0], [230e9], L, data, 1e-7)
            graph.dparams.zero_()
            out.append(graph.replay()[1].cpu().numpy().reshape(10, 21).T)
        cache.close()
        return out

    want = calls()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    held = torch.empty(free - 600 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        got = calls()
    finally:
        del held
        torch.cuda.empty_cache()
    tol = 1e-11 if precision == ks.KS_FP64 else 1e-5
    for x, y in zip(got, want):
        assert np.all(np.isfinite(x)) and rel(x, y) < tol
    if precision == ks.KS_MIXED:
        assert rel(got[4], got[1]) < 1e-12


def test_a_failed_allocation_is_over_with_its_call():
    """A call that finds no memory raises MemoryError, and the calls after it, on this context and on a new one, run."""
    import torch
    m = ks.PolarizedSplats(wide_splats(3, 31))
    cam = ks.Camera((-8.9, 9.3), (-9.1, 8.7), 96)
    cache = ks.regenerate(ks.GeodesicCache(cam, 1024), A, THO)
    small = cache_of(7, 6, 32)
    want = np.asarray(ks.render(small, m, [0.0], [230e9], L, precision=ks.KS_MIXED))
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - 200 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(MemoryError):
            ks.render(cache, m, [0.0], [230e9], L, precision=ks.KS_MIXED)   # a stream of 0.3 GB
        assert np.array_equal(ks.render(small, m, [0.0], [230e9], L, precision=ks.KS_MIXED), want)
        cache_of(5, 4, 16).close()
    finally:
        del held
        torch.cuda.empty_cache()
    assert np.abs(np.asarray(ks.render(cache, m, [0.0], [230e9], L, precision=ks.KS_MIXED))).max() > 0
    cache.close()
    small.close()


@pytest.mark.parametrize("shift", [-8.0, 0.0, 2.0])
@pytest.mark.parametrize("nf", [1, 3])
def test_fp32_gradient_by_rows(shift, nf):
    """Each of the 21 parameter rows of the FP32 gradient by itself within 1e-3 of FP64's, the criterion of the gradient
    as a whole (a row below 1e-6 of the largest, in units of the parameters, against that), over weak to strong plasmas:
    measured 1.3e-5 at ordinary densities, 1.2e-4 in the densest at 86 GHz, where the Faraday depth amplifies the
    rounding of the image (7e-5 on FP64 geodesics)."""
    rng = np.random.Generator(np.random.PCG64(32))
    p = wide_splats(14, 33)
    p[12] += shift
    cache, m, nus = cache_of(23, 19, 160), ks.PolarizedSplats(p), [230e9, 86e9, 345e9][:nf]
    ds = rng.standard_normal((nf, 1, cache.npix, 4))
    g = np.asarray(ks.adjoint(cache, m, [2.0], nus, L, ds))
    h = np.asarray(ks.adjoint(cache, m, [2.0], nus, L, ds, precision=ks.KS_MIXED))
    norm = np.linalg.norm(g, axis=1)
    unit = np.array([1.0] * 10 + [10.0] + [1.0] * 9 + [0.1])
    floor = 1e-6 * np.max(norm * unit) / unit
    err = np.linalg.norm(h - g, axis=1) / np.maximum(norm, floor)
    assert np.all(err < 1e-3), err
    cache.close()


@pytest.mark.parametrize("precision,rays,tol", [(ks.KS_MIXED, 6144, 5e-6), (ks.KS_MIXED_GEO64, 6144, 5e-6), (ks.KS_FP64, 8192, 1e-12)])
def test_both_sides_of_the_block_march(precision, rays, tol):
    """Eight segments a ray at 512 samples: below `rays` rays a block marches 32 of them together, above a thread each.
    The same rays on both sides: FP64 to its rounding, FP32 to that of a composition by other segments."""
    cam = ks.Camera((-14.9, 15.3), (-15.1, 14.7), (96, 90))
    rng = np.random.Generator(np.random.PCG64(34))
    m = ks.PolarizedSplats(scenes.thermal_params(rng, 12, A, rlo=3.0, rhi=9.0))
    order = rng.permutation(cam.npix)
    out = []
    for n in (rays - 40, rays + 40):
        q = order[:n]
        cache = ks.regenerate(ks.GeodesicCache(ks.Camera(cam.alpha[q], cam.beta[q]), 512), A, THO)
        out.append(np.asarray(ks.render(cache, m, [1.0], [230e9], L, precision=precision))[0, 0, :rays - 40])
        if precision == ks.KS_MIXED_GEO64:
            assert rel(out[-1], np.asarray(ks.render(cache, m, [1.0], [230e9], L))[0, 0, :rays - 40]) < 1e-4
        cache.close()
    assert np.abs(out[0]).max() > 0
    assert rel(out[0], out[1]) < tol


def test_a_closed_context_leaves_no_graph():
    """Contexts closed with both their graphs captured give the device's memory back (a graph holds some 150 KB, 44 MB in
    all; the driver takes memory in pieces, so some of that may stay)."""
    import torch
    m = ks.PolarizedSplats(torch.tensor(wide_splats(3, 36), device="cuda"))

    def one():
        cache = cache_of(9, 7, 32)
        data = torch.zeros((1, 1, cache.npix, 4), dtype=torch.float64, device="cuda")
        ks.capture_render(cache, m, [0.0], [230e9], L).replay()
        ks.capture_chi2_gradient(cache, m, [0.0], [230e9], L, data, 1e-6).replay()
        cache.close()

    for _ in range(3):
        one()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(300):
        one()
    assert before - torch.cuda.mem_get_info()[0] <= 16 * 2 ** 20


@pytest.mark.parametrize("kappa", [3.05, 7.0, 12.0, 25.0])
def test_fp32_steep_kappa_distributions(kappa):
    """Kappa splats so steep that their image is 1e-20 of an ordinary one's (1e-26): the FP32 image is within 1e-4 of
    FP64, its budget."""
    rng = np.random.Generator(np.random.PCG64(35))
    p = scenes.kappa_params(rng, 4, A)
    p[3:6] = np.log(rng.uniform(0.8, 2.0, (3, 4)))
    p[13], p[14] = kappa, -2.0
    cache, m = cache_of(9, 7, 70), ks.KappaSplats(p)
    img = np.asarray(ks.render(cache, m, [0.0], [230e9], L))
    assert np.all(np.isfinite(img)) and np.abs(img).max() > 0
    assert rel(ks.render(cache, m, [0.0], [230e9], L, precision=ks.KS_MIXED), img) < 1e-4
    cache.close()
