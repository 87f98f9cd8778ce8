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
