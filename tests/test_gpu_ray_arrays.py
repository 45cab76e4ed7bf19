"""Ray queries over separate arrays equal the same queries over packed records, refuse the same rays
with the same message, and run from several threads at once.
"""

import ctypes as C
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from minirender_b200 import _abi, scene as sc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from minirender_b200 import api as a
    return a


@pytest.fixture(scope="module", params=[False, True], ids=["flat", "two-level"])
def scene(api, request):
    return api.Scene(sc.job_scene(12_000, 5).snapshot(), two_level=request.param)


def packed_intersect(api, scene, *rays):
    """mr_intersect and mr_occluded on records."""
    records = api.pack_rays(*rays)
    n = len(records)
    hits, occluded = np.zeros(n, api.HIT_DTYPE), np.zeros(n, np.uint8)
    pointer = C.cast(records.ctypes.data, C.POINTER(_abi.Ray))
    lib = scene.lib
    _abi.check(lib.mr_intersect(scene.handle, pointer, n,
                                C.cast(hits.ctypes.data, C.POINTER(_abi.Hit)), None), lib)
    _abi.check(lib.mr_occluded(scene.handle, pointer, n,
                               occluded.ctypes.data_as(C.POINTER(C.c_uint8)), None), lib)
    return hits, occluded.astype(bool)


def rays(n, seed=3):
    rng = np.random.default_rng(seed)
    o = rng.uniform((-0.45, 0.05, -0.45), (0.45, 0.95, 0.45), (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o, d.astype(np.float32), rng.uniform(0, 0.2, n).astype(np.float32), \
        rng.uniform(0.2, 2.0, n).astype(np.float32)


@pytest.mark.parametrize("n", [0, 1, 31, 127, 129, 5000])
def test_arrays_equal_records(api, scene, n):
    o, d, lo, hi = rays(n)
    for interval in ((1e-5, np.inf), (lo, hi), (lo, 1.0), (0.1, hi)):
        hits, _ = scene.intersect(o, d, *interval)
        occluded, _ = scene.occluded(o, d, *interval)
        expected, expected_occluded = packed_intersect(api, scene, o, d, *interval)
        np.testing.assert_array_equal(hits, expected)
        np.testing.assert_array_equal(occluded, expected_occluded)
    # Strided, double-precision and broadcast inputs are the same rays.
    again, _ = scene.intersect(np.asfortranarray(o.astype(np.float64)), d[:, ::-1][:, ::-1], lo, hi)
    np.testing.assert_array_equal(again, scene.intersect(o, d, lo, hi)[0])
    if n:
        one, _ = scene.intersect(o, d[:1], lo, hi)
        np.testing.assert_array_equal(one, scene.intersect(o, np.repeat(d[:1], n, 0), lo, hi)[0])


@pytest.mark.parametrize("bad", [0, 200, 256])
@pytest.mark.parametrize("field,value,message", [
    ("o", np.nan, "must be finite"), ("o", np.inf, "must be finite"), ("d", 0.9, "unit length"),
    ("lo", -1e-6, "0 <= minimum"), ("lo", np.inf, "0 <= minimum"), ("hi", np.nan, "0 <= minimum"),
    ("hi", 0.0, "0 <= minimum")])
def test_invalid_rays_are_refused(api, scene, field, value, message, bad):
    o, d, lo, hi = rays(257)
    lo += np.float32(1e-3)
    if field == "d":
        d[bad] *= np.float32(value)
    else:
        {"o": o, "lo": lo, "hi": hi}[field][bad] = value
    for call in (scene.intersect, scene.occluded, lambda *r: packed_intersect(api, scene, *r)):
        with pytest.raises(api.MiniRenderError, match=message):
            call(o, d, lo, hi)
    o, d, lo, hi = rays(257)
    assert len(scene.intersect(o, d, lo, hi)[0]) == 257  # the next call is unaffected


def test_threads_share_the_pools(api, scene):
    inputs = [rays(1000 + 37 * k, k) for k in range(12)]
    settings = api.IntegratorSettings("mis", 4, True, 3)
    tracer = api.PathTracer(scene, settings)
    expected = [scene.intersect(*r)[0] for r in inputs]
    images = [tracer.render(api.RenderSettings(40 + k, 30, 2, k + 1))[0] for k in range(12)]

    def work(k):
        return scene.intersect(*inputs[k])[0], tracer.render(api.RenderSettings(40 + k, 30, 2, k + 1))[0]

    with ThreadPoolExecutor(6) as pool:
        for _ in range(3):
            for k, (hits, image) in enumerate(pool.map(work, range(12))):
                np.testing.assert_array_equal(hits, expected[k])
                np.testing.assert_array_equal(image, images[k])
