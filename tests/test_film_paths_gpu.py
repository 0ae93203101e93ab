"""The film resolve's fast evaluations against the reference's arithmetic in FP64 (numpy)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _resolve(film, fmt, param=0.0):
    import torch
    from spica_gb300 import gpu
    dev = torch.from_numpy(np.ascontiguousarray(film, np.float32)).cuda()
    return gpu.film_resolve(gpu.Context(0), dev, fmt, param).cpu().numpy()


def _near(values, weight, ulps=(-3, -1, 0, 1, 3)):
    """Film sums whose quotient by the weight lies on or a few float32 ulps beside the values."""
    c = (np.asarray(values, np.float64) * weight).astype(np.float32)
    return np.concatenate([c + np.float32(k) * np.spacing(c) for k in ulps])


def _rows(sums, weight, rng):
    """A film of one row: each sum as red, green and blue of some pixel."""
    rgb = np.stack([sums, rng.permutation(sums), rng.permutation(sums)], 1).astype(np.float32)
    return np.concatenate([rgb, np.full((rgb.shape[0], 1), weight, np.float32)], 1)[None]


ODD_PIXELS = np.array([[0, 0, 0, 0], [0, 0, 0, 4], [1, 2, 3, 0], [1e-30, 0, 0, 1], [1e30, 1e20, 1, 1], [5, 5, 5, 1e-6],
                       [17 * 16, 12 * 16, 4 * 16, 16], [1, 1, 1, 1], [3e38, 1, 0, 2], [0.5, 0.25, 0.125, 1],
                       [-1, 2, 3, 1], [np.inf, 1, 2, 1], [1, np.nan, 2, 1], [1, 2, 3, 3e9]], np.float32)


@pytest.mark.parametrize("gamma", [2.2, 1.0, 0.5, 0.02, 7.0])
@pytest.mark.parametrize("weight", [1.0, 3.0, 16.0, 1000.5])
def test_gamma_bytes_at_their_steps(gpulib, gamma, weight):
    """Bytes of values on and beside every step (k / 255)^gamma, at random, and of pixels with
    unusual weights and values: equal to the FP64 evaluation, save that a value within an ulp or
    two of FP64 of a step may take either byte, as the two pow functions differ by that."""
    from spica_gb300 import gpu
    rng = np.random.default_rng(3)
    steps = (np.arange(256) / 255.0) ** gamma
    sums = np.concatenate([_near(steps, weight), (rng.random(5000) ** 3 * 1.5 * weight).astype(np.float32)])
    film = np.concatenate([_rows(sums, weight, rng), ODD_PIXELS[None]], 1)
    got = _resolve(film, gpu.FILM_GAMMA_BYTES, gamma).astype(int)
    f = film.astype(np.float64)
    with np.errstate(all="ignore"):
        v = 255.0 * np.fmax(0.0, np.fmin(np.fmin(np.fmax((f[..., :3] / (f[..., 3:] + 1e-12)) ** (1.0 / gamma), 0.0),
                                                 1.0), 1.0))
    want = v.astype(int)
    tie = np.abs(v - np.round(v)) < 255 * 2e-15
    assert np.all((got == want) | (tie & (np.abs(got - want) <= 1))), np.argwhere(got != want)[:5]


@pytest.mark.parametrize("weight", [1.0, 3.0, 16.0, 1000.5])
def test_rgbe_at_its_steps(gpulib, weight):
    """RGBE of values on and beside the mantissa steps and the exponents' limits, and of unusual
    pixels, against HDRPixel in FP64 (core/image.cc:72-88)."""
    from spica_gb300 import gpu
    rng = np.random.default_rng(4)
    values = np.concatenate([np.arange(1, 257) / 256.0, np.arange(1, 257) / 16.0, 2.0 ** np.arange(-30.0, 30.0)])
    sums = np.concatenate([_near(values, weight), rng.lognormal(0, 3, 5000).astype(np.float32) * np.float32(weight)])
    odd = ODD_PIXELS[np.isfinite(ODD_PIXELS).all(1) & (ODD_PIXELS >= 0).all(1)]
    film = np.concatenate([_rows(sums, weight, rng), odd[None]], 1)
    got = _resolve(film, gpu.FILM_RGBE)
    c = film[..., :3].astype(np.float64) / (film[..., 3:].astype(np.float64) + 1e-12)
    d = c.max(-1)
    m, e = np.frexp(d)
    with np.errstate(all="ignore"):
        scale = np.where(d <= 1e-32, 0.0, m * 256.0 / d)
    want = np.concatenate([(c * scale[..., None]).astype(np.uint8),
                           np.where(d <= 1e-32, 0, e + 128).astype(np.uint8)[..., None]], -1)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("width, height", [(1, 1), (1, 9), (9, 1), (2, 2), (63, 65), (64, 64), (129, 5), (1920, 3),
                                           (1921, 3), (3, 1921), (2100, 7), (5, 4000)])
def test_durand_chunked_filter(gpulib, width, height):
    """The line filter in chunks, and in tiles for lines longer than a block holds, against the
    restatement's serial recursion (2e-6 relative, the float32 output's tolerance in
    test_film_gpu.py)."""
    from oracle import tmo_oracle
    from spica_gb300 import gpu
    rng = np.random.default_rng(width * 7 + height)
    film = np.concatenate([rng.lognormal(0, 1.5, (height, width, 3)), np.full((height, width, 1), 4.0)], -1)
    film = film.astype(np.float32)
    film[rng.random((height, width)) < 0.05, :3] = 0.0
    if width * height == 1:
        film[...] = (1.0, 2.0, 3.0, 4.0)
    got = _resolve(film, gpu.FILM_DURAND, 5.0)
    with np.errstate(all="ignore"):
        want = tmo_oracle.durand(film, 5.0)
    np.testing.assert_allclose(got, want, rtol=2e-6, atol=1e-12)


def test_durand_non_finite_pixel(gpulib):
    """One infinite pixel: the recursion carries it to every pixel, and a NaN channel clamps to 0."""
    from oracle import tmo_oracle
    from spica_gb300 import gpu
    film = np.ones((40, 50, 4), np.float32)
    film[17, 49, 1] = np.inf
    with np.errstate(all="ignore"):
        want = tmo_oracle.durand(film, 5.0)
    np.testing.assert_array_equal(_resolve(film, gpu.FILM_DURAND, 5.0), want)


@pytest.mark.parametrize("odd", [(-5e-7, -5e-7, -5e-7, 1.0), (0.0, 0.0, 0.0, 0.0), (1.0, 2.0, 3.0, 0.0),
                                 (1e30, 1.0, 1.0, 1.0)])
@pytest.mark.parametrize("contrast", [0.5, 5.0, 200.0])
def test_durand_odd_pixels(gpulib, contrast, odd):
    """The detail layer as a factor where the reference takes its logarithm: a negative one has
    none, and its pixel clamps to 0 (tolerances as in test_durand_chunked_filter)."""
    from oracle import tmo_oracle
    from spica_gb300 import gpu
    rng = np.random.default_rng(3)
    film = np.concatenate([rng.lognormal(0, 2.0, (33, 47, 3)), np.full((33, 47, 1), 4.0)], -1).astype(np.float32)
    film[rng.random((33, 47)) < 0.05, :3] = 0.0
    film[12, 20] = odd
    with np.errstate(all="ignore"):
        want = tmo_oracle.durand(film, contrast)
    np.testing.assert_allclose(_resolve(film, gpu.FILM_DURAND, contrast), want, rtol=2e-6, atol=1e-12)


@pytest.mark.parametrize("odd", [None, (0.0, 0.0, 0.0, 0.0), (-1.0, 0.2, 0.1, 1.0), (1.0, 2.0, 3.0, 0.0),
                                 (np.inf, 1.0, 1.0, 4.0), (1.0, np.nan, 1.0, 4.0)])
@pytest.mark.parametrize("param", [0.18, 0.5, 0.85, 1.0, 1.7])
def test_reinhard_and_drago_with_odd_pixels(gpulib, param, odd):
    """The operators' reduced FP64 arithmetic on films over six decades, with black pixels and one
    unusual one (a negative, infinite or NaN channel, no weight), against the restatement (2e-6
    relative, as in test_film_gpu.py; the same values not finite)."""
    from oracle import tmo_oracle
    from spica_gb300 import gpu
    rng = np.random.default_rng(9)
    film = np.concatenate([rng.lognormal(0, 2.5, (37, 53, 3)), np.full((37, 53, 1), 4.0)], -1).astype(np.float32)
    film[rng.random((37, 53)) < 0.05, :3] = 0.0
    if odd is not None:
        film[20, 31] = odd
    for fmt, op in ((gpu.FILM_REINHARD, tmo_oracle.reinhard), (gpu.FILM_DRAGO, tmo_oracle.drago)):
        with np.errstate(all="ignore"):
            want = op(film, param).astype(np.float32)
        np.testing.assert_allclose(_resolve(film, fmt, param), want, rtol=2e-6, atol=1e-30)
