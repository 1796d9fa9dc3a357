"""Ridge filters on the GPU path: frangi, meijering, sato and the hybrid
hessian filter against the oracle, and the invariants of cuCIM's own ridge
tests (filters/tests/test_ridges.py:18-227: null images, energy decrease,
linearity) on the GPU outputs.

Tolerances. The Hessian passes are bit-exact float32; the eigenvalues are
computed in float64 on the GPU and in numpy, whose transcendental functions
may differ in the last float64 bit, which after rounding to float32 very
rarely moves a value by one ulp. frangi and the hybrid hessian filter must
therefore be bit-identical wherever the output is at least 1e-3 of its
maximum, and within 1e-9 of the maximum elsewhere (the full 256^3 benchmark
volume meets both); float64 results within 1e-12. meijering and sato outputs are compared with a relative
tolerance of 1e-6 (sato's square root is CUDA's powf against the host's
powf, each within 2 ulp)."""

import numpy as np
import pytest
import torch

from oracle import restate as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def filters(cuda):
    from cucim_b200.skimage import filters as f

    return f


def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.cpu().numpy()


def frangi_close(got, exp):
    scale = float(np.abs(exp).max())
    if exp.dtype == np.float64:
        # float64 results carry the last-bit differences of the two exp()s
        np.testing.assert_allclose(got, exp, rtol=1e-12, atol=1e-14 * scale)
        return
    big = np.abs(exp) >= 1e-3 * scale
    np.testing.assert_array_equal(got[big], exp[big])
    assert np.abs(got.astype(np.float64) - exp).max() <= 1e-9 * max(scale, 1e-30)


def segments(shape, seed):
    from cucim_b200 import synthetic

    return synthetic.segments_volume(shape, n_segments=12, seed=seed,
                                     length_range=(8, 30), radius_range=(1.0, 2.5))


@pytest.mark.parametrize("shape,black,sigmas", [((40, 44), True, [1, 2]),
                                                ((18, 20, 22), False, [1, 2]),
                                                ((33, 35, 37), False, [1, 2, 3]),
                                                ((64, 70), False, [1.5, 3.0])])
def test_frangi_matches_oracle(filters, shape, black, sigmas):
    x = segments(shape, 11) if len(shape) == 3 else np.random.default_rng(1).random(shape).astype(np.float32)
    got = host(filters.frangi(dev(x), sigmas=sigmas, black_ridges=black))
    frangi_close(got, R.frangi(x, sigmas=sigmas, black_ridges=black))


@pytest.mark.parametrize("shape", [(40, 44), (18, 20, 22)])
@pytest.mark.parametrize("black", [True, False])
def test_hessian_ridge_matches_oracle(filters, shape, black):
    x = np.random.default_rng(2).random(shape).astype(np.float32)
    got = host(filters.hessian(dev(x), sigmas=[1, 2], black_ridges=black))
    frangi_close(got, R.hessian_ridge(x, sigmas=[1, 2], black_ridges=black))


@pytest.mark.parametrize("name", ["meijering", "sato"])
@pytest.mark.parametrize("shape,mode", [((40, 44), "reflect"), ((18, 20, 22), "reflect"),
                                        ((30, 31), "constant"), ((16, 17, 18), "nearest")])
@pytest.mark.parametrize("black", [True, False])
def test_meijering_sato_match_oracle(filters, name, shape, mode, black):
    x = (segments(shape, 3) if len(shape) == 3
         else np.random.default_rng(3).random(shape).astype(np.float32))
    got = host(getattr(filters, name)(dev(x), sigmas=[1, 2], black_ridges=black, mode=mode))
    exp = getattr(R, name)(x, sigmas=[1, 2], black_ridges=black, mode=mode)
    assert got.dtype == exp.dtype == np.float32
    np.testing.assert_allclose(got, exp, rtol=1e-6, atol=1e-7 * float(np.abs(exp).max()))


def test_ridge_filters_float64(filters):
    x = np.random.default_rng(4).random((24, 26))
    for name, ref in (("meijering", R.meijering), ("sato", R.sato)):
        got = host(getattr(filters, name)(dev(x), sigmas=[1, 2]))
        assert got.dtype == np.float64
        np.testing.assert_allclose(got, ref(x, sigmas=[1, 2]), rtol=1e-12, atol=1e-14)
    frangi_close(host(filters.frangi(dev(x), sigmas=[1, 2])), R.frangi(x, sigmas=[1, 2]))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kw", [{"gamma": 1e-155}, {"alpha": 1e-155}, {"beta": 1e-155},
                                {"gamma": 0.0}, {"alpha": 1e160, "gamma": 1e160}])
def test_frangi_extreme_parameters(filters, dtype, kw):
    """Squares of the parameters whose reciprocals overflow, zero and infinite
    ones: flat regions (r_g = 0) stay 0 and not nan, like the quotients."""
    x = np.zeros((24, 26), dtype)
    x[10:12, 3:20] = 1
    with np.errstate(all="ignore"):
        exp = R.frangi(x, sigmas=[1, 2], black_ridges=False, **kw)
    got = host(filters.frangi(dev(x), sigmas=[1, 2], black_ridges=False, **kw))
    np.testing.assert_array_equal(np.isnan(got), np.isnan(exp))
    np.testing.assert_allclose(got, exp, rtol=1e-6 if dtype == np.float32 else 1e-12, atol=1e-30)


def test_float64_vesselness_keeps_its_precision(cuda):
    """The vesselness of float64 eigenvalues whose squares are exact, with an
    exponent near 10 that makes the quotient's rounding visible: no further from
    the extended-precision value than the same statements in float64 on the host."""
    import ctypes

    from cucim_b200 import _arrays, _lib

    n = 400_000
    l1, l2 = np.random.default_rng(9).integers(900_000, 1_100_000, n) / 2.0 ** 20, np.ones(n)
    beta, gamma = 0.24, 0.01  # gamma: the second factor is 1

    def value(F):
        return np.exp(-(l1.astype(F) ** 2) / F(2 * beta * beta))

    ls = [dev(l1), dev(l2)]
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    elems = (_lib.CimxArray * 2)(*[_arrays.to_cimx(t) for t in ls])
    rc = _lib.lib.cimx_frangi_accumulate(elems, 2, ctypes.byref(_arrays.to_cimx(out)), 0.5,
                                         beta, gamma, 1, None, _arrays.stream_of(out))
    assert rc == 0, _lib.last_error()
    exact = value(np.longdouble)

    def rms(x):
        return float(np.sqrt(np.mean(np.square((x - exact) / exact))))

    assert rms(host(out)) <= 1.1 * rms(value(np.float64))


def test_float64_eigenvalues_keep_their_precision(cuda):
    """Eigenvalues of 3 x 3 float64 matrices v v' + w w' (well conditioned in the
    largest one): no further from the extended-precision value of the closed form
    than its float64 statements are, evaluated one by one on the host. 400 000
    matrices put the sampling error of the rms ratio below 1 %."""
    from cucim_b200.skimage.feature import symmetric_compute_eigenvalues

    v, w = np.random.default_rng(8).standard_normal((2, 3, 400_000))
    # corner.py's element order: 00, 01, 02, 11, 12, 22
    elems = [v[i] * v[j] + w[i] * w[j] for i in range(3) for j in range(i, 3)]

    def largest(F):
        a, d, f, b, e, c = [m.astype(F) for m in elems]
        ta, tb, tc = 2 * a - b - c, 2 * b - a - c, 2 * c - a - b
        x2 = -ta * tb * tc + 9 * (tc * d * d + tb * f * f + ta * e * e) - 54 * (d * e * f)
        x1 = a * a + b * b + c * c - a * b - a * c - b * c + 3 * (d * d + e * e + f * f)
        pi = F(4) * np.arctan(F(1))
        phi = np.arctan(np.sqrt(np.maximum(4 * x1 ** 3 - x2 * x2, 0)) / x2)
        phi = np.where(x2 < 0, phi + pi, phi)
        return (a + b + c) / 3 + F(2) / 3 * np.sqrt(x1) * np.cos((phi - pi) / 3)

    exact = largest(np.longdouble)
    got = host(symmetric_compute_eigenvalues([dev(m) for m in elems]))[0]

    def rms(x):
        return float(np.sqrt(np.mean(np.square((x - exact) / exact))))

    assert np.finfo(np.longdouble).nmant >= 63
    assert rms(got) <= 1.05 * rms(largest(np.float64)), (rms(got), rms(largest(np.float64)))


# ---- the invariants of filters/tests/test_ridges.py:18-227 on the GPU path

def _invert_u8(a):
    return 255 - a


@pytest.mark.parametrize("shape", [(3, 3), (3, 3, 5)])
def test_null_matrix(filters, shape):
    a_black = np.zeros(shape, np.uint8)
    a_white = _invert_u8(a_black)
    zeros, ones = np.zeros(shape), np.ones(shape)
    atol_m = 1e-1 if len(shape) == 3 else 0
    np.testing.assert_allclose(host(filters.meijering(dev(a_black), black_ridges=True)), zeros,
                               atol=atol_m)
    np.testing.assert_allclose(host(filters.meijering(dev(a_white), black_ridges=False)), zeros,
                               atol=atol_m)
    np.testing.assert_array_equal(host(filters.sato(dev(a_black), black_ridges=True,
                                                    mode="reflect")), zeros)
    np.testing.assert_array_equal(host(filters.sato(dev(a_white), black_ridges=False,
                                                    mode="reflect")), zeros)
    np.testing.assert_allclose(host(filters.frangi(dev(a_black), black_ridges=True)), zeros,
                               atol=1e-3)
    np.testing.assert_allclose(host(filters.frangi(dev(a_white), black_ridges=False)), zeros,
                               atol=1e-3)
    np.testing.assert_array_equal(host(filters.hessian(dev(a_black), black_ridges=False,
                                                       mode="reflect")), ones)
    np.testing.assert_array_equal(host(filters.hessian(dev(a_white), black_ridges=True,
                                                       mode="reflect")), ones)


@pytest.mark.parametrize("shape", [(5, 5), (5, 5, 5)])
def test_energy_decrease(filters, shape):
    a_black = np.zeros(shape, np.uint8)
    a_black[(2,) * len(shape)] = 255
    a_white = _invert_u8(a_black)
    for name, kw in (("meijering", {}), ("sato", {"mode": "reflect"}), ("frangi", {}),
                     ("hessian", {"mode": "reflect"})):
        f = getattr(filters, name)
        assert host(f(dev(a_black), black_ridges=True, **kw)).std() < a_black.std(), name
        assert host(f(dev(a_white), black_ridges=False, **kw)).std() < a_white.std(), name


@pytest.mark.parametrize("shape", [(3, 3), (3, 3, 5)])
def test_linearity(filters, shape):
    a_black = np.ones(shape, np.uint8)
    a_white = _invert_u8(a_black)
    for name, kw in (("meijering", {}), ("sato", {"mode": "reflect"}), ("frangi", {}),
                     ("hessian", {"mode": "reflect"})):
        f = getattr(filters, name)
        np.testing.assert_allclose(host(f(dev(1 * a_black), black_ridges=True, **kw)),
                                   host(f(dev(10 * a_black), black_ridges=True, **kw)),
                                   atol=1e-3, err_msg=name)
        np.testing.assert_allclose(host(f(dev(1 * a_white), black_ridges=False, **kw)),
                                   host(f(dev(10 * a_white), black_ridges=False, **kw)),
                                   atol=1e-3, err_msg=name)


@pytest.mark.parametrize("shape", [(36, 41), (14, 17, 19)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("gamma", [None, 0.7])
def test_fused_frangi_epilogue_equals_two_step(filters, shape, dtype, gamma):
    """cimx_frangi_hessian_accumulate (eigenvalues and vesselness in one
    kernel) against cimx_eigvals_sym + cimx_frangi_accumulate, bit for bit,
    over three scales (the first with the automatic gamma goes through
    the eigenvalue images, the others through the fused kernel)."""
    import ctypes

    from cucim_b200 import _arrays, _lib
    from cucim_b200.skimage.feature import _hessian_matrix_with_gaussian

    x = dev(np.random.default_rng(12).random(shape).astype(dtype))
    nd = len(shape)
    g = float("nan") if gamma is None else gamma
    outs = [torch.empty_like(x), torch.empty_like(x)]
    states = [torch.zeros(2, dtype=torch.int64, device="cuda") for _ in range(2)]
    for i, sigma in enumerate([1.0, 2.0, 3.0]):
        H = [h.contiguous() for h in _hessian_matrix_with_gaussian(x, sigma)]
        hs = (_lib.CimxArray * len(H))(*[_arrays.to_cimx(h) for h in H])
        a0 = _arrays.to_cimx(outs[0])
        assert _lib.lib.cimx_frangi_hessian_accumulate(
            hs, len(H), ctypes.byref(a0), 0.5, 0.5, g, int(i == 0),
            ctypes.c_void_p(states[0].data_ptr()), None) == 0, _lib.last_error()
        ev = torch.empty((nd,) + tuple(shape), dtype=x.dtype, device="cuda")
        evs = (_lib.CimxArray * nd)(*[_arrays.to_cimx(ev[k]) for k in range(nd)])
        assert _lib.lib.cimx_eigvals_sym(hs, len(H), evs, 0, 1, None) == 0
        a1 = _arrays.to_cimx(outs[1])
        assert _lib.lib.cimx_frangi_accumulate(evs, nd, ctypes.byref(a1), 0.5, 0.5, g,
                                               int(i == 0),
                                               ctypes.c_void_p(states[1].data_ptr()),
                                               None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(host(outs[0]), host(outs[1]))
