"""The strip and column kernels (csrc/cimx_strip.cuh) against the oracle, bit
for bit, where their geometry changes: around a group of 8 rows, a tile's
columns, the tap-count bounds, unequal and partly zero taps, odd row lengths
and base addresses, axes shorter than the taps."""

import numpy as np
import pytest
import torch

from oracle import restate as R

pytestmark = pytest.mark.gpu

MODES = ["reflect", "mirror", "nearest", "constant", "wrap"]
PAIRS = [("float32", "float32"), ("uint16", "float32"), ("uint16", "uint16"),
         ("uint8", "float32"), ("uint8", "uint8"), ("uint8", "uint16")]


@pytest.fixture(scope="module")
def ndi(cuda):
    from cucim_b200 import ndimage

    return ndimage


def _data(shape, dtype, seed=0):
    r = np.random.default_rng(seed)
    if dtype == "float32":
        return r.standard_normal(shape).astype(np.float32)
    return r.integers(0, np.iinfo(dtype).max + 1, shape).astype(dtype)


def _taps(K, kind, seed=0):
    """plain: positive, sum 1; signed: any sign, sum of magnitudes 2 (integer
    outputs wrap or saturate); centre / holes: zeros the skip rule leaves out."""
    w = np.random.default_rng(seed + K).random(K) + 0.1
    if kind == "signed":
        w *= np.where(np.arange(K) % 3, 1, -1) * 2
    w /= np.abs(w).sum() / (2 if kind == "signed" else 1)
    if kind == "centre":
        w[K // 2] = 0
    if kind == "holes":
        w[1::3] = 0
    return w


def _run(ndi, x, passes, output, **kw):
    """The passes as one call of the library, and one by one in the oracle."""
    xd = torch.as_tensor(x).cuda()
    got = ndi._run(xd, [(ax, w, m, o, False) for ax, w, m, o in passes], np.dtype(output),
                   kw.get("cval", 0.0))
    exp = x
    for ax, w, m, o in passes:
        exp = R.correlate1d(exp, w, ax, output=np.dtype(output), mode=m, origin=o,
                            cval=kw.get("cval", 0.0))
    np.testing.assert_array_equal(got.cpu().numpy(), exp)


@pytest.mark.parametrize("pair", PAIRS, ids=lambda p: "-".join(p))
@pytest.mark.parametrize("K", [2, 5, 6, 9, 10, 13, 17, 18, 25, 32, 33, 34, 41, 57, 65])
def test_tap_bounds(ndi, pair, K):
    """Both tail passes (fused or apart) and each alone, at every tap bound."""
    x = _data((2, 37, 75), pair[0], K)
    for kind in ("plain", "signed"):
        w = _taps(K, kind)
        for mode in ("reflect", "constant"):
            _run(ndi, x, [(1, w, mode, 0), (2, w, mode, 0)], pair[1], cval=3.0)
            _run(ndi, x, [(1, w, mode, 0)], pair[1], cval=3.0)
            _run(ndi, x, [(2, w, mode, 0)], pair[1], cval=3.0)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("ky,kx", [(1, 9), (9, 3), (17, 5), (8, 17), (33, 9), (18, 33), (65, 21)])
def test_unequal_and_zero_taps(ndi, mode, ky, kx):
    """Unequal counts, a zero centre tap and zeros between taps, with values
    that make a skipped tap matter, origins and a fill value."""
    x = _data((3, 30, 53), "float32", ky)
    x[0, 5, 7], x[1, 20, 50], x[2, 0, 0] = np.inf, np.nan, -np.inf
    for kind in ("plain", "centre", "holes"):
        wy, wx = _taps(ky, kind), _taps(kx, kind)
        if not (wy.any() and wx.any()):
            continue
        _run(ndi, x, [(1, wy, mode, 0), (2, wx, mode, 0)], "float32", cval=1.5)
        _run(ndi, x, [(1, wy, mode, (ky - 1) // 2), (2, wx, mode, -(kx // 2))], "float32",
             cval=np.inf if mode == "constant" else 0.0)
        _run(ndi, x, [(0, wx, mode, 0)], "float32", cval=-2.0)


@pytest.mark.parametrize("rows", [1, 3, 7, 8, 9, 16, 23])
@pytest.mark.parametrize("cols", [1, 2, 31, 32, 112, 113, 496, 497, 504, 1021])
def test_tile_edges(ndi, rows, cols):
    """Rows around the group of 8, columns around the tile widths; 17 taps
    are longer than the short axes, whose halo folds more than once."""
    w = _taps(17, "plain")
    for mode in MODES:
        x = _data((2, rows, cols), "float32", rows * cols)
        _run(ndi, x, [(1, w, mode, 0), (2, w, mode, 0)], "float32", cval=2.0)
    x = _data((2, rows, cols), "uint16", rows * cols)
    _run(ndi, x, [(1, w, "mirror", 0), (2, w, "wrap", 0)], "uint16")
    _run(ndi, x, [(0, w[:5], "reflect", 0), (2, w, "nearest", 0)], "uint16")


@pytest.mark.parametrize("pair", PAIRS, ids=lambda p: "-".join(p))
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 6, 7, 8])
def test_short_slabs(ndi, pair, rows):
    """Slabs of up to 8 rows with up to 5 taps share groups of rows: whole slabs
    per group, slab counts around it, axes shorter than the taps."""
    for count in (1, 2, 8 // rows, 8 // rows + 1, 37):
        for cols in (3, 70, 253, 600):
            x = _data((count, rows, cols), pair[0], count + cols)
            if pair[0] == "float32":
                x[0, 0, 1], x[-1, -1, 2] = np.inf, np.nan
            for ky, kx, kind in ((3, 5, "plain"), (5, 3, "signed"), (4, 2, "plain"),
                                 (3, 3, "centre"), (1, 5, "plain")):
                wy, wx = _taps(ky, kind if ky > 1 else "plain"), _taps(kx, kind)
                mode = MODES[(ky + kx + cols + count) % 5]
                _run(ndi, x, [(1, wy, mode, 0), (2, wx, "reflect", 0)], pair[1], cval=2.0)
                _run(ndi, x, [(1, wy, "constant", (ky - 1) // 2), (2, wx, mode, -(kx // 2))],
                     pair[1], cval=7.0)
    x = _data((4000, rows, 90), pair[0], rows)  # several groups per chunk
    for mode in MODES:
        _run(ndi, x, [(1, _taps(5, "plain"), mode, 0), (2, _taps(3, "plain"), mode, 0)], pair[1],
             cval=1.0)


@pytest.mark.parametrize("pair", PAIRS, ids=lambda p: "-".join(p))
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_base_alignment(ndi, pair, offset):
    """Contiguous arrays whose first element lies off the vector boundary."""
    shape, w = (4, 19, 64), _taps(9, "plain")
    n = int(np.prod(shape))
    flat = _data(n + 4, pair[0], offset)
    x = flat[offset:offset + n].reshape(shape)
    xd = torch.as_tensor(flat).cuda()[offset:offset + n].view(shape)
    out = torch.empty(n + 4, dtype=ndi._arrays.torch_dtype(np.dtype(pair[1])),
                      device="cuda")[4 - offset:n + 4 - offset].view(shape)
    exp = x
    for ax in (1, 2):
        exp = R.correlate1d(exp, w, ax, output=np.dtype(pair[1]), mode="reflect")
    ndi._run(xd, [(1, w, "reflect", 0, False), (2, w, "reflect", 0, False)], out, 0.0)
    np.testing.assert_array_equal(out.cpu().numpy(), exp)


def test_long_tail_passes_without_scratch_memory(ndi):
    """Tail passes that run faster apart take scratch memory; where there is none
    they run as one launch all the same."""
    import ctypes

    from cucim_b200 import _lib

    fn = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p, ctypes.c_void_p)
    rel = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p,
                           ctypes.c_void_p)
    refuse, ignore = fn(lambda *a: None), rel(lambda *a: None)
    set_allocator = _lib.lib.cimx_set_allocator
    set_allocator(ctypes.cast(refuse, ctypes.c_void_p), ctypes.cast(ignore, ctypes.c_void_p), None)
    try:
        for ky, kx in ((57, 57), (33, 9), (64, 33)):
            _run(ndi, _data((3, 40, 70), "float32"),
                 [(1, _taps(ky, "centre"), "reflect", 0), (2, _taps(kx, "holes"), "wrap", 0)],
                 "float32")
        x = np.random.default_rng(1).standard_normal((700, 12, 64))
        w = _taps(33, "plain")
        _run(ndi, x, [(1, w, "reflect", 0), (2, w, "wrap", 0)], "float64")
    finally:
        set_allocator(None, None, None)


@pytest.mark.parametrize("K", [22, 25, 26, 57, 66, 73, 74, 97, 128, 129, 130])
@pytest.mark.parametrize("shape", [(150, 70), (64, 321), (41, 129), (257, 33), (300, 64),
                                   (63, 32), (64, 32)])
def test_long_passes(ndi, K, shape):
    """Long passes each in a launch of their own (cimx_ring.cuh along a strided
    axis), around its step of 64 rows, 64 columns and the tap bounds."""
    x = _data(shape, "float32", K)
    x[3, 5], x[20, 30], x[40, 11] = np.inf, np.nan, -np.inf
    for i, kind in enumerate(("plain", "centre", "holes")):
        w = _taps(K, kind)
        for mode in MODES[i % 2::2]:
            for ax in (0, 1):
                _run(ndi, x, [(ax, w, mode, 0)], "float32", cval=2.5)
        _run(ndi, x, [(0, w, MODES[i], (K - 1) // 2), (1, w, MODES[4 - i], -(K // 2))],
             "float32", cval=np.inf if i == 1 else 0.5)
    flat = _data(shape[0] * shape[1] + 1, "float32", K)  # off the vector boundary
    xd = torch.as_tensor(flat).cuda()[1:].view(shape)
    got = ndi.correlate1d(xd, w, axis=0).cpu().numpy()
    np.testing.assert_array_equal(got, R.correlate1d(flat[1:].reshape(shape), w, 0))


@pytest.mark.parametrize("K", [1, 3, 9, 10, 17, 18, 25, 33, 41, 42, 49, 50])
@pytest.mark.parametrize("shape", [(8, 32), (17, 33), (2, 31, 207), (70, 257), (9, 700)])
def test_float64_tail_passes(ndi, K, shape):
    """Both tail passes of a float64 array in one launch (cimx_strip_f64.cu),
    around its groups of 8 rows, 32 and 256 columns and the tap bounds."""
    x = np.random.default_rng(K).standard_normal(shape)
    x[..., 2, 5], x[..., 6, 20] = np.inf, np.nan
    y, nd = x[..., ::-1].copy(), x.ndim
    w, v = _taps(K, "plain"), _taps(max(K - 1, 1), "signed")
    for mode in MODES:
        _run(ndi, x, [(nd - 2, w, mode, 0), (nd - 1, w, mode, 0)], "float64", cval=1.25)
        _run(ndi, y, [(nd - 2, v, mode, (v.size - 1) // 2), (nd - 1, w, mode, -(K // 2))],
             "float64", cval=np.inf)


@pytest.mark.parametrize("K", [25, 33, 49])
@pytest.mark.parametrize("shape", [(700, 12, 63), (300, 12, 256), (20, 256, 127), (40, 65, 480)])
def test_float64_tail_passes_large(ndi, K, shape):
    """Larger float64 arrays on both sides of the rule between the strip and the
    generic kernels."""
    x = np.random.default_rng(K).standard_normal(shape)
    w = _taps(K, "plain")
    for mode in ("mirror", "constant"):
        _run(ndi, x, [(1, w, mode, 0), (2, w, mode, 0)], "float64", cval=-0.5)


def test_column_pass_along_sixty_million_samples(ndi):
    """More rows than a grid's y extent has short chunks for: compared with the
    oracle at both ends and in the middle."""
    K, n = 45, 62_000_000
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randint(0, 256, (n, 32), device="cuda", generator=g, dtype=torch.uint8)
    w = _taps(K, "plain")
    got = ndi.correlate1d(x, w, 0, mode="reflect")
    for lo in (0, n // 2, n - 3000):
        part = R.correlate1d(x[lo:lo + 3000].cpu().numpy(), w, 0, mode="reflect")
        a = 0 if lo == 0 else K
        b = 3000 if lo == n - 3000 else 3000 - K
        np.testing.assert_array_equal(got[lo + a:lo + b].cpu().numpy(), part[a:b])


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("shape", [(1, 41, 34), (3, 7, 66), (2, 200, 258), (300, 9, 32)])
def test_column_pairs(ndi, dtype, shape):
    """Up to 5 taps of 8- and 16-bit values to float32 along strided axes, two
    columns per thread on aligned pairs and one elsewhere."""
    n = int(np.prod(shape))
    for off_in, off_out in ((0, 0), (1, 0), (0, 1), (2, 2)):
        flat = _data(n + 2, dtype, n + off_in)
        x, xd = flat[off_in:off_in + n].reshape(shape), torch.as_tensor(flat).cuda()
        xd = xd[off_in:off_in + n].view(shape)
        out = torch.empty(n + 2, device="cuda")[off_out:off_out + n].view(shape)
        for K, kind in ((1, "plain"), (2, "signed"), (3, "centre"), (4, "plain"), (5, "signed")):
            w = _taps(K, kind)
            for mode in MODES:
                for ax in (0, 1):
                    ndi.correlate1d(xd, w, ax, out, mode, 3.0, origin=-((K - 1) // 2))
                    exp = R.correlate1d(x, w, ax, output=np.dtype(np.float32), mode=mode,
                                        origin=-((K - 1) // 2), cval=3.0)
                    np.testing.assert_array_equal(out.cpu().numpy(), exp)
