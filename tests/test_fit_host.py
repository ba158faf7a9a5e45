"""The device fit code compiled for the host (tests/host/fit_host.cc)
against the oracle: the FP64 kernels' arithmetic restates the reference
operation by operation, so on the host, where both use the same math
library, the two agree to the last bit.  On the device only the
transcendental functions differ (tests/test_gpu_riemann.py, test_gpu_parity.py).  The
mixed-precision Riemann fit is checked for finite results on tuples where
single-precision intermediates used to cancel."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

import oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEYS = ("state", "cov", "pt", "eta", "chi2")


@pytest.fixture(scope="module")
def host_lib():
    out = os.path.join(tempfile.mkdtemp(), "libfithost.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "pixeltrack-standalone_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "fit_host.cc"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    for f in (lib.hf_fit_riemann, lib.hf_fit_broken_line):
        f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_uint32] + [ctypes.c_void_p] * 2 + \
            [ctypes.c_double] + [ctypes.c_void_p] * 5
    lib.hf_chain_tile.argtypes = [ctypes.c_int] + [ctypes.c_uint32] * 2 + [ctypes.c_void_p]
    lib.hf_chain_tile.restype = ctypes.c_uint32
    return lib


def host_fit(lib, N, hits, ge, mixed, algo="riemann"):
    n = hits.shape[0]
    h = np.ascontiguousarray(hits[:, :N, :], dtype=np.float64)
    g = np.ascontiguousarray(ge[:, :N, :], dtype=np.float32)
    out = {"state": np.zeros((n, 5), np.float32), "cov": np.zeros((n, 15), np.float32),
           "pt": np.zeros(n, np.float32), "eta": np.zeros(n, np.float32), "chi2": np.zeros(n, np.float32)}
    assert getattr(lib, "hf_fit_" + algo)(N, int(mixed), n, h.ctypes.data, g.ctypes.data, 0.0114256972711507,
                                          *[out[k].ctypes.data for k in KEYS]) == 0
    return out


def check_equal(got, want):
    for k in KEYS:
        a, b = got[k], want[k]
        assert np.all((a == b) | (np.isnan(a) & np.isnan(b))), k


@pytest.mark.parametrize("nh,N", [(3, 3), (4, 4), (5, 4)])
def test_device_riemann_arithmetic_equals_oracle(host_lib, default_detector, nh, N):
    import pixgpu
    hits, ge, _ = pixgpu.fit_tuples(51 + nh, 20000, nh)
    check_equal(host_fit(host_lib, N, hits, ge, False),
                oracle.Oracle(default_detector.es).fit(N, hits, ge, riemann=True))


@pytest.mark.parametrize("nh,N", [(3, 3), (4, 4), (5, 4)])
def test_device_broken_line_arithmetic_equals_oracle(host_lib, default_detector, nh, N):
    import pixgpu
    hits, ge, _ = pixgpu.fit_tuples(51 + nh, 20000, nh)
    check_equal(host_fit(host_lib, N, hits, ge, False, "broken_line"),
                oracle.Oracle(default_detector.es).fit(N, hits, ge))


def special_tuples(N):
    """Tuples with one element of a hit or of its covariance replaced by an
    infinite, NaN, zero or huge value: 20 of each."""
    import pixgpu
    hits, ge, _ = pixgpu.fit_tuples(61 + N, 20, N)
    hs, gs = [], []
    with np.errstate(over="ignore"):
        for value in (np.inf, -np.inf, np.nan, 0.0, 1e20, -1e38):
            for i in range(N):
                for k in range(9):
                    h, g = hits.copy(), ge.copy()
                    if k < 3:
                        h[:, i, k] = value
                    else:
                        g[:, i, k - 3] = value
                    hs.append(h)
                    gs.append(g)
    return np.concatenate(hs), np.concatenate(gs)


@pytest.mark.parametrize("N", [3, 4])
@pytest.mark.parametrize("algo", ["broken_line", "riemann"])
def test_device_fit_of_special_values_equals_oracle(host_lib, default_detector, algo, N):
    """Where a fit's matrices have constant zeros whose products the kernels
    leave out, an infinite or NaN factor still makes the result NaN."""
    hits, ge = special_tuples(N)
    check_equal(host_fit(host_lib, N, hits, ge, False, algo),
                oracle.Oracle(default_detector.es).fit(N, hits, ge, riemann=algo == "riemann"))


def grid_covariances(n, N):
    ge = np.zeros((n, N, 6), np.float32)
    ge[:, :, [0, 2, 5]] = 1e-4
    return ge


@pytest.mark.parametrize("N", [3, 4])
def test_device_broken_line_on_a_small_grid_equals_oracle(host_lib, default_detector, N):
    """Hits on integer points: equal hits, straight lines, and chords that
    equal the circle's diameter, where the reference's Jacobian is 0 / 0."""
    hits = np.random.default_rng(1).integers(-2, 3, (20000, N, 3)).astype(np.float64)
    ge = grid_covariances(len(hits), N)
    want = oracle.Oracle(default_detector.es).fit(N, hits, ge)
    assert (np.isfinite(want["state"]).all(1) & np.isnan(want["cov"][:, 0])).sum() >= 10
    check_equal(host_fit(host_lib, N, hits, ge, False, "broken_line"), want)


@pytest.mark.parametrize("hits", [[[-1, 1, 2], [2, -1, -2], [2, 1, 1]],
                                  [[1, 1, 1], [-2, 2, 1], [0, 0, 0], [-1, 0, 1]]])
def test_mixed_broken_line_with_a_chord_of_the_diameter(host_lib, hits):
    """The covariance of a track whose chord equals the diameter in single
    precision is NaN as in the FP64 fit, its state finite."""
    got = host_fit(host_lib, len(hits), np.array([hits], np.float64), grid_covariances(1, len(hits)), True,
                   "broken_line")
    assert np.isfinite(got["state"]).all() and np.isnan(got["cov"][0, [0, 1, 2, 5, 6, 9]]).all()


@pytest.mark.parametrize("nh,N,index", [(3, 3, 139459), (5, 4, 102442), (5, 4, 126818)])
def test_mixed_riemann_stays_finite_where_single_precision_cancels(host_lib, nh, N, index):
    """Tuples of the seeded sets of the mixed-precision test whose radial hit
    variance cancels to ~1e-16 in double precision (0 in single precision)."""
    import pixgpu
    hits, ge, _ = pixgpu.fit_tuples(4242 + nh, index + 1, nh)
    got = host_fit(host_lib, N, hits[index:], ge[index:], True)
    assert np.isfinite(got["state"]).all() and np.isfinite(got["pt"]).all()


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_a_thread_of_the_chain_fits_writes_only_its_own_inputs(host_lib, threads):
    """The warps of a block may be at different tiles, one at 4-hit tuples
    while the next is at 3-hit ones: no byte that a thread fills for one width
    is another thread's for either width, and all lie in the block's memory."""
    owner = None
    for N in (3, 4):
        for t in range(threads):
            r = (ctypes.c_uint32 * 4)()
            size = host_lib.hf_chain_tile(N, t, threads, r)
            if owner is None:
                owner = np.full(size, -1)
            for a, b in ((r[0], r[1]), (r[2], r[3])):
                assert a < b <= size and a % 4 == 0
                assert np.isin(owner[a:b], (-1, t)).all(), (N, t)
                owner[a:b] = t
