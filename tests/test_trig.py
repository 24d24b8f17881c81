"""The fixed-point sine and cosine (networkdynamics.jl_gb300/csrc/nd_trig.cuh) and the integer
division (nd_exact.cuh) of the FP64 kernels against extended precision and IEEE-754 division on the
host, and the device build against the host build, bit for bit."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "networkdynamics.jl_gb300" / "csrc"
NATIVE = Path(__file__).resolve().parent / "native"


@pytest.fixture(scope="module")
def host():
    out = NATIVE / "_build" / "libtrig_host.so"
    out.parent.mkdir(exist_ok=True)
    src = NATIVE / "trig_host.cpp"
    deps = [src, CSRC / "nd_trig.cuh", CSRC / "nd_exact.cuh"]
    if not out.exists() or out.stat().st_mtime < max(d.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", f"-I{CSRC}", str(src),
                        "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    lib.nd_trig_host.argtypes = [C.c_void_p] * 3 + [C.c_int64]
    lib.nd_trig_times_host.argtypes = [C.c_void_p] * 4 + [C.c_int64]
    lib.nd_exact_div_host.argtypes = [C.c_void_p] * 3 + [C.c_int64]

    def run(x, f=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        s, c = np.empty_like(x), np.empty_like(x)
        if f is None:
            lib.nd_trig_host(x.ctypes.data, s.ctypes.data, c.ctypes.data, x.size)
        else:
            lib.nd_trig_times_host(f.ctypes.data, x.ctypes.data, s.ctypes.data, c.ctypes.data, x.size)
        return s, c

    def div(a, b):
        out = np.empty_like(a)
        lib.nd_exact_div_host(a.ctypes.data, b.ctypes.data, out.ctypes.data, a.size)
        return out
    run.div = div
    return run


def factors(n, seed):
    """Line weights of every size, zeros and the ends of the exponent range."""
    rng = np.random.default_rng(seed)
    f = rng.uniform(5, 10, n) * 10.0 ** rng.choice([0, 0, 0, -5, 5], n) * rng.choice([1.0, -1.0], n)
    f[:8] = [0.0, -0.0, 5e-324, 1e-300, 1e308, np.inf, np.nan, 1.0]
    return f


def quotients(n, seed):
    """Operands of ordinary size, any bit pattern, powers of two, and quotients next to a
    halfway point (a = RN(b (q + 1/2 ulp)))."""
    rng = np.random.default_rng(seed)
    bits = lambda: rng.integers(0, 2 ** 64, n, dtype=np.uint64).view(np.float64)  # noqa: E731
    b, q = rng.uniform(0.5, 2, n), rng.uniform(0.5, 2, n)
    yield rng.normal(size=n), rng.normal(size=n) * 10.0 ** rng.integers(-20, 20, n)
    yield bits(), bits()
    yield np.ones(n), rng.integers(1, 1 << 53, n).astype(np.float64)
    yield 2.0 ** rng.integers(-1074, 1024, n), 2.0 ** rng.integers(-1074, 1024, n)
    yield (b.astype(np.longdouble) * (q.astype(np.longdouble) + np.spacing(q) / 2)).astype(np.float64), b
    z = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 1.7976931348623157e308, 2.2250738585072014e-308])
    a, b = np.meshgrid(z, z)
    yield a.ravel().copy(), b.ravel().copy()


def same_bits(a, b):
    return np.all((a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b)))


def test_host_division_matches_ieee(host):
    with np.errstate(all="ignore"):
        for a, b in quotients(400_000, 3):
            assert same_bits(host.div(a, b), a / b)


def arguments(n, seed=0):
    """Phase differences of every size, the neighbours of the multiples of π/2 (where the
    reduction cancels) and the edges of the fixed-point range (2^-27, 2^17)."""
    rng = np.random.default_rng(seed)
    k = rng.integers(1, 83000, n // 8)
    near = k * np.longdouble("1.5707963267948966192313216916397514421")
    near = near.astype(np.float64)
    edges = np.concatenate([2.0 ** np.arange(-40, 20), np.nextafter(2.0 ** np.arange(-40, 20), 0.0)])
    x = np.concatenate([rng.uniform(-np.pi, np.pi, n // 2), rng.normal(scale=1e3, size=n // 8),
                        2.0 ** rng.uniform(-40, 17, n // 4), near, near * (1 + 10.0 ** rng.uniform(-15, -3, k.size)),
                        edges])
    return x * rng.choice([-1.0, 1.0], x.size)


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="needs an extended-precision long double")
def test_host_error_below_051_ulp(host):
    """0.5 ulp of the one rounding plus under 0.01 of the fixed-point errors (V and r are
    within 2^-61 of their values, 2^-8 ulp each)."""
    x = arguments(800_000)
    s, c = host(x)
    xl = x.astype(np.longdouble)
    for got, ref in ((s, np.sin(xl)), (c, np.cos(xl))):
        ulp = np.spacing(np.abs(ref.astype(np.float64)))
        assert float(np.max(np.abs(got.astype(np.longdouble) - ref) / ulp)) <= 0.51
    # the products: once more 2^-61 (the library's and tiny arguments take the plain product)
    f = factors(x.size, 1)[8:]
    x = x[8:]
    xl, fl = x.astype(np.longdouble), f.astype(np.longdouble)
    half_pi = np.longdouble("1.5707963267948966192313216916397514421")
    k = np.rint(xl / half_pi)
    plain = (np.abs(x) >= 2.0 ** 17) | (np.abs(x) < 2.0 ** -27) | ((np.abs(xl - k * half_pi) < 2.0 ** -17) & (k != 0))
    for got, ref in zip(host(x, f), (fl * np.sin(xl), fl * np.cos(xl))):
        err = np.abs(got.astype(np.longdouble) - ref) / np.spacing(np.abs(ref.astype(np.float64)))
        assert float(np.max(err[~plain])) <= 0.51


def test_host_symmetry_and_special_values(host):
    x = arguments(100_000, seed=1)
    s, c = host(x)
    sn, cn = host(-x)
    assert np.array_equal(sn, -s) and np.array_equal(cn, c)
    f = factors(x.size, 2)
    with np.errstate(all="ignore"):
        for got, ref in zip(host(x[:8], f[:8].copy()), (f[:8] * np.sin(x[:8]), f[:8] * np.cos(x[:8]))):
            np.testing.assert_allclose(got, ref, rtol=2.0 ** -51, atol=5e-324)
    s, c = host([0.0, -0.0, 5e-324, -2.0 ** -1030, np.inf, -np.inf, np.nan])
    assert np.array_equal(s[:4], [0.0, -0.0, 5e-324, -2.0 ** -1030]) and np.signbit(s[1]) and not np.signbit(s[0])
    assert np.array_equal(c[:4], np.ones(4)) and np.isnan(s[4:]).all() and np.isnan(c[4:]).all()


@pytest.mark.gpu
def test_device_matches_host(host, cuda):
    """The device build gives the host build's bits wherever neither calls the library
    function, and the library's accuracy (1 ulp, both sides) where they do."""
    import torch
    from nd_gb300 import _capi as capi
    x = arguments(400_000, seed=2)
    xt = torch.from_numpy(x).to(cuda)
    st, ct = torch.empty_like(xt), torch.empty_like(xt)
    lib = capi.load()
    capi.check(lib.nd_selftest_trig(xt.data_ptr(), st.data_ptr(), ct.data_ptr(), x.size,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    half_pi = np.longdouble("1.5707963267948966192313216916397514421")
    k = np.rint(x.astype(np.longdouble) / half_pi)
    library = (np.abs(x) >= 2.0 ** 17) | ((np.abs(x - k * half_pi) < 2.0 ** -17) & (k != 0))
    for got, ref in zip((st.cpu().numpy(), ct.cpu().numpy()), host(x)):
        np.testing.assert_array_equal(got[~library], ref[~library])
        assert np.all(np.abs(got - ref)[library] <= 2 * np.spacing(np.abs(ref[library])))
    for a, b in quotients(400_000, 4):
        at, bt = torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda)
        qt = torch.empty_like(at)
        capi.check(lib.nd_selftest_exact_div(at.data_ptr(), bt.data_ptr(), qt.data_ptr(), a.size,
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        with np.errstate(all="ignore"):
            assert same_bits(qt.cpu().numpy(), a / b)
    sm = torch.empty_like(xt)
    capi.check(lib.nd_selftest_trig((-xt).data_ptr(), sm.data_ptr(), ct.data_ptr(), x.size,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(sm, -st)
