"""The fixed-point pair arithmetic (csrc/gmi_pairs_fx.cuh) against the FP64
oracle, on the host: the formulas are plain C++ on integers and floats there and on
the GPU.

Tolerance: a term of the fixed-point sum is rounded at about 2^-55 of its load,
so the difference is the oracle's own, whose sums of n FP64 terms are each
within n 2^-53 of the terms' size; n 2^-52 of the largest velocity is allowed.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT, rel_err

KINDS = {"ss": 0, "bb": 2, "sb": 3, "bs": 4}


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fx") / "fx_host.so")
    csrc = os.path.join(ROOT, "generic_mobility_interface_class_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-x", "c++", "-I", csrc,
                    os.path.join(ROOT, "tests", "fx_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    d, p = ctypes.c_double, ctypes.c_void_p
    lib.fx_host_sum.argtypes = [ctypes.c_int, ctypes.c_int, p, ctypes.c_int, p, p, d, d, d, p]
    return lib


def fx_sum(lib, kind, xt, xs, f, a, b, mu=1.0):
    xt, xs, f = (np.ascontiguousarray(v) for v in (xt, xs, f))
    out = np.zeros((len(xt), 6 if kind in ("ss", "sb") else 3))
    status = lib.fx_host_sum(KINDS[kind], len(xt), xt.ctypes.data, len(xs), xs.ctypes.data, f.ctypes.data, a, b, mu,
                             out.ctypes.data)
    return status, out


def oracle_sum(rpy, kind, xt, xs, f, a, b, mu=1.0):
    if kind == "ss":
        return rpy.mss(xs, f, a, mu)
    if kind == "bb":
        return rpy.mbb(xs, f, a, mu)
    if kind == "sb":
        return rpy.msb(xt, xs, f, a, b, mu)
    return rpy.mbs(xt, xs, f, a, b, mu)


def in_range(xt, xs, radius):
    """Positions lie within 512 U of the first source rounded to 256 U, U the
    largest power of two not above the radius."""
    u = 2.0 ** np.floor(np.log2(radius))
    origin = np.rint(xs[0] / (256 * u)) * (256 * u)
    return max(np.abs(xt - origin).max(), np.abs(xs - origin).max()) < 512 * u


def cloud(kind, layout, n, a, seed):
    rng = np.random.default_rng(seed)
    size = {"far": 100.0, "dense": 3.0, "wide": 250.0, "near_copies": 20.0}[layout] * a
    xs = rng.uniform(-size, size, size=(n, 3))
    if layout == "near_copies":  # coincident particles, and pairs 2^-1 .. 2^-58 radii apart
        for i in range(0, n - 1, 3):
            xs[i + 1] = xs[i] + a * np.ldexp(rng.normal(size=3), -(i % 58)) * (i % 9 > 0)
    f = rng.normal(size=(n, 6 if kind in ("ss", "bs") else 3))
    xt = xs if kind in ("ss", "bb") else np.concatenate([xs[:20], rng.uniform(-size, size, size=(30, 3))])
    return xt, xs, f


@pytest.mark.parametrize("layout", ["far", "dense", "wide", "near_copies"])
@pytest.mark.parametrize("kind,a,b", [("ss", 1.0, 1.0), ("ss", 1.999, 1.999), ("ss", 1e-3, 1e-3), ("bb", 1.0, 1.0),
                                      ("bb", 0.75, 0.75), ("sb", 1.0, 1.0), ("sb", 1.0, 2.0), ("sb", 1.3, 0.7),
                                      ("bs", 1.0, 1.0), ("bs", 0.5, 1.0), ("bs", 1.0, 0.6)])
def test_fixed_point_sums_against_oracle(host, oracle_built, kind, a, b, layout):
    n = 333
    xt, xs, f = cloud(kind, layout, n, max(a, b), seed=5)
    status, got = fx_sum(host, kind, xt, xs, f, a, b, mu=1.7)
    if not in_range(xt, xs, min(a, b)):
        assert status == 2
        return
    assert status == 0
    want = oracle_sum(oracle_built, kind, xt, xs, f, a, b, 1.7)
    for block in range(0, want.shape[1], 3):
        assert rel_err(got[:, block:block + 3], want[:, block:block + 3]) < n * 2.0 ** -52


@pytest.mark.parametrize("kind", ["sb", "bs"])
@pytest.mark.parametrize("small", [1.0, 1.42, 1.89, 1.95, 1.999, 0.95])
@pytest.mark.parametrize("ratio", [1.5, 1.8, 2.0])
@pytest.mark.parametrize("swap", [False, True])
def test_near_field_limit_of_unequal_radii(host, oracle_built, kind, small, ratio, swap):
    """Overlapping particles over the whole range of radii held: the limit of
    the near field, ((a + b) / U)^2, reaches 36."""
    a, b = (small, ratio * small)[::-1] if swap else (small, ratio * small)
    n = 300
    xt, xs, f = cloud(kind, "dense", n, small, seed=12)
    status, got = fx_sum(host, kind, xt, xs, f, a, b)
    assert status == 0
    want = oracle_sum(oracle_built, kind, xt, xs, f, a, b)
    for block in range(0, want.shape[1], 3):
        assert rel_err(got[:, block:block + 3], want[:, block:block + 3]) < n * 2.0 ** -52


@pytest.mark.parametrize("kind", ["ss", "bb"])
def test_loads_of_very_different_sizes(host, oracle_built, kind):
    """Loads from 1e-9 to 1e9 in one tile, zero loads, and a whole tile of zeros."""
    n = 400
    xt, xs, f = cloud(kind, "far", n, 1.0, seed=6)
    f *= 10.0 ** np.random.default_rng(7).uniform(-9, 9, size=(n, 1))
    f[5] = 0.0
    f[128:256] = 0.0
    status, got = fx_sum(host, kind, xt, xs, f, 1.0, 1.0)
    assert status == 0
    assert rel_err(got, oracle_sum(oracle_built, kind, xt, xs, f, 1.0, 1.0)) < n * 2.0 ** -52


def extended_sum(kind, xt, xs, f):
    """The sums at radii and viscosity 1 in extended precision, and for each
    target the sum of its terms' sizes (|coefficient| |load|, v and w)."""
    R = np.longdouble
    xt, xs, f = xt.astype(R), xs.astype(R), f.astype(R)
    d = xt[:, None] - xs[None]
    r = np.sqrt((d * d).sum(-1))
    s = np.where(r > 0, r, R(1))
    e = d / s[..., None]
    F, T = f[None, :, :3], f[None, :, 3:] if f.shape[1] == 6 else np.zeros((1, len(f), 3), R)
    k8 = 1 / (8 * R("3.14159265358979323846264338327950288"))
    far = r > 2
    A = np.where(far, k8 / s * (1 + 2 / (3 * s * s)), k8 * (R(4) / 3 - 3 * r / 8))
    B = np.where(far, k8 / s * (1 - 2 / (s * s)), k8 * r / 8)
    Ar = np.where(far, -k8 / (2 * s ** 3), k8 * (1 - 27 * r / 32 + 5 * r ** 3 / 64))
    Br = np.where(far, 3 * k8 / (2 * s ** 3), k8 * (9 * r / 32 - 3 * r ** 3 / 64))
    C = np.where(far, k8 / (s * s), k8 * r / 2 * (1 - 3 * r / 8))
    A, B, Ar, Br, C = (c[..., None] for c in (A, B, Ar, Br, C))
    cross = lambda p, q: np.cross(np.broadcast_to(p, d.shape), q)
    dot = lambda p: (e * p).sum(-1)[..., None]
    v = (A * F + B * dot(F) * e + C * cross(T, e)).sum(1)
    w = (C * cross(F, e) + Ar * T + Br * dot(T) * e).sum(1)
    size = lambda p: np.sqrt((p * p).sum(-1))[..., None]
    v_size = ((A + B) * size(F) + C * size(T)).sum((1, 2))
    w_size = (C * size(F) + (abs(Ar) + Br) * size(T)).sum((1, 2))
    if kind in ("ss", "sb"):
        return np.concatenate([v, w], 1), np.stack([v_size, w_size], 1)
    return v, v_size[:, None]


@pytest.mark.parametrize("distance", [30.0, 120.0, 300.0, 450.0])
@pytest.mark.parametrize("other", [1.0, 1e-3, 1e-6, 1e-9, 0.0])
@pytest.mark.parametrize("kind,force,torque", [("ss", 1, 1), ("ss", 0, 1), ("ss", 1, 0), ("ss", 1e-2, 1), ("ss", 1, 1e-7),
                                               ("bb", 1, 0), ("sb", 1, 0), ("bs", 0, 1), ("bs", 1e-2, 1), ("bs", 1, 1)])
def test_every_target_of_uneven_loads(host, kind, force, torque, other, distance):
    """Each target's error, however small its velocity: a group of particles,
    and a distant one whose loads are `other` times as large.

    Tolerance: a term (force and torque apart) is rounded at about 2^-54 of its size,
    a sum of sums once more at 2^-53 of its own, so a few times that of the
    sum of the terms' sizes; 2^-51 of it is allowed."""
    rng = np.random.default_rng(int(distance) + 17)
    xs = rng.uniform(-15.0, 15.0, size=(180, 3))
    xs[0] = 0.0
    xs[90:, 0] += distance
    xt = xs if kind in ("ss", "bb") else xs + rng.normal(size=xs.shape)
    f = rng.normal(size=(180, 6)) * np.repeat([force, torque], 3)
    f[90:] *= other
    if kind in ("bb", "sb"):
        f = f[:, :3].copy()
    status, got = fx_sum(host, kind, xt, xs, f, 1.0, 1.0)
    assert status == 0
    want, size = extended_sum(kind, xt, xs, f)
    for b in range(size.shape[1]):
        error = np.sqrt(((got[:, 3 * b:3 * b + 3] - want[:, 3 * b:3 * b + 3]) ** 2).sum(1))
        assert (error <= 2.0 ** -51 * size[:, b]).all(), float((error[size[:, b] > 0] / size[size[:, b] > 0, b]).max())


@pytest.mark.parametrize("distance", [1.0, 0.1, 1e-2, 1e-4, 1e-7])
@pytest.mark.parametrize("kind,force,torque", [("ss", 0, 1), ("ss", 1, 0), ("ss", 1, 1e-9), ("ss", 1, 1), ("bb", 1, 0)])
def test_every_target_of_close_pairs(host, kind, force, torque, distance):
    """Three particles that overlap almost wholly, so that the cross products, which
    vanish with the distance, are all that torques give to v and forces to w.

    Tolerance: as test_every_target_of_uneven_loads, and the positions are
    multiples of the formats' quantum there."""
    rng = np.random.default_rng(19)
    for _ in range(20):
        x = 3.3 + distance * rng.normal(size=(3, 3))
        x = np.rint(np.ldexp(x, 51)) * 2.0 ** -51
        f = rng.normal(size=(3, 6)) * np.repeat([force, torque], 3)
        f = f if kind == "ss" else f[:, :3].copy()
        status, got = fx_sum(host, kind, x, x, f, 1.0, 1.0)
        assert status == 0
        want, size = extended_sum(kind, x, x, f)
        for b in range(size.shape[1]):
            error = np.sqrt(((got[:, 3 * b:3 * b + 3] - want[:, 3 * b:3 * b + 3]) ** 2).sum(1))
            assert (error <= 2.0 ** -51 * size[:, b]).all(), float((error / size[:, b]).max())


@pytest.mark.parametrize("size", [1.0, 2.5, 8.0])
@pytest.mark.parametrize("radius", [1.0, 1.4, 1.99])
@pytest.mark.parametrize("force,torque", [(0, 1), (1, 0), (1, 1)])
def test_overlapping_segments_of_any_radius(host, radius, force, torque, size):
    """Radii over the octave that shares a unit: near it the near-field
    scalars are as small as an eighth of their range.

    Tolerance, in the 2-norm over all targets: the FP64 formulas' own error is 4e-16
    to 6e-16 here (200 terms); 2^-51 is allowed."""
    rng = np.random.default_rng(20)
    xs = radius * rng.uniform(-size, size, size=(200, 3)) + 3.3
    f = rng.normal(size=(200, 6)) * np.repeat([force, torque], 3)
    status, got = fx_sum(host, "ss", xs, xs, f, radius, radius)
    assert status == 0
    a = np.longdouble(radius)
    scaled = f.astype(np.longdouble) / np.repeat([a / a, a], 3)
    want, _ = extended_sum("ss", xs.astype(np.longdouble) / a, xs.astype(np.longdouble) / a, scaled)
    want /= np.repeat([a, a * a], 3)
    for b in (0, 3):
        error, norm = ((v ** 2).sum() for v in (got[:, b:b + 3] - want[:, b:b + 3], want[:, b:b + 3]))
        assert error <= (2.0 ** -51) ** 2 * norm, float(np.sqrt(error / norm))


@pytest.mark.parametrize("kind", ["sb", "bs"])
@pytest.mark.parametrize("a,b", [(1.96, 3.9), (3.9, 1.96), (1.0, 1.9), (1.9, 1.0)])
def test_cross_products_of_overlapping_unequal_radii(host, oracle_built, kind, a, b):
    """The angular velocities from forces, and the velocities from torques, of
    overlapping segments and blobs, against the FP64 oracle, whose sums of 300
    terms differ from the exact ones by about 1e-15 in the 2-norm."""
    rng = np.random.default_rng(26)
    xt, xs = (min(a, b) * rng.uniform(-1.0, 1.0, size=(n, 3)) + 3.3 for n in (200, 300))
    f = rng.normal(size=(300, 6 if kind == "bs" else 3))
    if kind == "bs":
        f[:, :3] = 0.0
    status, got = fx_sum(host, kind, xt, xs, f, a, b)
    assert status == 0
    want = oracle_sum(oracle_built, kind, xt, xs, f, a, b)
    error = (got - want)[:, -3:]
    assert np.linalg.norm(error) < 2.0 ** -49 * np.linalg.norm(want[:, -3:])


def test_translation_and_range(host, oracle_built):
    """Far from the origin the positions stay exact; a cloud too wide, loads
    too large or not finite, and radii too different are reported."""
    xt, xs, f = cloud("ss", "far", 200, 1.0, seed=8)
    for shift in (1e3, 1e6, 1e9):
        x = xs + shift * np.array([1.0, -0.7, 0.3])
        status, got = fx_sum(host, "ss", x, x, f, 1.0, 1.0)
        assert status == 0
        assert rel_err(got, oracle_built.mss(x, f)) < 200 * 2.0 ** -52
    assert fx_sum(host, "ss", 8 * xs, 8 * xs, f, 1.0, 1.0)[0] == 2
    for bad in (np.nan, np.inf, 1e300):
        g = f.copy()
        g[17, 4] = bad
        assert fx_sum(host, "ss", xs, xs, g, 1.0, 1.0)[0] == 2
    assert fx_sum(host, "sb", xs, xs, f[:, :3], 1.0, 2.1)[0] == 1


def test_conversions_round_once(host):
    """FP64 to fixed point and back by integer instructions: the nearest, ties
    to even, as exact arithmetic rounds (no tolerance)."""
    host.fx_host_fixed.argtypes = [ctypes.c_double, ctypes.c_int, ctypes.c_void_p]
    host.fx_host_value.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int]
    host.fx_host_value.restype = ctypes.c_double
    rng = np.random.default_rng(11)
    values = [0.0, -0.0, 0.5, 1.5, -2.5, 2.0 ** 52 + 0.5, 2.0 ** 61, -(2.0 ** 62 - 512), 2.0 ** 62, 5e-324, np.inf, np.nan]
    values += list(rng.normal(size=200) * 2.0 ** rng.integers(-70, 64, 200))
    for v in values:
        for s in (-3, 0, 1, 11):
            r = ctypes.c_longlong(7)
            held = host.fx_host_fixed(v, s, ctypes.byref(r))
            exact = round(Fraction(v) * Fraction(2) ** s) if np.isfinite(v) else None
            fits = exact is not None and abs(Fraction(v)) * Fraction(2) ** s < 2 ** 62
            assert held == fits and r.value == (exact if fits else 0)
    sums = [(0, 0), (0, 1), (0, 2 ** 34), (-1, 0), (-1, 2 ** 32 - 1), (-1, 2 ** 32), (2 ** 20, 1), (2 ** 21 - 1, 2 ** 32 - 1),
            (2 ** 53 + 1, 0), (2 ** 53 + 1, 1), (2 ** 21 + 2 ** 10, 2 ** 31), (-2 ** 62, 0), (2 ** 62, 2 ** 34)]
    sums += [(int(a) >> int(k), int(b)) for a, k, b in zip(rng.integers(-2 ** 62, 2 ** 62, 300), rng.integers(0, 63, 300),
                                                           rng.integers(0, 2 ** 34, 300))]
    for a, b in sums:
        for e in (0, 84, -37):
            assert host.fx_host_value(a, b, e) == float(Fraction(a * 2 ** 32 + b) * Fraction(2) ** (e - 84))


def test_split_rule_over_all_sizes(host):
    """Sources per split: a power of two from 8, no larger than it takes to
    hold all of them, and no more splits than allowed."""
    for groups in (1, 3, 40, 400, 3647, 3648, 4000, 100000, 60000000):
        for n in (1, 7, 128, 5000, 131072, 2000000):
            for most in (1, 5, 1 << 20):
                chunk = host.fx_host_chunk(groups, n, 152, most)
                assert 8 <= chunk < max(2 * n, 256) and chunk & (chunk - 1) == 0, (groups, n, most)
                assert -(-n // chunk) <= most
