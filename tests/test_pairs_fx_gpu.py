"""The fixed-point pair kernel (FP64 precision, no wall) at the edges of its
tiles, splits and formats, against the FP64 oracle.

Tolerance: as test_pairs_fx_cpu.py, n 2^-52 of the largest velocity (the
oracle's own rounding over n terms), and 2^-50 at least.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import rel_err

pytestmark = pytest.mark.gpu


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def N(t):
    return t.detach().cpu().numpy()


def tol(n):
    return max(n * 2.0 ** -52, 2.0 ** -50)


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 2.6 * max(n, 8) ** (1 / 3), size=(n, 3))
    return x, rng.normal(size=(n, 6))


def check_all(ctx, rpy, xs, fs, xb, fb, b=1.3, bound=None):
    bound = tol(len(xs) + len(xb)) if bound is None else bound
    assert rel_err(N(ctx.mss(T(xs), T(fs))), rpy.mss(xs, fs)) < bound
    assert rel_err(N(ctx.mbb(T(xb), T(fb))), rpy.mbb(xb, fb)) < bound
    v = np.random.default_rng(1).normal(size=(len(xs), 6))
    got = T(v)
    ctx.msb(T(xs), T(xb), T(fb), got, a_blob=b)
    assert rel_err(N(got), rpy.msb(xs, xb, fb, 1.0, b, v_in=v)) < bound
    assert rel_err(N(ctx.mbs(T(xb), T(xs), T(fs), a_blob=b)), rpy.mbs(xb, xs, fs, 1.0, b)) < bound


@pytest.mark.parametrize("ns,nb", [(1, 1), (31, 2), (32, 33), (33, 127), (127, 128), (129, 257), (320, 642),
                                   (511, 512), (513, 1025), (963, 1281), (3001, 2047), (1537, 4099)])
def test_sizes_against_oracle(gpu_ctx, oracle_built, ns, nb):
    xs, fs = cloud(ns, 3)
    xb, fb = cloud(nb, 4)
    gpu_ctx.set_precision(0)
    check_all(gpu_ctx, oracle_built, xs, fs, xb, fb[:, :3])


def test_tiles_outside_the_formats(gpu_ctx, oracle_built):
    """A particle far out (its tile, and it as a target, in FP64), a huge load
    (its tile), the others beside them in fixed point."""
    xs, fs = cloud(700, 5)
    xb, fb = cloud(500, 6)
    xs[300] += 5000.0
    xb[60] -= 2.0e5
    fs[40, 2] = 1e295
    gpu_ctx.set_precision(0)
    check_all(gpu_ctx, oracle_built, xs, fs, xb, fb[:, :3])


@pytest.mark.parametrize("n", [33, 300, 1100])
@pytest.mark.parametrize("b", [0.6, 1.0, 1.3])
def test_whole_sets_outside_the_formats(gpu_ctx, oracle_built, n, b):
    """Sets spread over thousands of radii, in FP64 throughout: distant,
    overlapping and coincident pairs."""
    rng = np.random.default_rng(n)
    def spread(m):
        x = rng.uniform(-4000.0, 4000.0, size=(m, 3))
        x[1::3] = x[0:-1:3][:len(x[1::3])] + rng.normal(size=(len(x[1::3]), 3))
        x[2::6] = x[0:-2:6][:len(x[2::6])]
        return x
    xs, xb = spread(n), spread(n + 40)
    xb[3::4] = xs[:len(xb[3::4])] + 0.7 * rng.normal(size=(len(xb[3::4]), 3))
    fs, fb = rng.normal(size=(n, 6)), rng.normal(size=(n + 40, 3))
    gpu_ctx.set_precision(0)
    check_all(gpu_ctx, oracle_built, xs, fs, xb, fb, b=b)
    xs[n // 2, 1] = 1e200  # the square overflows: as far as can be
    got, want = N(gpu_ctx.mss(T(xs), T(fs))), oracle_built.mss(xs, fs)
    assert np.isfinite(want).all() and rel_err(got, want) < tol(n)


def test_not_finite_loads_and_positions(gpu_ctx, oracle_built):
    """A NaN load reaches every target, an infinite one too; a NaN position
    its own row and, as a source, all."""
    xs, fs = cloud(300, 7)
    gpu_ctx.set_precision(0)
    bad = fs.copy()
    bad[200, 1] = np.nan
    assert np.isnan(N(gpu_ctx.mss(T(xs), T(bad)))[:, :3]).all()
    bad[200, 1] = np.inf
    assert not np.isfinite(N(gpu_ctx.mss(T(xs), T(bad)))[:, :3]).any()
    x = xs.copy()
    x[10, 0] = np.nan
    assert np.isnan(N(gpu_ctx.mss(T(x), T(fs)))).all()


def test_slices_and_radii_ratio(gpu_ctx, oracle_built):
    """Target slices that start inside a group of 32, and radii whose ratio
    the formats do not hold (the FP64 kernels)."""
    rpy = oracle_built
    xs, fs = cloud(900, 8)
    xb, fb = cloud(400, 9)
    gpu_ctx.set_precision(0)
    got = N(gpu_ctx.mss(T(xs), T(fs), start=45, num=333))
    assert rel_err(got, rpy.mss(xs, fs)[45:378]) < tol(900)
    for b in (0.5, 2.0, 0.3, 5.0):
        check_all(gpu_ctx, rpy, xs, fs, xb, fb[:, :3], b=b)


@pytest.mark.parametrize("a,b", [(0.95, 1.9), (1.9, 0.95), (1.95, 3.9), (3.7, 1.89)])
def test_overlapping_unequal_radii(gpu_ctx, oracle_built, a, b):
    """Radii whose near field, in the formats' units, ends furthest out."""
    rng = np.random.default_rng(13)
    xs, xb = (rng.uniform(-3.0 * min(a, b), 3.0 * min(a, b), size=(n, 3)) for n in (300, 200))
    fs, fb, v = rng.normal(size=(300, 6)), rng.normal(size=(200, 3)), rng.normal(size=(300, 6))
    gpu_ctx.set_precision(0)
    got = T(v)
    gpu_ctx.msb(T(xs), T(xb), T(fb), got, a_seg=a, a_blob=b)
    assert rel_err(N(got), oracle_built.msb(xs, xb, fb, a, b, v_in=v)) < tol(500)
    assert rel_err(N(gpu_ctx.mbs(T(xb), T(xs), T(fs), a_seg=a, a_blob=b)), oracle_built.mbs(xb, xs, fs, a, b)) < tol(500)


@pytest.mark.parametrize("n", [90, 700, 2300])
@pytest.mark.parametrize("force,torque,other", [(0, 1, 1e-6), (1e-2, 1, 1), (1, 1e-7, 1e-3), (1, 1, 1e-8)])
def test_every_target_of_uneven_loads(gpu_ctx, n, force, torque, other):
    """As test_pairs_fx_cpu.py's test of that name, with loads whose forces,
    torques and particles differ much in size: 40 of the targets, of sums
    whose CTAs pack their own sources and (2300) of sums with a pack kernel."""
    from test_pairs_fx_cpu import extended_sum
    rng = np.random.default_rng(n)
    size = 1.6 * n ** (1 / 3)
    xs, xt = (rng.uniform(-size, size, size=(n, 3)) for _ in range(2))
    xs[n // 3:, 1] += 260.0
    xt[n // 3:, 1] += 260.0
    fs = rng.normal(size=(n, 6)) * np.repeat([force, torque], 3)
    fs[n // 3:] *= other
    fb = fs[:, :3].copy()
    gpu_ctx.set_precision(0)
    few = slice(n // 3 - 20, n // 3 + 20)
    v = torch.zeros((n, 6), dtype=torch.float64, device="cuda")
    for kind, x, f, got in (("ss", xs, fs, gpu_ctx.mss(T(xs), T(fs))),
                            ("sb", xt, fb, gpu_ctx.msb(T(xt), T(xs), T(fb), v)),
                            ("bs", xt, fs, gpu_ctx.mbs(T(xt), T(xs), T(fs)))):
        want, terms = extended_sum(kind, x[few], xs, f)
        got = N(got)[few]
        for b in range(terms.shape[1]):
            error = np.sqrt(((got[:, 3 * b:3 * b + 3] - want[:, 3 * b:3 * b + 3]) ** 2).sum(1))
            assert (error <= 2.0 ** -51 * terms[:, b]).all(), kind


def test_targets_that_fill_the_gpu_many_times(gpu_ctx, oracle_built):
    """More targets than 24 CTAs per SM take: one slice of the sources."""
    rng = np.random.default_rng(16)
    xt, xs = rng.uniform(-60.0, 60.0, size=(150_000, 3)), rng.uniform(-60.0, 60.0, size=(300, 3))
    fs = rng.normal(size=(300, 6))
    gpu_ctx.set_precision(0)
    got = N(gpu_ctx.mbs(T(xt), T(xs), T(fs)))
    rows = rng.integers(0, len(xt), 400)
    assert rel_err(got[rows], oracle_built.mbs(xt[rows], xs, fs, 1.0, 1.0)) < tol(300)


@pytest.mark.parametrize("ns,nt", [(8, 3000), (300, 2000)])
def test_sums_into_their_inputs(gpu_ctx, ns, nt):
    """Velocities that overwrite positions or loads: as with arrays apart, also
    where one split of the sources would let a CTA write at once (8)."""
    rng = np.random.default_rng(18)
    xs, fs, xt = T(rng.uniform(-9, 9, (ns, 3))), T(rng.normal(size=(ns, 6))), T(rng.uniform(-30, 30, (nt, 3)))
    gpu_ctx.set_precision(0)
    want = N(gpu_ctx.mbs(xt, xs, fs)) + 0.0
    x = xt.clone()
    np.testing.assert_array_equal(N(gpu_ctx.mbs(x, xs, fs, out=x)), want)
    v = torch.zeros((nt, 3), dtype=torch.float64, device="cuda")
    loads = v.view(-1)[-6 * ns:].view(ns, 6)
    loads.copy_(fs)
    np.testing.assert_array_equal(N(gpu_ctx.mbs(xt, xs, loads, out=v)), want)
    f = fs.clone()
    np.testing.assert_array_equal(N(gpu_ctx.mss(xs, f, out=f)), N(gpu_ctx.mss(xs, fs)))
    f = fs.clone()
    x = xs + torch.tensor([0.0, 0.0, 12.0], dtype=torch.float64, device="cuda")
    np.testing.assert_array_equal(N(gpu_ctx.mss_wall(x, f, out=f)), N(gpu_ctx.mss_wall(x, fs)))


def test_pinned_fp64_shape_keeps_its_kernel(gmi_lib, oracle_built):
    """A shape pinned in FP64 runs the FP64 kernel of that shape."""
    from generic_mobility_interface_class_gb300.mobility import Context
    xs, fs = cloud(700, 10)
    with Context(0) as ctx:
        auto = N(ctx.mss(T(xs), T(fs)))
        ctx.set_shape(0, 700, 700, 64, 1, 3, 1)
        assert ctx.tuned_shape(0, 700, 700) == (64, 1, 3, True)
        pinned = N(ctx.mss(T(xs), T(fs)))
        assert rel_err(pinned, auto) < tol(700)
        ctx.autotune(0, 700, 700)
        assert ctx.tuned_shape(0, 700, 700)[3]
        np.testing.assert_array_equal(N(ctx.mss(T(xs), T(fs))), auto)


def test_autotuned_fp64_outside_the_formats(gmi_lib, oracle_built):
    """Radii that the formats do not hold after a call to the autotuner: the
    FP64 kernel that it found (a few hundred sources: the warp kernel, seven
    times faster than the tiled ones), or the same as without the call."""
    from generic_mobility_interface_class_gb300.mobility import Context
    xs, fs = cloud(300, 14)
    xb, fb = cloud(280, 15)
    with Context(0) as ctx, Context(0) as plain:
        ctx.autotune(0, 300, 300)
        tiny = 1e-70
        np.testing.assert_array_equal(N(ctx.mss(T(xs), T(fs), a=tiny)), N(plain.mss(T(xs), T(fs), a=tiny)))
        ctx.autotune(3, 300, 280)
        ctx.autotune(4, 280, 300)
        assert ctx.tuned_shape(3, 300, 280)[0] == 32 and ctx.tuned_shape(4, 280, 300)[0] == 32
        for b in (0.3, 1.0):
            got = [N(c.mbs(T(xb), T(xs), T(fs), a_blob=b)) for c in (ctx, plain)]
            assert rel_err(got[0], oracle_built.mbs(xb, xs, fs, 1.0, b)) < tol(300)
            if b == 1.0:
                np.testing.assert_array_equal(*got)
