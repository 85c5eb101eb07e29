"""The FP64 wall kernel at the edges of its target groups and source splits,
against the FP64 oracle.

Tolerance: a pair's coefficients come from some 40 rounded operations whose
terms are up to about ten times the pair's own velocity near the wall, so
2^-44 of the largest velocity.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import rel_err

pytestmark = pytest.mark.gpu


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


@pytest.mark.parametrize("n", [1, 4, 31, 33, 129, 320, 1281, 2999])
def test_wall_sizes_against_oracle(gpu_ctx, oracle_built, n):
    rng = np.random.default_rng(n)
    side = 3.0 * max(n, 4) ** (1 / 3)
    x = rng.uniform(0.0, side, size=(n, 3)) + np.array([0.0, 0.0, 1.05])
    f = rng.normal(size=(n, 6))
    gpu_ctx.set_precision(0)
    want = oracle_built.mss_wall(x, f)
    assert rel_err(gpu_ctx.mss_wall(T(x), T(f)).cpu().numpy(), want) < 2.0 ** -44
    if n > 300:  # a slice of the targets, not on a group's edge
        got = gpu_ctx.mss_wall(T(x), T(f), start=37, num=211).cpu().numpy()
        assert rel_err(got, want[37:248]) < 2.0 ** -44


def test_wall_separations_whose_square_overflows(gpu_ctx, oracle_built):
    """Finite velocities, as from 1 / inf = 0; a position that is not finite still
    makes every target NaN."""
    rng = np.random.default_rng(2)
    x = rng.uniform(0.0, 9.0, size=(40, 3)) + np.array([0.0, 0.0, 1.05])
    f = rng.normal(size=(40, 6))
    x[17, 0] = 1e170
    gpu_ctx.set_precision(0)
    want = oracle_built.mss_wall(x, f)
    assert np.isfinite(want).all()
    assert rel_err(gpu_ctx.mss_wall(T(x), T(f)).cpu().numpy(), want) < 2.0 ** -44
    for bad in (np.nan, np.inf):
        x[17, 0] = bad
        assert not np.isfinite(gpu_ctx.mss_wall(T(x), T(f)).cpu().numpy()[:, :3]).any()


def test_wall_source_without_loads_in_a_targets_place(gpu_ctx, oracle_built):
    """It changes nothing but its own velocity, which is its neighbour's less
    the neighbour's own."""
    rng = np.random.default_rng(3)
    x = rng.uniform(0.0, 9.0, size=(60, 3)) + np.array([0.0, 0.0, 1.05])
    f = rng.normal(size=(60, 6))
    gpu_ctx.set_precision(0)
    want = oracle_built.mss_wall(x, f)
    got = gpu_ctx.mss_wall(T(np.concatenate([x, x[:1]])), T(np.concatenate([f, np.zeros((1, 6))])), num=60)
    assert rel_err(got.cpu().numpy(), want) < 2.0 ** -44
