"""The solver's host arrays are views of its pinned memory."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_views_outlive_the_solver(gmi_lib):
    """An array taken from a solver that is gone still shows its memory (it
    read unmapped memory), and close() ends the solver at once."""
    from generic_mobility_interface_class_gb300.solver import MobilitySolver
    solver = MobilitySolver(nfil=2, nseg=5, nblob=42)
    x = solver.x_segs_host
    x[:] = np.arange(30.0).reshape(10, 3)
    row = x[3]
    del solver, x
    gc.collect()
    np.testing.assert_array_equal(row, [9.0, 10.0, 11.0])
    with MobilitySolver(nfil=1, nseg=4, nblob=42) as other:
        owner = other._owner
        assert other.v_segs_host.shape == (4, 6) and other.v_segs_host.flags.writeable
    assert owner.handle is None and other.handle is None
