"""The device time step against the reference's own simulator.

tests/golden/sim_*.npz were produced by the reference's unmodified
cilia_sim_main.cpp and solver classes compiled for the CPU
(tests/golden/make_golden_sim.py): small_swimmer, one free-swimming sphere of
162 blobs with 4 end-force-driven filaments of 20 segments, 12 steps (Euler,
then BDF2 with both multiplier-extrapolation stages); two_swimmers, two such
swimmers, 8 steps; wall_filaments, nine filaments on an infinite no-slip wall
(INFINITE_PLANE_WALL), 10 steps; config1, 642 blobs and 16 x 20 segments, 100 steps (every
10th stored).  Every stored step is compared: Broyden
iteration count, segment quaternions, body position and orientation, segment
and body velocities.  Differences come from GMRES (CGS2 vs MGS Arnoldi,
tolerance 1e-10), the approximate-Jacobian inverse (Gauss-Jordan vs LAPACK)
and summation order, so state agrees to ~1e-12 and velocities to the GMRES tolerance (~1e-9)
when the Broyden iteration counts agree, which they must, step by step.
"""
import numpy as np
import pytest

from conftest import load_golden, rel_err

pytestmark = pytest.mark.gpu

TRAJ_TOL = 1e-10
VEL_TOL = 1e-7


def run_against_golden(case, state_tol, vel_tol, precision=0, doubling_steps=None):
    """Step through the golden case; Broyden counts must match at every step
    (FP64).  The state and velocity bounds hold at step 0 and, when
    doubling_steps is given, double every doubling_steps steps: differences
    at the GMRES tolerance grow while the filaments' instability develops."""
    from generic_mobility_interface_class_gb300.sim import Simulation
    g = load_golden(case, prefix="sim_")
    wall = bool(g["wall"]) if "wall" in g else False
    sim = Simulation.from_golden(g, precision=precision)
    sim.prepare()
    kept = {int(s): k for k, s in enumerate(g["steps"])}
    worst = {"q": 0.0, "body": 0.0, "v": 0.0, "body_v": 0.0}
    for nt in range(int(g["steps"][-1]) + 1):
        biters, _ = sim.step(nt)
        if precision == 0:
            assert biters == int(g["broyden_iters"][nt]), (nt, biters, int(g["broyden_iters"][nt]))
        if nt not in kept:
            continue
        k = kept[nt]
        grow = 2.0 ** (nt / doubling_steps) if doubling_steps else 1.0
        err = {"q": rel_err(sim.state("seg_q").ravel(), g["seg_q"][k])}
        # the reference writes each swimmer's body state as x (3) then q (4)
        bs = np.hstack([sim.state("body_x"), sim.state("body_q")]).ravel()
        err["body"] = float(np.max(np.abs(bs - g["body_state"][k])))
        err["body_v"] = 0.0 if wall else rel_err(sim.state("body_v").ravel(), g["body_v"][k])
        err["v"] = max(rel_err(sim.state("seg_v").ravel(), g["seg_v"][k]), err["body_v"])
        for key in worst:
            worst[key] = max(worst[key], err[key])
        assert err["q"] < state_tol * grow and err["body"] < state_tol * 10 * grow and err["v"] < vel_tol * grow, \
            (nt, err)
    sim.close()
    return worst


def test_jacobian_inverse_paths_agree(gmi_lib, monkeypatch):
    """The filament Jacobians inverted with one CTA each (GMI_GJ_CLUSTER=0),
    spread over thread-block clusters (the default for few filaments), and
    with the columns stepped through shared memory instead of registers
    (GMI_GJ_REGISTERS=0) perform the same arithmetic: three steps of the
    4-filament swimmer give the same state."""
    from generic_mobility_interface_class_gb300.sim import Simulation
    g = load_golden("small_swimmer", prefix="sim_")
    out = {}
    for mode, (cluster, registers) in {"one-cta": ("0", "1"), "cluster": ("1", "1"),
                                       "one-cta-shared": ("0", "0"), "cluster-shared": ("1", "0")}.items():
        monkeypatch.setenv("GMI_GJ_CLUSTER", cluster)
        monkeypatch.setenv("GMI_GJ_REGISTERS", registers)
        sim = Simulation.from_golden(g, precision=0)
        sim.prepare()
        iters = [sim.step(nt)[0] for nt in range(3)]
        out[mode] = (iters, sim.state("seg_q").copy(), sim.state("seg_v").copy())
        sim.close()
    for mode in ("cluster", "one-cta-shared", "cluster-shared"):
        assert out[mode][0] == out["one-cta"][0], mode
        assert rel_err(out[mode][1].ravel(), out["one-cta"][1].ravel()) < 1e-13, mode
        assert rel_err(out[mode][2].ravel(), out["one-cta"][2].ravel()) < 1e-9, mode


def test_fp32_jacobian_inverse_in_mixed_precision(gmi_lib, monkeypatch):
    """Mixed-precision (FP32C) steps invert the approximate Jacobians in FP32
    by default (GMI_GJ_FP32=0: FP64).  The inverse only starts each Broyden
    iteration, so both take the same Broyden iterations (to one per step) and
    end at the same state to the Broyden tolerance: two runs that each stop
    at a residual of 1e-4 differ in the velocities by up to a few times that
    (3e-4 here, max-normalised); with one CTA per matrix and with clusters."""
    from generic_mobility_interface_class_gb300.sim import Simulation
    g = load_golden("small_swimmer", prefix="sim_")
    out = {}
    for gj in ("0", "1"):
        for cluster in ("0", "1"):
            monkeypatch.setenv("GMI_GJ_FP32", gj)
            monkeypatch.setenv("GMI_GJ_CLUSTER", cluster)
            sim = Simulation.from_golden(g, precision=1)
            sim.prepare()
            iters = [sim.step(nt)[0] for nt in range(6)]
            out[gj, cluster] = (iters, sim.state("seg_q").copy(), sim.state("seg_v").copy())
            sim.close()
    ref = out["0", "0"]
    for key, (iters, q, v) in out.items():
        assert all(abs(a - b) <= 1 for a, b in zip(iters, ref[0])), (key, iters, ref[0])
        assert rel_err(q.ravel(), ref[1].ravel()) < 1e-6, key
        assert rel_err(v.ravel(), ref[2].ravel()) < 3e-4, key


@pytest.mark.parametrize("nseg,nfil", [(5, 3), (6, 90), (11, 4), (20, 1), (21, 170)])
def test_fp32_inverse_in_registers_keeps_its_bits(gmi_lib, monkeypatch, nseg, nfil):
    """The FP32 Jacobian inverse held in registers (6 nseg <= 128) performs the
    arithmetic of the shared-memory path (GMI_GJ_REGISTERS=0): the same state,
    bit for bit, around its 32, 64 and 128 rows and for few and many matrices."""
    from generic_mobility_interface_class_gb300 import seeding, workloads
    from generic_mobility_interface_class_gb300._lib import GmiError
    from generic_mobility_interface_class_gb300.sim import Simulation
    out = {}
    for registers in ("0", "1"):
        monkeypatch.setenv("GMI_GJ_REGISTERS", registers)
        fils = seeding.fibonacci_sphere(nfil)
        sim = Simulation(**workloads.free_swimmer(seeding.fibonacci_sphere(400), fils, radius=14.0, nseg=nseg, seed=3),
                         precision=1)
        sim.prepare()
        iters = []
        try:
            for nt in range(2):
                iters.append(sim.step(nt)[0])
        except GmiError as e:  # a step that Broyden's method gives up on does so either way
            iters.append(str(e))
        out[registers] = (iters, sim.state("seg_q").copy(), sim.state("seg_v").copy())
        sim.close()
    assert out["0"][0] == out["1"][0]
    np.testing.assert_array_equal(out["0"][1], out["1"][1])
    np.testing.assert_array_equal(out["0"][2], out["1"][2])


def test_trajectory_matches_reference(gmi_lib):
    """12 steps of a 4-filament swimmer, every step compared."""
    run_against_golden("small_swimmer", TRAJ_TOL, VEL_TOL)


def test_two_swimmers_match_reference(gmi_lib):
    """Two identical swimmers (4 x 20 segments and 162 blobs each, placed as
    the reference places them), 8 steps: the per-swimmer offsets of every
    kernel of the time step, and the preconditioner's Minv^(W - n) scaling."""
    run_against_golden("two_swimmers", TRAJ_TOL, VEL_TOL)


def test_wall_filaments_match_reference(gmi_lib):
    """Nine filaments on the infinite no-slip wall (Swan-Brady mobility,
    wall barrier, no rigid body, no linear solve), 10 steps."""
    run_against_golden("wall_filaments", TRAJ_TOL, VEL_TOL)


def test_config1_100_steps_match_reference(gmi_lib):
    """BASELINE config-1 geometry (642 blobs, 16 x 20 segments), 100 steps:
    identical Broyden iteration counts at every step, and the state at every
    10th step against the reference's own run.  This case solves GMRES to
    1e-8, and the end-force instability amplifies differences at that level
    about twofold every 10 steps; the bounds start at 1e-8 (state) and 1e-6
    (velocities) and double every 10 steps."""
    run_against_golden("config1", 1e-8, 1e-6, doubling_steps=10)


def test_config1_mixed_precision_trajectory(gmi_lib):
    """The FP32C pair sums with FP64 solves follow the FP64 trajectory:
    swimmer (body) velocities within 1e-5 of the reference's at every stored
    step of the 100."""
    worst = run_against_golden("config1", 1e-6, 1e-5, precision=1, doubling_steps=20)
    assert worst["body_v"] < 1e-5
