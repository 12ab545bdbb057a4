"""Edge cases of the timestep on the GPU: an empty system, a single
particle, a crowded cell far above the mean occupancy, and particles on the
box faces.  Each runs the production pass against the stand-alone stage
kernels (bit-identical trajectories) and checks that no particle is lost."""
from __future__ import annotations

import numpy as np
import pytest

from master_b200 import capi
from master_b200.system import System
from master_b200.workloads import Workload, simulators_per_cell_weight
from test_parity_gpu import load_case

pytestmark = pytest.mark.gpu


def pair(case, r, v):
    z, meta, s, g = load_case(case)
    A = System(s, g, init_particles=False)
    B = System(s, g, init_particles=False)
    A.set_particles(r, v)
    B.set_particles(r, v)
    return A, B


def run_both(A, B, K):
    A.step(K)
    for _ in range(K):
        B.accelerate_and_move()
        B.update_molecule_cells()
        B.collide()
        B.sample()
    ra, va, ca = A.get_particles(with_cells=True)
    rb, vb, cb = B.get_particles(with_cells=True)
    assert np.array_equal(ra, rb) and np.array_equal(va, vb) and np.array_equal(ca, cb)
    ta, tb = A.tallies(), B.tallies()
    for k in ("collisions", "wall_collisions", "candidates", "reseeds"):
        assert getattr(ta, k) == getattr(tb, k), k
    return ra, va


def test_empty_system_steps():
    z, meta, s, g = load_case("small_dt1")
    S = System(s, g, init_particles=False)
    S.set_particles(np.zeros((0, 3)), np.zeros((0, 3)))
    S.step(4)
    t = S.tallies()
    assert S.num_molecules == 0
    assert t.step == 4 and t.collisions == 0 and t.wall_collisions == 0 and t.particle_steps == 0
    r, v = S.get_particles()
    assert r.shape == (0, 3)
    assert not S.profile_sums().any()


def test_single_particle():
    z, meta, s, g = load_case("small_dt5")
    A, B = pair("small_dt5", z["r0"][:1], z["v0"][:1])
    r, v = run_both(A, B, 20)
    assert A.num_molecules == 1 and A.tallies().collisions == 0


@pytest.mark.parametrize("crowd", [110, 230])
def test_crowded_cell_spills_and_keeps_every_particle(crowd):
    """One cell starts with `crowd` particles (the mean is 15): its members
    take the production pass's large-cell paths, its neighbours overflow as
    the crowd spreads and the host repacks, and both paths still agree and
    keep every particle."""
    z, meta, s, g = load_case("small_dt5")
    r = z["r0"].copy()
    v = z["v0"].copy()
    N = r.shape[0]
    cell = z["cell0"]
    target = np.bincount(cell).argmax()
    home = r[np.flatnonzero(cell == target)[0]]
    others = np.flatnonzero(cell != target)[: crowd - int((cell == target).sum())]
    r[others] = home
    A, B = pair("small_dt5", r, v)
    assert A.cells()["count"].max() >= crowd
    assert A.ctx.pass_info()["pipelined"] == 1
    run_both(A, B, 6)
    assert A.num_molecules == N


def test_particles_on_the_box_faces():
    """Positions at 0 and one ulp below L in each direction (in the first and
    last voxel layers) wrap and move exactly as the stage kernels do."""
    z, meta, s, g = load_case("small_dt1")
    r = z["r0"].copy()
    v = z["v0"].copy()
    L = np.array([s.Lx, s.Ly, s.Lz])
    n = np.array(g.shape)
    vox = L / n
    used = set()
    for d in range(3):
        for upper in (False, True):
            layer = r[:, d] >= L[d] - vox[d] if upper else r[:, d] < vox[d]
            i = next(int(j) for j in np.flatnonzero(layer) if int(j) not in used)
            used.add(i)
            r[i, d] = np.nextafter(L[d], 0) if upper else 0.0
            v[i, d] = abs(v[i, d]) if upper else -abs(v[i, d])  # heading out of the box
    A, B = pair("small_dt1", r, v)
    ra, _ = A.get_particles()
    for i in used:
        assert (ra[i] >= 0).all() and (ra[i] < L).all()
    run_both(A, B, 5)
    assert A.num_molecules == r.shape[0]


def test_graph_replay_equals_plain_launches():
    """The production pass replayed from captured CUDA graphs (the default)
    and launched kernel by kernel (as with the per-kernel timers on) give
    bit-identical trajectories."""
    z, meta, s, g = load_case("small_dt5")
    A = System(s, g, init_particles=False)
    B = System(s, g, init_particles=False)
    A.set_particles(z["r0"], z["v0"])
    B.set_particles(z["r0"], z["v0"])
    B.ctx.set_timing(True)
    for k in (1, 3, 7):  # batches of several passes, every buffer parity and occupancy set
        A.step(k)
        B.step(k)
    ra, va, ca = A.get_particles(with_cells=True)
    rb, vb, cb = B.get_particles(with_cells=True)
    assert np.array_equal(ra, rb) and np.array_equal(va, vb) and np.array_equal(ca, cb)
    assert A.tallies().collisions == B.tallies().collisions
    assert B.ctx.pass_times()["passes"] > 0


@pytest.mark.parametrize("capacity", [None, (1.5, 3), (1.0, 0)])
def test_device_layout_follows_the_capacity_rule(capacity):
    """Cell capacities are computed on the device whenever the buffers are
    laid out: ceil(factor * max(expected, present) + pad) per active cell,
    expected = particles * free voxels of the cell / free voxels of the
    system (rounded without fused multiply-add), and the slots total their
    sum.  The counts come back through the device table as well."""
    from master_b200.system import cells_layout
    z, meta, s, g = load_case("small_dt5")
    S = System(s, g, init_particles=False)
    factor, pad = capacity or (2.0, 24)
    if capacity:
        S.ctx.check(S.ctx.lib.dsmc_ctx_set_capacity(S.ctx.handle, factor, pad))
    S.set_particles(z["r0"], z["v0"])
    cells = S.cells()
    lay = cells_layout(s, g)
    assert np.array_equal(cells["global_index"], lay["global_index"])
    present = cells["count"].astype(np.float64)
    assert present.sum() == z["r0"].shape[0]
    pix = lay["pixels"].astype(np.float64)
    expect = (z["r0"].shape[0] * pix) / pix.sum()
    cap = np.maximum(np.ceil(factor * np.maximum(expect, present) + pad), 1.0)
    assert S.info().slots == int(cap.sum())


@pytest.mark.parametrize("precision", [capi.PREC_SPLIT32, capi.PREC_FP64])
@pytest.mark.parametrize("where", ["r_nan", "v_nan", "v_inf"])
def test_non_finite_state_is_refused_and_the_system_keeps_its_particles(precision, where):
    """A non-finite position or velocity handed to dsmc_particles_set is
    refused (DSMC_ERR_STATE, the message says why) before it reaches a
    kernel; the system keeps the particles it had and steps on."""
    z, meta, s, g = load_case("small_dt1")
    S = System(s, g, precision=precision, init_particles=False)
    S.set_particles(z["r0"], z["v0"])
    r_before, v_before = S.get_particles()
    r, v = z["r0"].copy(), z["v0"].copy()
    if where == "r_nan":
        r[len(r) // 2, 1] = np.nan
    elif where == "v_nan":
        v[3, 0] = np.nan
    else:
        v[-1, 2] = np.inf
    with pytest.raises(capi.DsmcError) as e:
        S.set_particles(r, v)
    assert e.value.code == capi.DSMC_ERR_STATE and "non-finite" in str(e.value)
    assert S.num_molecules == len(z["r0"])
    r_after, v_after = S.get_particles()
    assert np.array_equal(r_after, r_before) and np.array_equal(v_after, v_before)
    S.step(3)
    err, _ = S.ctx.device_status()
    assert err & capi.EBIT_FATAL == 0
    r3, v3 = S.get_particles()
    assert np.isfinite(r3).all() and np.isfinite(v3).all() and S.tallies().step == 3


@pytest.mark.parametrize("n,per_cell,dt_si,model,alpha_n", [
    (16, 20, 1e-11, 0, 0.0), (16, 20, 1e-11, 2, 0.5), (16, 20, 5e-11, 1, 0.0), (32, 20, 2e-11, 2, 0.8),
    (34, 20, 5e-11, 0, 0.0), (64, 60, 1e-10, 0, 0.0), (64, 60, 1e-10, 2, 1.0)])
def test_wall_flights_few_and_many(n, per_cell, dt_si, model, alpha_n):
    """place_walls with a handful of wall flights (claims of one entry per
    warp) up to more than its grid holds at 32 a warp, under each wall model;
    the Cercignani-Lampis sampler, whose trials the warp shares, at an
    accommodation where it takes many trials and where it takes few.  Bit for
    bit the stage kernels, which run one flight per lane and one trial at a
    time."""
    w = Workload("walls", n=n, radius_voxels=3.0, porosity=0.6, geometry_seed=5, cells=n // 2,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, 2, per_cell), dt_si=dt_si)
    g = w.geometry()
    s = w.settings(rng_seed=11, statistics_interval=10 ** 9)
    s.surface_model = model
    if model == 2:
        s.alpha_n, s.alpha_t = alpha_n, 0.8
    A, B = System(s, g), System(s, g)
    run_both(A, B, 3)
    assert A.tallies().wall_collisions > 0


@pytest.mark.parametrize("cells,per_cell,dt_si,model", [(64, 3, 2e-11, 0), (64, 3, 2e-11, 1), (32, 60, 1e-10, 0), (16, 20, 1e-11, 0)])
def test_wall_flights_own_and_listed(cells, per_cell, dt_si, model):
    """place_movers with a quarter of an SM's blocks and with all: at 64^3
    cells (1.6e5 active) the first lists its wall flights and the second has
    each warp move its own; at 32^3 and 16^3 both move their own, the first with several
    turns of 32 flights per warp.  The state is the same bit for bit."""
    from master_b200 import autotune
    w = Workload("walls", n=64, radius_voxels=3.0, porosity=0.6, geometry_seed=5, cells=cells,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, 2, per_cell * (cells / 32.0) ** 3), dt_si=dt_si)
    g = w.geometry()
    s = w.settings(rng_seed=11, statistics_interval=10 ** 9)
    s.surface_model = model
    A, B = System(s, g), System(s, g)
    autotune.set_tuning(A.ctx, (0, 0, 1, 0, 0))
    for S in (A, B):
        assert S.ctx.pass_info()["pipelined"] == 1
        S.step(4)
    (ra, va), (rb, vb) = A.get_particles(), B.get_particles()
    assert np.array_equal(ra, rb) and np.array_equal(va, vb)
    ta, tb = A.tallies(), B.tallies()
    assert ta.wall_collisions == tb.wall_collisions > 0 and ta.collisions == tb.collisions
    assert A.ctx.device_status()[0] & capi.EBIT_FATAL == 0


@pytest.mark.parametrize("precision", [capi.PREC_SPLIT32, capi.PREC_FP64])
@pytest.mark.parametrize("n", [1, 1000, (1 << 20) - 1, (1 << 20) + 3, 9 * (1 << 19) + 1])
def test_state_in_and_out_by_ranges(n, precision):
    """Uploads and downloads of one, two and eight ranges of ids, in an order that
    is not the cells': velocities and cells come back exact, positions within
    the rounding of a voxel's fp32 offset (two roundings of 2^-24), and every
    particle is counted in its cell."""
    w = Workload("io", n=64, radius_voxels=3.0, porosity=0.6, geometry_seed=2, cells=64,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, 2, 20))
    g = w.geometry()
    s = w.settings(rng_seed=3, statistics_interval=10 ** 9)
    base = System(s, g, precision=precision)
    r0, v0, c0 = base.get_particles(with_cells=True)
    pick = np.random.default_rng(n).integers(0, len(r0), n)
    S = System(s, g, precision=precision, init_particles=False)
    S.set_particles(r0[pick], v0[pick])
    r, v, c = S.get_particles(with_cells=True)
    assert np.abs(r - r0[pick]).max() <= 2.0 ** -22 * r0.max() / 64
    assert np.array_equal(v, v0[pick]) and np.array_equal(c, c0[pick])
    cells = S.cells()
    want = np.bincount(c, minlength=64 ** 3)
    assert np.array_equal(cells["count"], want[cells["global_index"]])


def test_steps_after_new_states_of_other_sizes():
    """A context's captured passes outlive a new state: the same steps follow
    from the same state whether the context held as many particles before,
    five times as many, or few (its buffers and launch shape then change)."""
    w = Workload("again", n=32, radius_voxels=3.0, porosity=0.6, geometry_seed=5, cells=16,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, 2, 40))
    g = w.geometry()
    s = w.settings(rng_seed=11, statistics_interval=10 ** 9)
    base = System(s, g)
    r, v = base.get_particles()
    out = []
    for k in (1, 5, 0):
        S = System(s, g, init_particles=False)
        first = (np.tile(r, (k, 1)), np.tile(v, (k, 1))) if k else (r[:100], v[:100])
        S.set_particles(*first)
        S.step(7)
        S.set_particles(r, v)
        c = S.cells()
        S.set_cell_state(np.full(len(c["count"]), 3.0), np.zeros(len(c["count"])))
        S.step(9)
        out.append(S.get_particles())
    for r1, v1 in out[1:]:
        assert np.array_equal(r1, out[0][0]) and np.array_equal(v1, out[0][1])


@pytest.mark.parametrize("n,cells,per_cell,model,launches", [
    (8, 4, 20, 0, 1), (24, 12, 20, 1, 1), (32, 16, 20, 1, 2), (32, 8, 60, 1, 2), (32, 16, 20, 2, 1), (48, 24, 20, 2, 2),
    (40, 20, 20, 0, 1), (64, 32, 20, 0, 2)])
def test_generic_pass_moves_or_lists_its_wall_flights(n, cells, per_cell, model, launches):
    """fp64 steps on both sides of the rule by which the cell pass moves its
    wall flights itself (one kernel a step) or lists them (two), for each wall model
    and for cells of more than 32 members: bit for bit the stage kernels."""
    w = Workload("walls", n=n, radius_voxels=3.0, porosity=0.6, geometry_seed=5, cells=cells,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, n // cells, per_cell), dt_si=2e-11)
    g = w.geometry()
    s = w.settings(rng_seed=11, statistics_interval=2)
    s.surface_model = model
    if model == 2:
        s.alpha_n, s.alpha_t = 0.8, 0.8
    A, B = System(s, g, precision=capi.PREC_FP64), System(s, g, precision=capi.PREC_FP64)
    assert A.ctx.pass_launches() == (launches, 0)
    run_both(A, B, 5)
    assert A.tallies().wall_collisions > 0


@pytest.mark.parametrize("n,per_cell,model,launches", [(32, 400, 0, 1), (64, 400, 2, 1), (32, 400, 1, 2), (160, 300, 0, 2)])
def test_generic_pass_of_large_cells_moves_or_lists_its_wall_flights(n, per_cell, model, launches):
    """Cells of more particles than the production pass stages (the generic pass in
    split precision), on both sides of the same rule: bit for bit the stage
    kernels."""
    w = Workload("walls", n=n, radius_voxels=4.0, porosity=0.6, geometry_seed=1, cells=n // 8,
                 atoms_per_molecule=simulators_per_cell_weight(2.5e24, 0.1, 8, per_cell))
    g = w.geometry()
    s = w.settings(rng_seed=11, statistics_interval=2)
    s.surface_model = model
    if model == 2:
        s.alpha_n, s.alpha_t = 0.8, 0.8
    A, B = System(s, g), System(s, g)
    assert A.ctx.pass_info()["pipelined"] == 0
    assert A.ctx.pass_launches() == (launches, 0)
    run_both(A, B, 3)
    assert A.tallies().wall_collisions > 0
