"""GPU parity of the fused fast path (sym_step in CONFIG mode) against the oracle.

FP64 storage: field relative L2 <= 1e-10 after the stated number of steps,
masks bit-exact, particle trajectories <= 1e-9.  FP32 and FP16 shifted storage:
relative L2 velocity error against FP64 <= 1e-3 (the precision target), with
the measured errors printed.
"""
import itertools

import numpy as np
import pytest

from oracle.oracle import Oracle, setup_workload as orc_setup
from symmetry_b200 import configs
from symmetry_b200.lib import Lattice, setup_workload
from symmetry_b200.params import particles_set
from tests.common import compare_masks, compare_particles, copy_oracle_to_lattice, rel_l2

pytestmark = pytest.mark.gpu

MACROS = ["rho", "ux", "uy", "uz", "rho_N"]


def fast_run(w, steps, storage="fp64", with_oracle=True):
    p = w.params.copy()
    p.storage = {"fp64": 0, "fp32": 1, "fp16": 2}[storage]
    o = orc_setup(w)
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    L.step(steps)
    L.call("calmacros")
    if with_oracle:
        o.step(steps)
        o.call("calmacros")
    return o, L


def errors(o, L, fields=MACROS, mask=None):
    """Relative L2 error per field; velocity as one vector field (a component
    that is symmetry noise is measured against the flow, not itself)."""
    out = {}
    m = (lambda a: np.where(mask, a, 0)) if mask is not None else (lambda a: a)
    for f in fields:
        if f in ("ux", "uy", "uz"):
            continue
        out[f] = rel_l2(m(L.get(f)), m(o.arr(f)))
    if any(f in fields for f in ("ux", "uy", "uz")):
        out["u"] = rel_l2(np.stack([m(L.get(k)) for k in ("ux", "uy", "uz")]),
                          np.stack([m(o.arr(k)) for k in ("ux", "uy", "uz")]))
    return out


def test_fast_fp64_c1_1000_steps():
    o, L = fast_run(configs.c1_thread(), 1000)
    e = errors(o, L)
    assert max(e.values()) <= 1e-10, e


def test_fast_fp64_ragged_periodic_domain():
    """Dimensions that are not multiples of the 32x8 tile footprint or the x chunk."""
    w = configs.c1_thread(nx=37, ny=13, nz=45, radius=4.0)
    o, L = fast_run(w, 200)
    e = errors(o, L)
    assert max(e.values()) <= 1e-10, e


@pytest.mark.parametrize("ratio,rates", [(5.0, {}), (0.2, dict(s_e=1.1, s_q=1.3)), (1.0, dict(s_eps=0.9, s_m=1.6))])
def test_fast_fp64_two_viscosities_and_rates(ratio, rates):
    """Node-local rates from the phase field (nu_r != nu_b) and from the
    runtime inputs, against the oracle: the FP64 parity bound, 1e-10."""
    w = configs.c1_thread(nx=21, ny=18, nz=40, radius=5.0)
    w.params.nu_b = w.params.nu_r / ratio
    for k in ("s_e", "s_eps", "s_q", "s_pi", "s_m"):
        setattr(w.params, k, rates.get(k, 0.0))
    o, L = fast_run(w, 200)
    e = errors(o, L)
    assert max(e.values()) <= 1e-10, e


def test_fast_fp64_walls_only():
    w = driven_channel()
    o, L = fast_run(w, 300)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, mask=fluid)
    assert max(e.values()) <= 1e-10, e


def test_fast_fp64_c2_walls_particle_300_steps():
    w = configs.c2_wall_particle(nx=32, ny=32, nz=64, rad=5.0, centre=(16.0, 16.0, 20.0), z0=20.0, z1=44.0)
    o, L = fast_run(w, 300)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, mask=fluid)
    assert max(e.values()) <= 1e-10, e
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])
    compare_particles(o, L, 1, 1e-9, ["center", "up", "rp"])


def test_fast_fp64_c2_interpolated_bounce_back_300_steps():
    """The moving sphere with the interpolated bounce-back of curve2
    (Source1.f90:1036-1101) in the fused path against the oracle."""
    w = configs.c2_wall_particle(nx=32, ny=32, nz=64, rad=5.0, centre=(16.0, 16.0, 20.0), z0=20.0, z1=44.0)
    w.params.bounce = 1
    o, L = fast_run(w, 300)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, mask=fluid)
    assert max(e.values()) <= 1e-10, e
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])
    compare_particles(o, L, 1, 1e-9, ["center", "up", "rp"])


def test_fast_fp64_c2_full_size_1000_steps():
    """The wetting-wall slab with one moving sphere at its full 64x64x128 size."""
    w = configs.c2_wall_particle()
    o, L = fast_run(w, 1000)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, mask=fluid)
    assert max(e.values()) <= 1e-10, e
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])
    compare_particles(o, L, 1, 1e-9, ["center", "up", "rp"])


def test_fast_fp64_mass_conservation():
    """Total mass is conserved to rounding; per-colour mass is not an invariant
    of the reference (Recolor moves a colour's residue below EVAP_LIM to the
    other colour, Source1.f90:718-723), so it is compared with the oracle."""
    w = configs.c1_thread()
    p = w.params.copy()
    L = Lattice(p)
    o = orc_setup(w)
    copy_oracle_to_lattice(o, L)
    m0 = L.mass_momentum()
    L.step(500)
    o.step(500)
    m1 = L.mass_momentum()
    assert abs((m1[0] + m1[1]) - (m0[0] + m0[1])) <= 1e-12 * (m0[0] + m0[1])
    assert abs(m1[0] - o.arr("ri").sum()) <= 1e-11 * m0[0]
    assert abs(m1[1] - o.arr("bi").sum()) <= 1e-11 * m0[1]


def driven_channel():
    """Slab between wetting walls, driven by the body force: a developed flow."""
    w = configs.c2_wall_particle(nx=24, ny=16, nz=48, z0=16.0, z1=32.0)
    w.params.par = 0
    w.particles = []
    w.params.body[2] = -1e-5
    return w


@pytest.mark.parametrize("storage,bound", [("fp32", 1e-4), ("fp16", 1e-3)])
def test_reduced_storage_driven_flow(storage, bound):
    """Velocity error of the reduced storage against the FP64 oracle on a
    developed (body-force driven) two-phase channel flow, 1000 steps, within
    the 1e-3 relative L2 target.  Measured: FP32 2.5e-5, 16-bit 3.8e-4 (the
    FP16 significand of the stored total deviation, 2^-11 relative, sets the
    floor)."""
    o, L = fast_run(driven_channel(), 1000, storage)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, ["ux", "uy", "uz", "rho", "rho_N"], mask=fluid)
    print(f"{storage} driven channel: {e}")
    assert e["u"] <= bound, e
    assert e["rho"] <= bound, e


@pytest.mark.parametrize("storage,bound", [("fp32", 3e-3), ("fp16", 5e-3)])
def test_reduced_storage_early_thread(storage, bound):
    """Early Rayleigh-Plateau thread (C1, 1000 steps): velocities are small
    (~1e-5) and the error is dominated by the seed noise.  Measured: FP32
    1.3e-3, 16-bit 2.0e-3."""
    o, L = fast_run(configs.c1_thread(), 1000, storage)
    e = errors(o, L, ["ux", "uy", "uz", "rho", "rho_N"])
    print(f"{storage} early thread: {e}")
    assert e["u"] <= bound, e


@pytest.mark.parametrize("storage,bound", [("fp32", 3e-3), ("fp16", 5e-3)])
@pytest.mark.parametrize("bounce", [0, 1])
@pytest.mark.parametrize("centre", [(16.0, 16.0, 20.0), (4.6, 31.2, 0.4)])
def test_reduced_storage_walls_and_particle(storage, bound, bounce, centre):
    """Wetting walls and a moving sphere in FP32 arithmetic against the oracle,
    the sphere inside the box and close to a wall across the periodic edges of
    y and z (rows of both halves of a tile, first and last tiles), with either
    bounce-back, 50 steps.  Bounds: those of the early thread, whose velocities
    are smaller."""
    w = configs.c2_wall_particle(nx=32, ny=35, nz=61, rad=3.4, centre=centre, z0=20.0, z1=44.0)
    w.params.bounce = bounce
    o, L = fast_run(w, 50, storage)
    fluid = o.arr("walls_all") == 0
    e = errors(o, L, ["ux", "uy", "uz", "rho", "rho_N"], mask=fluid)
    assert e["u"] <= bound and e["rho"] <= 1e-4 and e["rho_N"] <= bound, e
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])


def test_reduced_storage_breakup_time():
    """Breakup time of the reduced storages within 1 % of FP64's on two
    unstable threads of the batched mix that break within 12,000 steps
    (26x26x244, tau 0.93; 54x54x102, tau 0.81), the three storages run side by
    side as in the precision study; the total mass drifts by less than 1e-5.
    Measured: FP32 0.002-0.003 %, 16-bit 0.035-0.054 %."""
    from symmetry_b200 import study
    ws = {w.name: w for w in study.mix_cases(6)}
    for name in ("c4_002", "c4_012"):
        r = study.run_case(ws[name], max_steps=14000, snap_every=4000, log=None)
        b = r["breakup_step"]
        assert b["fp64"] is not None and b["fp64"] > 0, (name, b)
        for m in ("fp32", "fp16"):
            assert b[m] is not None and abs(b[m] - b["fp64"]) <= 0.01 * b["fp64"], (name, m, b)
        for row in r["snapshots"]:
            for m in ("fp64", "fp32", "fp16"):
                assert abs(row["mass_drift"][m]) <= 1e-5, (name, row)


@pytest.mark.parametrize("storage", ["fp64", "fp16"])
def test_get_macros_leaves_stepping_state_untouched(storage):
    """sym_get_macros on a fused state returns calmacros of the current
    populations and changes nothing: a run that reads the fields midway ends
    bit for bit where an unread run ends, and the fields equal calmacros of
    the exported populations."""
    w = configs.c2_wall_particle(nx=24, ny=24, nz=48, rad=4.0, centre=(12.0, 12.0, 16.0), z0=16.0, z1=32.0)
    w.params.storage = {"fp64": 0, "fp16": 2}[storage]
    from symmetry_b200.lib import setup_workload
    a, b = setup_workload(w), setup_workload(w)
    a.step(30)
    b.step(30)
    m = a.macros()
    a.step(20)
    b.step(20)
    assert np.array_equal(a.get("ri"), b.get("ri")) and np.array_equal(a.get("bi"), b.get("bi"))
    c = setup_workload(w)
    c.step(30)
    m2 = c.macros()
    c.call("calmacros")   # exports the fused state, then the reference calmacros
    fluid = c.get("walls_all") == 0
    for k in ("rho", "ux", "uy", "uz", "rho_N"):
        assert np.array_equal(m[k], m2[k]), k
        ref = c.get(k)
        scale = max(np.abs(ref[fluid]).max(), 1e-300)
        assert np.abs(m[k][fluid] - ref[fluid]).max() <= 1e-12 * scale, k


@pytest.mark.parametrize("rad,centre,up", [
    (3.28, (13.39, 12.67, 13.44), (0.31, -0.30, -0.07)),
    (2.2, (12.3, 11.51, 9.34), (0.38, -0.31, 0.15)),
    (2.61, (13.68, 9.12, 0.11), (0.12, -0.21, -0.38)),
])
def test_fast_fp64_node_uncovered_beside_a_covered_one(rad, centre, up):
    """A sphere that moves by a third of a node uncovers nodes next to nodes it
    covers in the same step.  The uncovered node's refill averages the
    neighbours that were fluid before (walls_old, the newly covered one among
    them).  A heavy sphere keeps its velocity; FP64 parity bounds of this
    file, the masks exact."""
    w = configs.c2_wall_particle(nx=28, ny=25, nz=32, rad=rad, centre=centre, z0=6.0, z1=20.0)
    w.params.mass *= 1e4
    w.params.inertia *= 1e4
    w.particles[0]["up"] = list(up)
    met = False
    for steps in (1, 2, 3):
        o, L = fast_run(w, steps, with_oracle=False)
        before = o.arr("walls_all").copy()
        for _ in range(steps):
            before = o.arr("walls_all").copy()
            o.step(1)
        uncovered = (before > 0) & (o.arr("walls_all") == 0)
        covered = (before == 0) & (o.arr("walls_all") > 0)
        links = [d for d in itertools.product((-1, 0, 1), repeat=3) if 1 <= sum(map(abs, d)) <= 2]
        met = met or any((uncovered & np.roll(covered, d, (0, 1, 2))).any() for d in links)
        o.call("calmacros")
        compare_masks(o, L, ["walls", "walls_old", "walls_all", "pin", "pout"])
        e = errors(o, L, mask=o.arr("walls_all") == 0)
        assert max(e.values()) <= 1e-10, e
        compare_particles(o, L, 1, 1e-9)
        L.close()
    assert met


def wall_layer(side, cita_deg):
    """A noise-free layer along both wetting walls: red (side 1), whose wall
    nodes' normals are exactly opposite to the walls', or blue (side -1),
    exactly parallel."""
    nx, ny, nz = 24, 10, 36
    p = configs.config_params(nx, ny, nz, tau_r=0.9, sigma=5e-3, wall_x=True, cita_deg=cita_deg)
    x = np.arange(nx, dtype=np.float64)[:, None, None]
    phi = side * np.tanh(4.0 - np.minimum(x, nx - 1 - x)) * np.ones((nx, ny, nz))
    o = Oracle(p)
    o.call("set_walls")
    o.init_phase(phi, np.ones_like(phi))
    o.call("derivatives")
    return p, o


@pytest.mark.parametrize("cita_deg", [30.0, 60.0, 90.0, 120.0])
@pytest.mark.parametrize("side", [1, -1])
@pytest.mark.parametrize("storage", [0, 1, 2])
def test_layer_along_a_wetting_wall(storage, side, cita_deg):
    """Contact-angle rotation of a normal opposite or parallel to the wall's:
    finite through 20 steps in every storage, derivatives (FP64 in every
    storage) as the oracle's to the per-call bound 1e-12, and the fused FP64
    step to 1e-10 after one step.  (Later steps multiply rounding: the
    rotation of a normal within 1e-5 of the wall's divides by sin(1e-5).)"""
    p, o = wall_layer(side, cita_deg)
    p.storage = storage
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    L.call("derivatives")
    for f in ("n_x", "n_y", "n_z", "gradx", "grady", "gradz"):
        assert np.abs(L.get(f) - o.arr(f)).max() <= 1e-12, f
    copy_oracle_to_lattice(o, L)
    L.step(1)
    o.step(1)
    m = L.macros()
    assert all(np.isfinite(v).all() for v in m.values())
    if storage == 0:
        fluid = o.arr("walls_all") == 0
        r, b = o.arr("ri").sum(-1), o.arr("bi").sum(-1)
        phi = np.where(fluid, (r - b) / (r + b), 0.0)
        assert np.abs(m["rho_N"] - phi).max() <= 1e-10
    L.step(19)
    assert all(np.isfinite(v).all() for v in L.macros().values())
    L.close()


@pytest.mark.parametrize("storage", ["fp64", "fp16"])
def test_noisy_thread_between_wetting_walls_stays_finite(storage):
    """A served job between wetting walls far from its thread: noise clipped at
    the pure phase leaves a few wall nodes' gradients exactly along the
    normal, opposite to it."""
    w = next(j.workload for j in configs.c5_jobs(storage=storage) if j.workload.name == "c5_0013")
    assert w.params.wall_x and w.params.par == 0
    L = setup_workload(w)
    L.step(20)
    assert all(np.isfinite(v).all() for v in L.macros().values())
    L.close()


def test_fast_sphere_moved_by_hand_refills_its_own_nodes_only():
    """A sphere put elsewhere between steps leaves marks outside its new
    surroundings behind (until set_walls).  A node uncovered there is next to
    those marks but not to the particle (pout 0): its densities stay as they
    were, and no node gets any that is not next to the particle."""
    w = configs.c2_wall_particle(nx=30, ny=24, nz=26, rad=3.1, centre=(11.7, 9.9, 6.9), z0=6.0, z1=18.0)
    w.params.mass *= 1e4
    w.params.inertia *= 1e4
    w.particles[0]["up"] = [0.2, -0.18, 0.19]
    L = setup_workload(w)
    s = L.particles()
    particles_set(s, "center", 1, [(19.5, 2.46, 14.0)])
    L.set_particles(s)
    before = {f: L.get(f).copy() for f in ("rho_R", "rho_B")}
    L.step(1)
    left = (L.get("walls_old") > 0) & (L.get("walls_all") == 0) & (L.get("pout") == 0)
    assert left.any()
    for f, v in before.items():
        assert np.array_equal(L.get(f)[left], v[left]), f


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16"])
def test_not_a_number_spreads_as_in_the_reference(storage, bad):
    """A population that is not finite reaches one node further a step, by
    streaming: a gradient taken from it is none (the reference's comparison
    with EVAP_LIM), so it does not reach the neighbours' curvature.  The nodes
    without a number are the oracle's, rows of both halves of a tile among
    them."""
    w = configs.c1_thread(nx=24, ny=21, nz=40, radius=5.0)
    p = w.params.copy()
    p.storage = {"fp64": 0, "fp32": 1, "fp16": 2}[storage]
    o = orc_setup(w)
    for at in ((9, 3, 7), (14, 11, 33)):
        o.arr("ri")[at + (0,)] = bad
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    for _ in range(3):
        L.step(1)
        o.step(1)
        with np.errstate(all="ignore"):
            want = ~np.isfinite(o.arr("ri").sum(-1) + o.arr("bi").sum(-1))
        assert np.array_equal(~np.isfinite(L.macros()["rho"]), want)
    assert want.any() and not want.all()
