"""GPU parity of the reference-structured kernels (one library call per
reference subroutine) against the CPU oracle.

The canonical kernels are compiled without fused multiply-add, so outside the
transcendental calls (acos/sin/cos in the wetting rotation and the Lagrange
points, tanh in the initial state) they round exactly like the oracle.
Tolerances: per-subroutine 1e-12 max-relative; after many steps the field
relative L2 error <= 1e-10 (the FP64 parity target), masks bit-exact, particle
trajectories <= 1e-9.
"""
import numpy as np
import pytest

from oracle.oracle import Oracle, setup_reference, setup_workload as orc_setup
from symmetry_b200 import configs, params
from symmetry_b200.lib import Lattice, setup_workload
from tests.common import (MASKS, SCALARS, compare_fields, compare_masks, compare_particles,
                          copy_oracle_to_lattice, rel_l2)

pytestmark = pytest.mark.gpu

SEQUENCE = ["calmacros", "lagrange_points", "capillary_force2", "momentum", "repulsive", "movement",
            "set_walls", "refilling", "derivatives", "collision", "recolor", "boundary",
            ("streaming", 0), ("streaming", 1), "curve"]
POPS = ["ri", "bi", "fi", "ffi"]


def small_c2():
    return configs.c2_wall_particle(nx=32, ny=32, nz=64, rad=5.0, centre=(16.0, 16.0, 20.0),
                                    z0=20.0, z1=44.0, steps=300)


def small_c1():
    return configs.c1_thread(nx=16, ny=16, nz=48, radius=4.0)


def small_c2_interp():
    w = small_c2()
    w.params.bounce = 1   # curve2, Source1.f90:1036-1101
    return w


def cases():
    return {
        "c1": lambda: orc_setup(small_c1()),
        "c2": lambda: orc_setup(small_c2()),
        "c2_interp": lambda: orc_setup(small_c2_interp()),
        "ref": lambda: setup_reference(params.reference_params(48, 88, 48)),
    }


@pytest.mark.parametrize("case", ["c1", "c2", "c2_interp", "ref"])
def test_subroutine_parity(case):
    o = cases()[case]()
    L = Lattice(o.p)
    copy_oracle_to_lattice(o, L)
    par = o.p.par
    for step in range(2):
        for sub in SEQUENCE:
            if isinstance(sub, tuple):
                o.streaming(sub[1]); L.streaming(sub[1]); name = f"streaming{sub[1]}"
            else:
                if par == 0 and sub in ("lagrange_points", "capillary_force2", "momentum", "repulsive",
                                        "movement", "refilling"):
                    continue
                o.call(sub); L.call(sub); name = sub
            try:
                compare_fields(o, L, SCALARS + POPS, 1e-12)
                compare_masks(o, L)
                if par:
                    compare_particles(o, L, par, 1e-11)
            except AssertionError as e:
                raise AssertionError(f"{case} step {step} after {name}: {e}")


def test_lagrange_points_parity():
    o = setup_reference(params.reference_params(48, 88, 48))
    L = Lattice(o.p)
    copy_oracle_to_lattice(o, L)
    o.call("calmacros"); L.call("calmacros")
    o.call("lagrange_points"); L.call("lagrange_points")
    g = L.lagrange()
    for k in ["Lax", "Lay", "Laz", "ds", "La_rhoN", "La_nx", "La_ny", "La_nz"]:
        a, b = g[k], o.arr(k)
        assert np.abs(a - b).max() <= 1e-11 * max(1.0, np.abs(b).max()), k
    assert (g["La_flag"] == o.arr("La_flag")).all()
    s = L.particles()
    assert np.allclose(list(s.shb)[:12], list(o.particles.shb)[:12], rtol=1e-12, atol=0)


def canonical_steps(L, n):
    """The reference loop body through the per-subroutine entry points
    (CONFIG-mode sym_step would run the fused path instead)."""
    for _ in range(n):
        for sub in SEQUENCE:
            if isinstance(sub, tuple):
                L.streaming(sub[1])
            elif L.p.par == 0 and sub in ("lagrange_points", "capillary_force2", "momentum", "repulsive",
                                          "movement", "refilling"):
                continue
            else:
                L.call(sub)


def _run_pair(w, steps):
    o = orc_setup(w)
    L = Lattice(w.params)
    phi, rho = w.phase()
    if w.params.par:
        copy_oracle_to_lattice(o, L)     # identical start, particles included
    else:
        L.call("set_walls")
        L.init_phase(phi, rho)
        L.call("derivatives")
    o.step(steps)
    canonical_steps(L, steps)
    o.call("calmacros")
    L.call("calmacros")
    return o, L


def test_c1_thread_1000_steps():
    """Plain FP64, periodic Rayleigh-Plateau thread 32x32x96, 1000 steps."""
    w = configs.c1_thread()
    o, L = _run_pair(w, 1000)
    for f in ["rho", "ux", "uy", "uz", "rho_N"]:
        e = rel_l2(L.get(f), o.arr(f))
        assert e <= 1e-10, (f, e)


def test_c2_walls_particle_300_steps():
    """Wetting walls (60 deg) + moving sphere, FP64, 32x32x64, 300 steps."""
    w = small_c2()
    o, L = _run_pair(w, 300)
    fluid = o.arr("walls_all") == 0
    for f in ["rho", "ux", "uy", "uz", "rho_N"]:
        e = rel_l2(np.where(fluid, L.get(f), 0), np.where(fluid, o.arr(f), 0))
        assert e <= 1e-10, (f, e)
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])
    compare_particles(o, L, 1, 1e-9, ["center", "up", "rp"])


def test_reference_mode_200_steps():
    """The reference's own geometry (mirrors, x=1/z=1 walls, 12 particles), 48x88x48, 200 steps."""
    p = params.reference_params(48, 88, 48)
    o = setup_reference(p)
    L = Lattice(p)
    L.initia_center()
    L.call("set_walls")
    L.initialization()
    L.call("derivatives")
    compare_masks(o, L)
    compare_particles(o, L, 12, 1e-13, ["center", "center0"])
    compare_fields(o, L, ["rho_N", "rho", "ri", "bi"], 1e-13)
    o.step(200)
    L.step(200)
    for f in ["rho", "ux", "uy", "uz", "rho_N"]:
        e = rel_l2(L.get(f), o.arr(f))
        assert e <= 1e-10, (f, e)
    compare_masks(o, L, ["walls", "walls_all", "pin", "pout"])
    compare_particles(o, L, 12, 1e-9, ["center", "up", "rp"])
    h1, y1 = L.output3()
    h2, y2 = o.output3()
    assert y1 == y2 and abs(h1 - h2) <= 1e-9 * abs(h2)


def test_device_init_thread_matches_host_generator():
    w = configs.c1_thread()
    L = setup_workload(w)
    phi, rho = w.phase()
    assert np.abs(L.get("rho_N") - phi).max() <= 1e-13
    assert np.abs(L.get("rho") - rho).max() <= 1e-13
    o = orc_setup(w)
    compare_fields(o, L, ["ri", "bi"], 1e-13)


def test_mass_conservation_and_diagnostics():
    """Total mass is conserved; per-colour mass matches the oracle (it is not
    itself invariant: Recolor, Source1.f90:718-723)."""
    w = configs.c1_thread()
    L = setup_workload(w)
    o = orc_setup(w)
    m0 = L.mass_momentum()
    canonical_steps(L, 200)
    o.step(200)
    m1 = L.mass_momentum()
    assert abs((m1[0] + m1[1]) - (m0[0] + m0[1])) <= 1e-12 * (m0[0] + m0[1])
    assert abs(m1[0] - o.arr("ri").sum()) <= 1e-12 * m0[0]
    L.call("calmacros")
    o.call("calmacros")
    assert abs(L.neck_radius() - o.neck_radius()) <= 1e-10


@pytest.mark.parametrize("runs", [(1, 1, 1), (2, 1), (3,), (1, 2)])
def test_reference_steps_leave_every_array(runs):
    """A run of whole steps merges passes over the populations and writes some
    arrays in its last step only; however the steps are split into runs, every
    array ends as the oracle's (the FP64 parity targets of this file: relative
    L2 1e-10, masks exact, particles 1e-9).  The normals are held through the
    gradients, |grad phi| n: a unit vector of a gradient just above 1e-8, in the
    tails of the interface, has an absolute error of 1e-16 / 1e-8 in any FP64
    evaluation."""
    p = params.reference_params(48, 88, 48)
    o = setup_reference(p)
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    o.step(sum(runs))
    for n in runs:
        L.step(n)
    compare_masks(o, L)
    for f in [f for f in SCALARS if f not in ("n_x", "n_y", "n_z")] + POPS:
        e = rel_l2(L.get(f), o.arr(f))
        assert e <= 1e-10, (f, e)
    compare_particles(o, L, 12, 1e-9)


def test_reference_run_covers_and_refills_nodes():
    """Inside a run the streamed populations of a node are stored only next to
    solids; particles that move half a node per step cover nodes whose
    populations were not stored and uncover others, in every kind of step of a
    run.  The same parity targets as above."""
    p = params.reference_params(48, 88, 48)
    o = setup_reference(p)
    s = o.particles
    params.particles_set(s, "up", 12, [(-0.5 + 0.02 * k, 0.04 * k - 0.2, -0.45) for k in range(12)])
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    before = L.get("walls_all").copy()
    o.step(6)
    L.step(6)
    compare_masks(o, L)
    after = L.get("walls_all")
    assert ((before > 0) & (after == 0)).any() and ((before == 0) & (after > 0)).any()
    for f in [f for f in SCALARS if f not in ("n_x", "n_y", "n_z")] + POPS:
        e = rel_l2(L.get(f), o.arr(f))
        assert e <= 1e-10, (f, e)
    compare_particles(o, L, 12, 1e-9)


@pytest.mark.parametrize("minority", ["bi", "ri"])
@pytest.mark.parametrize("steps", [1, 2])
def test_reference_step_at_the_evaporation_limit(steps, minority):
    """A colour of density 1e-8 (1 +- 1e-11) in one of density 0.05: whether it
    is above EVAP_LIM decides if a node's minority colour empties, so each
    colour's density must have its own 16 digits.  A wrong decision is off by
    1e-8 w_i; a right one to the rounding of the majority's populations."""
    p = params.reference_params(20, 24, 22)
    p.par = 0
    o = Oracle(p)
    rng = np.random.default_rng(8)
    shape = (p.nx, p.ny, p.nz)
    small = 1e-8 * (1.0 + 1e-11 * rng.uniform(0.1, 1.0, shape) * rng.choice([-1.0, 1.0], shape))
    large = 0.05 * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, shape))
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    o.call("set_walls")
    o.init_phase(np.ones(shape), np.full(shape, p.rho0))
    o.call("derivatives")
    f = w * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, shape + (19,)))
    f /= f.sum(-1, keepdims=True)
    o.arr(minority)[...] = f * small[..., None]
    o.arr("ri" if minority == "bi" else "bi")[...] = f * large[..., None]
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    o.step(1)
    emptied = (o.arr(minority) == 0.0).mean()   # the oracle's first step decides both ways
    assert 0.05 < emptied < 0.95
    o.step(steps - 1)
    L.step(steps)
    assert np.abs(L.get(minority) - o.arr(minority)).max() <= 1e-14


@pytest.mark.parametrize("bounce", [0, 1])
def test_reference_steps_between_streaming_calls(bounce):
    """Streaming one colour leaves the arrays in another arrangement, and a
    handle keeps a bounded number of captured steps: runs of 1 to 9 steps
    between single streaming calls meet every arrangement of the arrays, more
    than are kept.  Every run has the oracle's result, relative L2 1e-10."""
    p = params.reference_params(9, 7, 8)
    p.par, p.bounce = 0, bounce
    o = Oracle(p)
    rng = np.random.default_rng(4)
    shape = (p.nx, p.ny, p.nz)
    o.call("set_walls")
    o.init_phase(0.02 * rng.uniform(-1.0, 1.0, shape), p.rho0 * (1.0 + 1e-3 * rng.uniform(-1.0, 1.0, shape)))
    o.call("derivatives")
    L = Lattice(p)
    for k in range(60):
        which, n = int(rng.integers(2)), int(rng.integers(1, 10))
        copy_oracle_to_lattice(o, L)
        for s in (o, L):
            s.streaming(which)
            s.step(n)
        for f in ("ri", "bi", "rho", "rho_N"):
            assert rel_l2(L.get(f), o.arr(f)) <= 1e-10, (k, f)


@pytest.mark.parametrize("moved,runs", [("by hand", (1, 1, 1)), ("by hand", (2, 2)), ("by hand", (1, 3)),
                                        ("by velocity", (1, 1, 1, 1)), ("by velocity", (4,)), ("by velocity", (3, 1))])
def test_reference_particles_that_jump(moved, runs):
    """Particles that move by about a node at once uncover nodes next to no
    particle, which nothing refills: the reference collides what their arrays
    were left with when they were covered.  Placed by hand between calls, or
    moving inside them; heavy particles.  The parity targets of this file."""
    p = params.reference_params(36, 42, 36)
    p.par, p.rad = 2, 4.0
    p.mass, p.inertia = 1e6 * p.mass, 1e6 * p.inertia
    at = np.array([(17.3, 13.0, 18.0), (18.0, 30.5, 16.2)])
    hand = np.array([(-1.22, 0.13, -0.23), (-0.61, 0.34, 1.08)]) * (moved == "by hand")
    up = np.array([(-0.27, 0.04, -0.99), (-0.83, -0.45, -0.13)]) * (moved == "by velocity")
    o = Oracle(p)
    params.particles_set(o.particles, "center", 2, at.tolist())
    params.particles_set(o.particles, "center0", 2, at.tolist())
    params.particles_set(o.particles, "up", 2, up.tolist())
    o.call("set_walls")
    o.call("initialization")
    o.call("derivatives")
    L = Lattice(p)
    copy_oracle_to_lattice(o, L)
    unfilled = 0
    for k, n in enumerate(runs):
        if k and moved == "by hand":
            s = L.particles()
            for q in (o.particles, s):
                params.particles_set(q, "center", 2, (at + k * hand).tolist())
            L.set_particles(s)
        L.step(n)
        for _ in range(n):
            o.step(1)
            unfilled += int(((o.arr("walls_old") > 0) & (o.arr("walls_all") == 0) & (o.arr("pout") == 0)).sum())
    assert unfilled
    compare_masks(o, L, ["walls", "walls_old", "walls_all", "pin", "pout"])
    for f in [f for f in SCALARS if f not in ("n_x", "n_y", "n_z")] + POPS:
        e = rel_l2(L.get(f), o.arr(f))
        assert e <= 1e-10, (f, e)
    compare_particles(o, L, 2, 1e-9)
