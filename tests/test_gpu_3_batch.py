"""Batches: uneven domains stepped by one persistent launch per kernel.

Each domain's result in a batch must equal its result stepped alone (same
kernels, same tiles), for every storage mode, including domains with walls
and particles and after the batch is rebuilt because a member was read back
between batch steps.
"""
import numpy as np
import pytest

from symmetry_b200 import configs
from symmetry_b200.lib import Batch, Server, job_spec, setup_workload
from symmetry_b200.params import particles_get

pytestmark = pytest.mark.gpu


def mix(storage):
    c4 = [w for w in configs.c4_manifest(n_domains=12, storage=storage) if w.params.par][:1]
    for w in c4:   # keep the test small: shorten the domain along z
        w.params.nz = min(w.params.nz, 96)
        w.gen["wavelength"] = float(w.params.nz)
        w.particles[0]["center"][2] = w.params.nz / 2.0
    return [
        configs.c1_thread(nx=20, ny=20, nz=64, radius=4.0, storage=storage),
        configs.c1_thread(nx=37, ny=13, nz=45, radius=4.0, storage=storage),
        configs.c2_wall_particle(nx=24, ny=24, nz=48, rad=4.0, centre=(12.0, 12.0, 16.0), z0=16.0, z1=32.0,
                                 storage=storage),
    ] + c4


def state(L):
    s = L.particles()
    return (L.get("ri"), L.get("bi"),
            np.array(particles_get(s, "center", L.p.par)) if L.p.par else None)


@pytest.mark.parametrize("storage", ["fp64", "fp16"])
def test_batch_equals_alone(storage):
    ws = mix(storage)
    alone = [setup_workload(w) for w in ws]
    for L in alone:
        L.step(25)
    _ = alone[0].get("rho_N")
    for L in alone:
        L.step(15)
    members = [setup_workload(w) for w in ws]
    B = Batch(members)
    B.step(25)
    # read back mid-run (the batch must rebuild; the 16-bit export/import
    # round trip re-encodes values, so the alone run above does the same)
    _ = members[0].get("rho_N")
    B.step(15)
    for w, a, m in zip(ws, alone, members):
        ra, ba, ca = state(a)
        rm, bm, cm = state(m)
        assert np.array_equal(ra, rm) and np.array_equal(ba, bm), w.name
        if ca is not None:
            assert np.array_equal(ca, cm), w.name
    B.close()


def test_batch_autotune_and_info():
    ws = mix("fp16")
    members = [setup_workload(w) for w in ws]
    B = Batch(members)
    taken = B.autotune(trial_steps=2)
    assert taken > 0
    for i in range(len(members)):
        assert B.xchunk(i) in (8, 12, 16, 24, 32, 64)
    info = B.info()
    assert info["nodes"] == sum(w.nodes for w in ws) and info["tiles"] > 0 and info["grid"] >= 148
    # stepping after tuning still matches a domain stepped alone with the same tiles
    B.step(3)
    B.close()


def test_batch_grid_size_does_not_change_results():
    """The persistent collide grid (resident CTAs per SM, an autotuning knob)
    changes which CTA takes which tile, never a tile's result."""
    ws = mix("fp64")
    runs = []
    for per_sm in (None, 1):
        members = [setup_workload(w) for w in ws]
        B = Batch(members)
        if per_sm:
            B.set_ctas_per_sm(per_sm)
            assert B.info()["grid"] % per_sm == 0
        B.step(12)
        runs.append([state(m) for m in members])
        B.close()
    for w, a, b in zip(ws, runs[0], runs[1]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), w.name


@pytest.mark.parametrize("storage", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("xchunk", [1, 5, 64])
def test_tile_extent_does_not_change_results(storage, xchunk):
    """The x extent of the collide tiles (one plane, a remainder, a whole
    domain) never changes a result: FP64's accumulated densities are integer
    sums of terms that do not depend on where a march starts.  Exact: equal
    bit for bit to each domain stepped alone with its own extent."""
    ws = mix(storage)
    alone = [setup_workload(w) for w in ws]
    for L in alone:
        L.step(9)
    members = [setup_workload(w) for w in ws]
    B = Batch(members)
    for i in range(len(members)):
        B.set_xchunk(i, xchunk)
    B.step(9)
    for w, a, m in zip(ws, alone, members):
        ra, ba, ca = state(a)
        rm, bm, cm = state(m)
        assert np.array_equal(ra, rm) and np.array_equal(ba, bm), w.name
    B.close()


@pytest.mark.parametrize("storage", ["fp64", "fp16"])
@pytest.mark.parametrize("n", [16, 17, 130])
def test_batch_sizes_of_the_descriptor_tables(storage, n):
    """A batch's descriptors are kernel parameters in a small or a large table,
    or in global memory beyond it: at the tables' edges each domain's result
    equals the one it gets alone, bit for bit."""
    ws = [configs.c1_thread(nx=6 + k % 5, ny=7 + k % 3, nz=9 + k % 7, radius=2.0, storage=storage) for k in range(n)]
    members = [setup_workload(w) for w in ws]
    B = Batch(members)
    B.step(4)
    for k in sorted({0, 1, n // 2, n - 2, n - 1}):
        a = setup_workload(ws[k])
        a.step(4)
        assert np.array_equal(a.get("ri"), members[k].get("ri")), k
        assert np.array_equal(a.get("bi"), members[k].get("bi")), k
    B.close()


@pytest.mark.parametrize("storage,rows", [("fp64", 8), ("fp32", 16), ("fp16", 16)])
def test_long_marches_do_not_change_results(storage, rows):
    """Long marches along x (the rings of phi, normals and reference pairs used
    over and over, densities carried over many planes) are taken only where a
    batch has columns enough to fill the GPU with them.  With one CTA per SM a
    domain of 1,520 columns of 40 planes is marched whole; the domains beside
    it (walls and sphere, and more planes than one tile) share its extent.
    Exact: every extent gives the same populations bit for bit, and those of
    the domains stepped alone with their own short tiles."""
    big = configs.c1_thread(nx=40, ny=40 * rows, nz=1216, radius=9.0, storage=storage)
    ws = [
        configs.c2_wall_particle(nx=40, ny=27, nz=45, rad=4.0, centre=(20.3, 12.1, 16.0), z0=16.0, z1=32.0,
                                 storage=storage),
        configs.c1_thread(nx=83, ny=19, nz=37, radius=4.0, storage=storage),
    ]
    sms = 148

    def columns(w):
        return -(-w.params.ny // rows) * -(-w.params.nz // 32)

    runs, fields = [], []
    for cap in (64, 5):
        members = [setup_workload(w) for w in [big] + ws]
        B = Batch(members)
        B.set_ctas_per_sm(1)
        for i in range(len(members)):
            B.set_xchunk(i, cap)
        B.step(7)
        info = B.info()
        assert info["grid"] == sms
        tiles = {64: [1, 1, 3], 5: [8, 8, 17]}[cap]   # of 40, 40 and 83 planes
        assert info["tiles"] == sum(t * columns(w) for t, w in zip(tiles, [big] + ws)), info
        runs.append([state(m) for m in members[1:]])
        fields.append(members[0].macros())
        B.close()
        for m in members:
            m.close()
    for k in fields[0]:
        assert np.array_equal(fields[0][k], fields[1][k]), k
    for w, long, short in zip(ws, *runs):
        L = setup_workload(w)
        L.step(7)
        for a, b, c in zip(long, short, state(L)):
            if a is not None:
                assert np.array_equal(a, b) and np.array_equal(a, c), w.name


def test_tile_extent_without_a_limit():
    """An extent far beyond any domain (a caller's "no limit") costs nothing
    and changes nothing, in a batch and in the server."""
    w = configs.c1_thread(nx=20, ny=20, nz=64, radius=4.0)
    alone, member = setup_workload(w), setup_workload(w)
    alone.step(6)
    B = Batch([member])
    B.set_xchunk(0, 2 ** 31 - 1)
    B.step(6)
    assert B.xchunk(0) == 2 ** 31 - 1
    assert np.array_equal(alone.get("ri"), member.get("ri"))
    B.close()
    done = []
    for x in (None, 2 ** 31 - 1):
        S = Server(slots=2, check_every=10)
        for size_class in range(3):
            if x:
                S.set_xchunk(size_class, x)
        i = S.submit(job_spec(w, 20))
        S.run_until_idle()
        done.append(S.result(i))
        S.close()
    assert done[0].status == done[1].status == 3 and done[0].steps == done[1].steps == 20
