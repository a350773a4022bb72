"""The team integrator (a warp's lanes per filament, one or two sites a lane)
against the CPU oracle, bit for bit, at the sizes where its layout changes:
filaments that fill a warp or leave one lane, the shortest ones, warps whose
last filaments are missing, two sites a lane with odd and even site counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(n_dim, n_seg, side, seed, min_bond_length=0.666):
    """Straight filaments on a grid with random directions: (system,
    filaments, sites) for bond counts n_seg."""
    rng = np.random.default_rng(seed)
    n = len(n_seg)
    per = int(np.ceil(n ** (1.0 / n_dim)))
    cells = np.stack(np.meshgrid(*[np.arange(per)] * n_dim, indexing="ij"), -1).reshape(-1, n_dim)
    length = np.maximum(n_seg * 1.5 * min_bond_length, 5.0)
    sites = []
    for i in range(n):
        u = rng.normal(size=n_dim)
        u /= np.linalg.norm(u)
        head = np.zeros(3)
        head[:n_dim] = (cells[i] + 0.5) * side / per - 0.5 * side
        step = np.zeros(3)
        step[:n_dim] = u * length[i] / n_seg[i]
        sites.append(head + np.arange(n_seg[i] + 1)[:, None] * step)
    system = dict(n_dim=n_dim, system_radius=0.5 * side, delta=1e-4, seed=seed)
    fils = [dict(length=float(l) * (1 + 1e-12), persistence_length=100.0, diameter=1.0,
                 min_bond_length=min_bond_length, friction_ratio=2.0) for l in length]
    return system, fils, np.concatenate(sites)


# (dimensions, bond counts, side): one site a lane ...
CASES = {
    "shortest": (3, [2] * 23, 40.0),
    "full_warp": (3, [31, 31, 30, 5], 60.0),
    "ragged": (2, [5, 31, 16, 7, 40, 9, 15, 16, 30, 6, 70, 5], 120.0),
    # ... and two, where that saves more than half the warps of a full chip.
    "two_odd_2d": (2, [16] * 3050, 900.0),
    "two_even_3d": (3, [17] * 3001, 260.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_team_integrator_bitwise(name):
    import simcore_b200 as sc
    from checkers import Oracle
    n_dim, n_seg, side = CASES[name]
    system, fils, sites = _lattice(n_dim, np.array(n_seg), side, seed=5,
                                   min_bond_length=2.0 if name == "shortest" else 0.666)
    assert [sc.filament_n_bonds(f) for f in fils] == n_seg
    ctx = sc.Context(system, fils, sites, precision="fp64")
    oracle = Oracle(system, fils, sites)
    for captured in (False, True):
        (ctx.step_graph if captured else ctx.step)(4)
        oracle.step(4)
        assert np.array_equal(ctx.sites(), oracle.sites())
        assert np.array_equal(ctx.random_forces(), oracle.random_forces())
    ctx.close()
    oracle.close()


@pytest.mark.parametrize("name", ["full_warp", "two_odd_2d", "two_even_3d"])
def test_fast_team_close_to_exact(name):
    """Without noise the fast variant differs from the exact one by FP64
    rounding alone: 1e-12 in the positions (about 100, rounding 1e-14, a few
    steps of the implicit tension solve)."""
    import simcore_b200 as sc
    n_dim, n_seg, side = CASES[name]
    system, fils, sites = _lattice(n_dim, np.array(n_seg), side, seed=6)
    system = dict(system, stoch_flag=0)
    got = []
    for fast in (False, True):
        ctx = sc.Context(system, fils, sites, precision="mixed")
        ctx.set_fast_integrator(fast)
        ctx.step(4)
        got.append(ctx.sites())
        ctx.close()
    assert np.abs(got[0] - got[1]).max() <= 1e-12 * max(1.0, side / 100.0)


def test_division_by_shared_reciprocal_special_values():
    """Straight, unloaded filaments without noise: every right-hand side is
    zero and the cosines are one, so the exact solves meet zero numerators."""
    import simcore_b200 as sc
    from checkers import Oracle
    system, fils, sites = _lattice(3, np.array([7, 12, 31]), 60.0, seed=9)
    system = dict(system, stoch_flag=0)
    ctx = sc.Context(system, fils, sites, precision="fp64")
    oracle = Oracle(system, fils, sites)
    ctx.step(6)
    oracle.step(6)
    assert np.array_equal(ctx.sites(), oracle.sites())
    ctx.close()
    oracle.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_packed_units_keep_systems_apart(precision):
    """Uneven filaments are packed into warps and blocks by size, within their
    system: each of two systems in one context gives the bits it gives alone
    (long filaments in both precisions' blocks, a system without any)."""
    import simcore_b200 as sc
    parts = [_lattice(2, np.array([5, 40, 31, 70, 9, 35, 33, 100, 8, 32]), 330.0, seed=3),
             _lattice(2, np.array([12, 7, 30, 5]), 90.0, seed=4)]
    fils = parts[0][1] + parts[1][1]
    sites = np.concatenate([parts[0][2], parts[1][2]])
    replicas = [dict(system_radius=p[0]["system_radius"], seed=p[0]["seed"],
                     n_filaments=len(p[1])) for p in parts]
    both = sc.Context(parts[0][0], fils, sites, precision=precision, replicas=replicas)
    both.step(3)
    both.step_graph(4)
    alone = []
    for system, f, x in parts:
        ctx = sc.Context(system, f, x, precision=precision)
        # One block size for all: the mixed blocks' noise follows it.
        ctx.set_integrator_layout(32, 128)
        ctx.step(3)
        ctx.step_graph(4)
        alone.append(ctx.sites())
        ctx.close()
    assert np.array_equal(both.sites(), np.concatenate(alone))
    both.close()


@pytest.mark.parametrize("n_fil", [3, 12, 70])
def test_long_pair_lists_bitwise(n_fil):
    """Bundles whose bonds have up to about 10, 40 and 230 pairs: the entries
    of a bond are sorted by its thread, by its warp, or in memory, and its
    forces are added in pair order."""
    import simcore_b200 as sc
    from checkers import Oracle
    rng = np.random.default_rng(n_fil)
    sites = []
    for i in range(n_fil):
        head = np.array([0.013 * i, 0.4 * rng.random(), 0.0])
        sites.append(head + np.arange(6)[:, None] * np.array([0.0, 0.0, 1.0]))
    fils = [dict(length=5.0 * (1 + 1e-12), persistence_length=100.0, diameter=1.0,
                 min_bond_length=0.666, friction_ratio=2.0)] * n_fil
    system = dict(n_dim=3, system_radius=12.0, delta=1e-7, seed=1)
    ctx = sc.Context(system, fils, np.concatenate(sites), precision="fp64")
    oracle = Oracle(system, fils, np.concatenate(sites))
    ctx.step(2)
    oracle.step(2)
    most = np.bincount(ctx.pairs().ravel()).max()
    assert most > {3: 2, 12: 16, 70: 128}[n_fil]
    assert np.array_equal(ctx.pairs(), oracle.pairs())
    for got, want in zip(ctx.bond_forces(), oracle.bond_forces()):
        assert np.array_equal(got, want)
    assert np.array_equal(ctx.sites(), oracle.sites())
    ctx.close()
    oracle.close()


@pytest.mark.parametrize("blocks", [(256, 224), (128, 96)])
def test_layouts_of_two_contexts(blocks):
    """Contexts with different block sizes share compiled kernels; the second
    one's smaller shared memory does not become the first one's limit."""
    import simcore_b200 as sc
    from checkers import Oracle
    # Two-bond filaments: as much shared memory a block as its size allows.
    system, fils, sites = _lattice(3, np.array([2] * 400), 60.0, seed=9, min_bond_length=2.0)
    ctxs = []
    for size in blocks:
        ctxs.append(sc.Context(system, fils, sites, precision="fp64"))
        ctxs[-1].set_integrator_layout(0, size)
    oracle = Oracle(system, fils, sites)
    oracle.step(4)
    for ctx in ctxs:
        ctx.step_graph(4)
        assert np.array_equal(ctx.sites(), oracle.sites())
    for ctx in ctxs:
        ctx.close()
    oracle.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name,scale", [("A", 0.05), ("B", 0.0204), ("B", 0.0206), ("E", 0.026)])
def test_chained_runs_match_host_path(name, scale, precision):
    """Small contexts' captured runs, launched without conditional nodes, take
    the bits, lists and rebuild counts of host-driven steps: fewer bonds than
    one block of the control kernel, just below and above one pass of its
    cluster (4,096 bonds), and buckling filaments whose list outgrows its
    storage inside a run."""
    import simcore_b200 as sc
    from simcore_b200 import workloads
    cfg = workloads.make(name, scale=scale, seed=4, **(dict(n_seg=40) if name == "E" else {}))
    a, b = (sc.Context(*cfg[:3], precision=precision) for _ in range(2))
    for n in ((400,) if name == "E" else (40, 1, 23)):
        a.step_graph(n)
        b.step(n)
        assert np.array_equal(a.sites(), b.sites())
        assert all(np.array_equal(x, y) for x, y in zip(a.pairs(), b.pairs()))
        ca, cb = a.counters(), b.counters()
        assert (ca.i_step, ca.n_rebuilds) == (cb.i_step, cb.n_rebuilds)
    assert name == "A" or ca.n_rebuilds > 1
    assert name != "E" or ca.n_list_regrowths > 0
    a.close()
    b.close()


def test_mixed_lengths_repeated_runs_bitwise():
    """A step of a mixed-length context is a block kernel and a team kernel on
    one pair stage's slots, their launches overlapping: runs in every form take
    the oracle's bits, each time."""
    import simcore_b200 as sc
    from checkers import Oracle
    rng = np.random.default_rng(8)
    n_seg = rng.integers(5, 90, size=240)
    system, fils, sites = _lattice(3, n_seg, 100.0, seed=8)
    oracle = Oracle(system, fils, sites)
    want = []
    for _ in range(4):
        oracle.step(10)
        want.append((oracle.sites(), oracle.bond_forces()))
    assert len(oracle.pairs()) > 2000
    for _ in range(6):
        ctx = sc.Context(system, fils, sites, precision="fp64")
        for i, (x, (f, t)) in enumerate(want):
            (ctx.step_graph if i % 2 else ctx.step)(10)
            assert np.array_equal(ctx.sites(), x)
            gf, gt = ctx.bond_forces()
            assert np.array_equal(gf, f) and np.array_equal(gt, t)
        ctx.close()
    oracle.close()


def test_autotune_cache_of_other_kernels_is_not_read(tmp_path):
    """A cached choice made for earlier integrator kernels (the third version
    of the cache) is left alone, and the shape is timed again."""
    import simcore_b200 as sc
    system, fils, sites = _lattice(3, np.array([10] * 200), 60.0, seed=2)
    cache = tmp_path / "tune.txt"
    a = sc.Context(system, fils, sites, precision="fp64")
    lay = a.autotune(str(cache))
    line = cache.read_text()
    key = line.split("|", 1)[1]
    other = "0 512 1.00 128"
    cache.write_text("v3|" + key.split("\t")[0] + "\t" + other + "\n")
    b = sc.Context(system, fils, sites, precision="fp64")
    b.autotune(str(cache))
    lines = cache.read_text().splitlines()
    assert len(lines) == 2 and lines[1].split("\t")[0] == line.split("\t")[0]
    # Each context goes on as an untuned one.
    c = sc.Context(system, fils, sites, precision="fp64")
    for ctx in (a, b, c):
        ctx.step(3)
        ctx.step_graph(4)
    assert np.array_equal(a.sites(), c.sites()) and np.array_equal(b.sites(), c.sites())
    assert lay[0] in (0, 32)


def test_noise_precision_follows_the_system():
    """The fast blocks of a system whose longest filaments have 33 sites draw
    the noise in FP32, whatever the other systems of the context hold: each of
    two systems gives the bits it gives alone with the same block size."""
    import simcore_b200 as sc
    parts = [_lattice(2, np.array([32, 32, 9, 32, 20, 32, 32]), 330.0, seed=3),
             _lattice(2, np.array([100, 7, 32, 70, 32]), 330.0, seed=4)]
    fils = parts[0][1] + parts[1][1]
    sites = np.concatenate([parts[0][2], parts[1][2]])
    replicas = [dict(system_radius=p[0]["system_radius"], seed=p[0]["seed"],
                     n_filaments=len(p[1])) for p in parts]
    both = sc.Context(parts[0][0], fils, sites, precision="mixed", replicas=replicas)
    both.set_integrator_layout(32, 256)
    both.step(4)
    alone = []
    for system, f, x in parts:
        ctx = sc.Context(system, f, x, precision="mixed")
        ctx.set_integrator_layout(32, 256)
        ctx.step(4)
        alone.append(ctx.sites())
        ctx.close()
    n = len(alone[0])
    got = both.sites()
    assert np.array_equal(got[n:], alone[1])
    assert np.array_equal(got[:n], alone[0])
    both.close()


def _two_a_lane(n_dim, side, seed, n=3100, extra=()):
    """Mostly 17 to 20 sites, which fill a warp one filament at a time and
    three at a time with two sites a lane; some short ones; `extra` bond counts.
    More warps than 20 per SM, and 2.25 times those of the two-site layout."""
    import torch
    rng = np.random.default_rng(seed)
    n_seg = np.concatenate([rng.choice([16, 17, 18, 19], n), [5, 8, 12] * 10, extra]).astype(int)
    rng.shuffle(n_seg)
    assert n > 20 * torch.cuda.get_device_properties(0).multi_processor_count
    assert n + 30 / 2 >= 2.25 * (n / 3 + 30 / 2 + 1)
    return n_seg, _lattice(n_dim, n_seg, side, seed)


def test_two_sites_a_lane_uneven_with_crosslinks_bitwise():
    """Both integrator kernels, the table's lanes with two sites and one, and
    tethers on the two bonds of a lane."""
    import simcore_b200 as sc
    from checkers import Oracle
    n_seg, (system, fils, sites) = _two_a_lane(3, 330.0, 11, extra=[33, 45, 60] * 6)
    first = np.concatenate([[0], np.cumsum(n_seg + 1)])
    a = first[:400] + 3 + np.arange(400) % 3
    b = first[1:401] + 2 + np.arange(400) % 4
    ctx = sc.Context(system, fils, sites, precision="fp64")
    oracle = Oracle(system, fils, sites)
    for x in (ctx, oracle):
        x.add_crosslinks(a, b, k_spring=0.05, rest_length=1.0)
    for captured in (False, True):
        (ctx.step_graph if captured else ctx.step)(4)
        oracle.step(4)
        assert np.array_equal(ctx.sites(), oracle.sites())
        assert np.array_equal(ctx.crosslink_forces(), oracle.crosslink_forces())
    assert np.abs(oracle.crosslink_forces()).max() > 0
    ctx.close()
    oracle.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_sites_a_lane_keep_systems_apart(precision):
    """Two systems of one context in the two-site layout give the bits that
    each gives alone, with one site a lane: fewer warps."""
    import simcore_b200 as sc
    parts = [_two_a_lane(2, 1400.0, 12)[1], _lattice(2, np.array([18, 16, 31, 7, 19]), 110.0, 13)]
    fils = parts[0][1] + parts[1][1]
    sites = np.concatenate([p[2] for p in parts])
    replicas = [dict(system_radius=p[0]["system_radius"], seed=p[0]["seed"],
                     n_filaments=len(p[1])) for p in parts]
    both = sc.Context(parts[0][0], fils, sites, precision=precision, replicas=replicas)
    both.step(3)
    both.step_graph(4)
    alone = []
    for system, f, x in parts:
        ctx = sc.Context(system, f, x, precision=precision)
        ctx.step(3)
        ctx.step_graph(4)
        alone.append(ctx.sites())
        ctx.close()
    if precision == "fp64":
        assert np.array_equal(both.sites(), np.concatenate(alone))
    else:  # another elimination order: FP64 rounding, a few steps of it
        n = len(alone[0])
        assert np.array_equal(both.sites()[:n], alone[0])
        assert np.abs(both.sites()[n:] - alone[1]).max() <= 1e-12 * 110.0
    both.close()


def test_two_sites_a_lane_fused_pairs():
    """Fused pairs (every bond evaluates its own) against the split interface,
    the lane's two bonds among them."""
    import simcore_b200 as sc
    system, fils, sites = _two_a_lane(2, 500.0, 14)[1]
    a, b = (sc.Context(system, fils, sites, precision="mixed") for _ in range(2))
    for c in (a, b):
        c.set_exact_near_parallel(False)
    a.set_fused_pairs(True)
    a.step(3)
    a.step_graph(6)
    for _ in range(9):
        b.interact()
        b.update_positions()
    assert len(b.pairs()) > 1000
    assert np.array_equal(a.sites(), b.sites())
    for x, y in zip(a.bond_forces(), b.bond_forces()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
