"""Captured runs (sc_step_graph) in both their forms, a CUDA graph's loop with
conditional nodes and a chain of launches with a control kernel between two
steps: each against the host-driven steps or the CPU oracle, bit for bit, on
systems small enough that the default would chain them all."""
import numpy as np
import pytest

from checkers import Oracle
from test_gpu_parity import (_ctx, _ctx_replicas, _replica_batch, _workload, _workload_E,
                             assert_same, compare_state)

pytestmark = pytest.mark.gpu

FORMS = ["graph", "chain"]


def _same_run(a, b):
    assert_same(a.sites(), b.sites(), "sites")
    assert_same(a.prev_sites(), b.prev_sites(), "prev sites")
    assert_same(a.pairs(), b.pairs(), "pairs")
    for x, y in zip(a.bond_forces(), b.bond_forces()):
        assert_same(x, y, "bond forces")
    assert_same(a.dr_tot(), b.dr_tot(), "dr_tot")
    ca, cb = a.counters(), b.counters()
    assert (ca.i_step, ca.n_rebuilds) == (cb.i_step, cb.n_rebuilds)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_form_matches_host_path(precision, form):
    system, fils, sites = _workload("B", 0.05, seed=6)
    a = _ctx(system, fils, sites, precision)
    b = _ctx(system, fils, sites, precision)
    a.set_run_form(form)
    for n in (40, 41, 20):
        a.step_graph(n)
        b.step(n)
        _same_run(a, b)
    assert a.counters().n_rebuilds > 0


@pytest.mark.parametrize("form", FORMS)
def test_form_replicas_match_oracle(form):
    from simcore_b200 import workloads
    system, fils, sites, reps = _replica_batch(5, 0.03, seed=2)
    ctx = _ctx_replicas(system, fils, sites, reps)
    ctx.set_run_form(form)
    oracles = [Oracle(*p) for p in workloads.split_replicas(system, fils, sites, reps)]
    independent = False  # the systems had rebuilt different numbers of times
    for n in (3, 40, 81):
        ctx.step_graph(n)
        s0 = 0
        for r, o in enumerate(oracles):
            o.step(n)
            assert_same(ctx.sites()[s0:s0 + o.n_sites, :2], o.sites()[:, :2], "system %d" % r)
            assert ctx.replica_counters()[0][r] == o.n_rebuilds
            s0 += o.n_sites
        independent = independent or len({o.n_rebuilds for o in oracles}) > 1
    assert independent


@pytest.mark.parametrize("form", FORMS)
def test_form_crosslinks_match_oracle(form):
    system, fils, sites, (a, b, k, rest) = _workload_E(0.01, seed=4)
    ctx = _ctx(system, fils, sites)
    ctx.set_run_form(form)
    o = Oracle(system, fils, sites)
    ctx.add_crosslinks(a, b, k_spring=k, rest_length=rest)
    o.add_crosslinks(a, b, k_spring=k, rest_length=rest)
    for n in (41, 60):
        ctx.step_graph(n)
        o.step(n)
        compare_state(ctx, o, 3, capture=False)
        assert_same(ctx.crosslink_forces(), o.crosslink_forces(), "tether forces")


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("case", ["C", "D", "E"])
def test_form_fused_pairs_match_host_path(case, form):
    """Mixed lengths (both integrator kernels), several systems, tethers."""
    from test_gpu_fused import _pair, _same_state
    a, b = _pair(case)
    a.set_run_form(form)
    for n in (40, 21):
        a.step_graph(n)
        b.step(n)
        _same_state(a, b)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_form_thermo_matches_host_path(precision, form):
    system, fils, sites = _workload("B", 0.02, seed=3)
    runs = []
    for captured in (True, False):
        ctx = _ctx(system, fils, sites, precision)
        ctx.set_run_form(form)
        ctx.set_thermo(6)
        (ctx.step_graph if captured else ctx.step)(50)
        runs.append((ctx, ctx.thermo_records(), ctx.potential_energy()))
    (a, ra, ea), (b, rb, eb) = runs
    _same_run(a, b)
    assert len(ra[0]) == 8
    for x, y in zip(ra, rb):
        assert_same(x, y, "records")
    assert_same(ea, eb, "potential energy")


@pytest.mark.parametrize("form", FORMS)
def test_form_reports_an_unphysical_displacement(form):
    """The run ends with the error of the host-driven steps (a filament moved
    by 80 accumulates more than 10000, include/simcore/species.hpp:114-118)."""
    import simcore_b200 as sc
    system, fils, sites = _workload("B", 0.02, seed=14)
    ctx = _ctx(system, fils, sites, "mixed")
    ctx.set_run_form(form)
    ctx.step(2)
    moved = ctx.sites()
    moved[:11, 0] += 80.0
    ctx.set_sites(moved)
    with pytest.raises(sc.ScError) as e:
        ctx.step_graph(20)
    assert e.value.code == 7


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_form_grows_an_overflowing_list(precision, form):
    from simcore_b200 import workloads
    cfg = workloads.make("E", scale=0.026, seed=4, n_seg=40)
    a, b = (_ctx(*cfg[:3], precision=precision) for _ in range(2))
    a.set_run_form(form)
    a.step_graph(400)
    b.step(400)
    _same_run(a, b)
    assert a.counters().n_list_regrowths > 0


# Bonds on both sides of the default's limit (12,288), and groups of 32 cells
# (32,768): cells of 1.1225 make 101 and 102 a side, 32,197 and 33,163 groups.
@pytest.mark.parametrize("n_fil,side", [(1228, 80.0), (1229, 80.0), (60, 113.93), (60, 115.05)])
def test_default_form_at_its_limits(n_fil, side):
    """Whatever form the default picks, the run's bits are the same."""
    import simcore_b200 as sc
    from test_gpu_team import _lattice
    system, fils, sites = _lattice(3, np.array([10] * n_fil), side, seed=n_fil)
    ctxs = []
    if n_fil == 60:
        assert sc.Context(system, fils, sites).counters().n_cells_1d == {113.93: 101, 115.05: 102}[side]
    for form in ["auto"] + FORMS:
        ctxs.append(_ctx(system, fils, sites))
        ctxs[-1].set_run_form(form)
        ctxs[-1].step_graph(30)
    for other in ctxs[1:]:
        _same_run(ctxs[0], other)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stopped_run_leaves_the_same_forces(precision):
    """A run that an error stops leaves the forces of its last step, whichever
    form it has: the launches that a chain still holds change nothing.  (A pair
    out of range keeps its stored force, so an evaluation of the positions after
    the last step would show.)"""
    import simcore_b200 as sc
    system, fils, sites = _workload("B", 0.05, seed=14)
    got = []
    for form in FORMS:
        ctx = _ctx(system, fils, sites, precision)
        ctx.set_run_form(form)
        ctx.set_thermo(10**6)
        ctx.step(2)
        moved = ctx.sites()
        moved[:11, 0] += 80.0
        ctx.set_sites(moved)
        with pytest.raises(sc.ScError):
            ctx.step_graph(60)
        got.append((ctx.sites(), ctx.pairs(), *ctx.bond_forces(), ctx.potential_energy()))
    for x, y in zip(*got):
        assert_same(x, y, "state after the stop")


def test_long_chain_is_queued_in_pieces():
    """2,070 steps, 1,035 BD steps, are three pieces of a chain (512 each): the
    graph's bits.  A run that stops in its first piece launches no more of it:
    the 4,000 steps of a run with an unphysical displacement would be 10,002
    launches, a piece is 512 times five (control, two pair and two integrator
    kernels) and three."""
    import simcore_b200 as sc
    system, fils, sites = _workload("B", 0.02, seed=14)
    runs = []
    for form in FORMS:
        ctx = _ctx(system, fils, sites)
        ctx.set_run_form(form)
        ctx.step_graph(2070)
        runs.append(ctx)
    _same_run(*runs)
    ctx = runs[1]
    moved = ctx.sites()
    moved[:11, 0] += 80.0
    ctx.set_sites(moved)
    before = ctx.counters().kernel_launches
    with pytest.raises(sc.ScError) as e:
        ctx.step_graph(4000)
    assert e.value.code == 7
    assert ctx.counters().kernel_launches - before <= 512 * 5 + 3


@pytest.mark.parametrize("side,form", [(80.0, "chain"), (16.0, "graph")])
def test_default_form_by_pairs(side, form):
    """A sparse small system takes the chain, a dense one (more than six pairs
    a bond) the graph: a run with rebuilds makes as many launches as that form
    (a rebuild's kernels are launches in the graph alone)."""
    from test_gpu_team import _lattice
    n_fil = 144
    system, fils, sites = _lattice(2, np.array([10] * n_fil), side, seed=3)
    system = dict(system, delta=1e-5, wca_eps=0.01)
    made = {}
    for f in ("auto", "graph", "chain"):
        ctx = _ctx(system, fils, sites, "mixed")
        ctx.set_run_form(f)
        n_pairs = ctx.counters().n_pairs
        before = ctx.counters()
        ctx.step_graph(3000)
        after = ctx.counters()
        assert after.n_rebuilds > before.n_rebuilds
        made[f] = after.kernel_launches - before.kernel_launches
    assert (n_pairs > 6 * 10 * n_fil) == (form == "graph")
    assert made["graph"] != made["chain"]
    assert made["auto"] == made[form]
