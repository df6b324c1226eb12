"""Parity of the chemistry kernels against the CPU oracle: the Wu-splitting
reaction step (point implicit and explicit, both schedules) and the explicit
finite-rate source, on seeded batches of H2/air reactors (Li-2004,
9 species / 19 reactions; PREMIX H2/O2/Ar, 9 species / 18 reactions).

Bar: per step from identical inputs, max |gpu - oracle| / max |oracle| of
every conserved-variable plane <= 1e-12; substep counts identical; the
work-queue schedule bit-identical to one thread per node.
"""
import numpy as np
import pytest

import cases
import mechanism
import pyoracle
from gpuzone import GpuZone, rel_err

pytestmark = pytest.mark.gpu


def _pair(case):
    oz = pyoracle.OracleZone(case)
    oz.call("orc_compute_cv_from_bv")
    gz = GpuZone(case)
    gz.ctx.cv_from_bv()
    gz.torch.cuda.synchronize()
    return oz, gz


def _nsub_tensor(gz):
    import torch
    return torch.zeros(gz.case.N, dtype=torch.int32, device="cuda:0")


@pytest.mark.parametrize("schedule", [0, 1])
@pytest.mark.parametrize("mech_name", ["li2004", "premix_h2_ar"])
def test_wu_reaction_point_implicit_per_step(schedule, mech_name):
    mech = mechanism.load(mech_name)
    if mech_name == "li2004":
        case = cases.reactor_batch(mech, 512, seed=7)
    else:  # stoichiometric H2/O2 diluted 70 % Ar
        X = np.zeros(mech.n_spec)
        X[mech.index("H2")], X[mech.index("O2")], X[mech.index("AR")] = 0.2, 0.1, 0.7
        T = np.linspace(1100.0, 1900.0, 300)
        case = cases.reactor(mech, T, 30000.0, X)
    oz, gz = _pair(case)
    nsub = _nsub_tensor(gz)
    dt = 1e-7
    for s in range(6):
        gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
        ns_o = oz.reaction_step(dt, want_nsub=True)
        gz.ctx.wu_reaction_step(dt, schedule=schedule, nsub_ptr=nsub.data_ptr())
        gz.ctx.sync()
        assert np.array_equal(nsub.cpu().numpy(), ns_o), f"substep counts differ at step {s}"
        e = rel_err(gz.get("cv"), oz["cv"])
        assert e <= 1e-12, f"step {s}: conserved-variable relative difference {e:.3e}"
        assert rel_err(gz.get("bv")[[0, 4, 5]], oz["bv"][[0, 4, 5]], momentum=()) <= 1e-12
        assert rel_err(gz.get("reaction_timeScale")[None], oz["reaction_timeScale"][None], momentum=()) <= 1e-12


def test_wu_reaction_explicit_per_step():
    mech = mechanism.load("li2004")
    case = cases.reactor_batch(mech, 256, seed=3)
    case.param["chem_advance_method"] = 0
    oz, gz = _pair(case)
    for s in range(4):
        gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
        oz.reaction_step(2e-8)
        gz.ctx.wu_reaction_step(2e-8, schedule=0)
        gz.ctx.sync()
        assert rel_err(gz.get("cv"), oz["cv"]) <= 1e-12


def test_work_queue_is_bit_identical_to_plain_schedule():
    mech = mechanism.load("li2004")
    case = cases.reactor_batch(mech, 4096, seed=11)
    a = GpuZone(case)
    b = GpuZone(case)
    for z in (a, b):
        z.ctx.cv_from_bv()
    na, nb = _nsub_tensor(a), _nsub_tensor(b)
    for _ in range(8):
        a.ctx.wu_reaction_step(1e-7, schedule=0, nsub_ptr=na.data_ptr())
        b.ctx.wu_reaction_step(1e-7, schedule=1, nsub_ptr=nb.data_ptr())
    a.ctx.sync()
    b.ctx.sync()
    assert np.array_equal(a.get("cv"), b.get("cv"))
    assert np.array_equal(na.cpu().numpy(), nb.cpu().numpy())
    assert na.cpu().numpy().max() > na.cpu().numpy().min()  # uneven work really occurred


def test_finite_rate_chemistry_source():
    mech = mechanism.load("li2004")
    case = cases.reactor_batch(mech, 300, seed=5)
    oz, gz = _pair(case)
    # advance a little so that radicals exist
    for _ in range(3):
        oz.reaction_step(1e-7)
    gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
    oz["dq"][:] = 0
    gz.t["dq"].zero_()
    oz.call("orc_finite_rate_chemistry")
    gz.ctx.finite_rate_chemistry()
    gz.ctx.sync()
    assert rel_err(gz.get("dq")[5:], oz["dq"][5:], momentum=()) <= 1e-12
    assert rel_err(gz.get("reaction_timeScale")[None], oz["reaction_timeScale"][None], momentum=()) <= 1e-12


def test_ignition_of_the_reference_reactor_case():
    """The reference's constant-volume example (1000 K, 2 atm, Li-2004) on the
    GPU: the final equilibrium matches the reference's golden trajectory and
    the ignition time (T = 1500 K) matches the oracle's (same integrator)."""
    import os
    golden = np.load(os.path.join(os.path.dirname(__file__), "golden", "reactor_li2004.npz"))
    mech = mechanism.load("li2004")
    X = np.zeros(9)
    X[mech.index("H2")], X[mech.index("O2")], X[mech.index("N2")] = 0.295775, 0.147887, 0.556338
    case = cases.reactor(mech, [1000.0], 202650.0, X)
    gz = GpuZone(case)
    gz.ctx.cv_from_bv()
    dt, t, Ts = 2e-7, 0.0, []
    while t < 1.2e-3 - 1e-12:
        gz.ctx.wu_reaction_step(dt, schedule=1)
        t += dt
        Ts.append(float(gz.t["bv"][5, 0].item()))
    Ts = np.array(Ts)
    ts = dt * np.arange(1, len(Ts) + 1)
    assert Ts[-1] == pytest.approx(golden["T"][-1], rel=1e-5)
    t_ign = np.interp(1500.0, Ts, ts)
    assert t_ign == pytest.approx(8.88e-4, rel=0.01)


@pytest.mark.parametrize("n", [1, 9, 10, 11, 39, 41, 121])
@pytest.mark.parametrize("long_side", [False, True])
def test_reaction_step_at_group_edges(n, long_side):
    """Node counts around the nodes of a warp (10) and of a CTA (40), both
    schedules, uneven substep counts.  long_side: a reaction with four
    molecules on a side, more than the lane-group kernels' molecule lists hold."""
    import dataclasses

    mech = mechanism.load("li2004")
    if long_side:
        r = next(k for k in range(mech.n_reac) if mech.stoi_f[k].max() == 2)
        f, b = np.array(mech.stoi_f), np.array(mech.stoi_b)
        f[r] *= 2
        b[r] *= 2
        mech = dataclasses.replace(mech, stoi_f=f, stoi_b=b)
    case = cases.reactor_batch(mech, n, seed=n)
    oz, gz = _pair(case)
    nsub = _nsub_tensor(gz)
    oz["reaction_timeScale"][:] = 1e-7 / (0.5 + 3 + np.arange(n) % 23)
    for s in range(3):
        ns_o = None
        for schedule in (0, 1):
            gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
            gz.ctx.wu_reaction_step(1e-7, schedule=schedule, nsub_ptr=nsub.data_ptr())
            gz.ctx.sync()
            out = {k: gz.get(k).copy() for k in ("cv", "bv", "sv", "reaction_timeScale")}
            if ns_o is None:
                first, ns_o = out, nsub.cpu().numpy().copy()
            else:
                assert all(np.array_equal(out[k], first[k]) for k in out)
        ns_r = oz.reaction_step(1e-7, want_nsub=True)
        assert np.array_equal(ns_o, ns_r)
        assert rel_err(out["cv"], oz["cv"]) <= 1e-12
        assert rel_err(out["sv"], oz["sv"], momentum=()) <= 1e-11  # the smallest species, against its own maximum


def _reference_state(mech, d):
    """The mechanism with the enthalpy of every H atom shifted by R d: another
    reference state of the element, which no reaction's energy depends on."""
    import dataclasses

    n_h = np.asarray(mech.elem_comp)[:, list(mech.elements).index("H")]
    low, high = np.array(mech.low), np.array(mech.high)
    low[:, 5] += n_h * d
    high[:, 5] += n_h * d
    return dataclasses.replace(mech, low=low, high=high)


def test_forward_rates_do_not_depend_on_the_elements_reference_state():
    """One substep of an irreversible mechanism: the rates, and with them the
    time scale, are those of A T^b exp(-Ea/T) and the concentrations alone, to
    the last bit, whatever the species' g."""
    import dataclasses

    mech = mechanism.load("li2004")
    mech = dataclasses.replace(mech, reac_type=np.zeros_like(mech.reac_type))
    ts = []
    for d in (0.0, 2e4, -2e4):
        gz = GpuZone(cases.reactor_batch(_reference_state(mech, d), 256, seed=5))
        gz.ctx.cv_from_bv()
        gz.t["cv"][5:] += 1e-6 * gz.t["cv"][:1]  # all species present
        gz.t["reaction_timeScale"].fill_(1.0)
        gz.ctx.wu_reaction_step(1e-9, schedule=0)
        ts.append(gz.get("reaction_timeScale"))
    assert ts[0].min() > 0 and ts[0].max() < 1.0
    assert np.array_equal(ts[0], ts[1]) and np.array_equal(ts[0], ts[2])


@pytest.mark.parametrize("d", [4e5, -4e5])
@pytest.mark.parametrize("schedule", [0, 1])
def test_reaction_step_with_a_remote_reference_state(schedule, d):
    """g of the hydrogen species beyond the range of exp (|d| / T > 709 a pair
    of atoms) while most of them are absent: only differences of g enter.
    Bar: g of some 900 carries about 5 roundings, four species a reaction, so
    the rates of both sides differ by 4 x 5 x 900 x 2^-53 = 2e-12, of which a
    step of 1e-7 s takes its share in 5 to 25 substeps."""
    mech = _reference_state(mechanism.load("li2004"), d)
    case = cases.reactor_batch(mech, 121, seed=8)
    oz, gz = _pair(case)
    oz["reaction_timeScale"][:] = 1e-7 / (0.5 + 5 + np.arange(121) % 20)
    for _ in range(3):
        gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
        gz.ctx.wu_reaction_step(1e-7, schedule=schedule)
        gz.ctx.sync()
        oz.reaction_step(1e-7)
        assert np.all(np.isfinite(gz.get("cv")))
        assert rel_err(gz.get("cv"), oz["cv"]) <= 1e-10
        assert rel_err(gz.get("bv")[[0, 4, 5]], oz["bv"][[0, 4, 5]], momentum=()) <= 1e-10


@pytest.mark.parametrize("mech_name", ["li2004", "premix_h2_ar"])
@pytest.mark.parametrize("dt", [1e-6, 1e-5])
def test_coarse_substeps_of_burning_states(mech_name, dt):
    """One substep far beyond the time scale, where the matrix is far from the
    identity and most nodes swap rows, from radical-rich states, both schedules.
    Bar: a change of the matrix by a rounding (1e-16) changes the solution of
    these systems by up to 4e-13 at 10 us, so rates that differ by rounding
    (3e-15) give 1e-11."""
    mech = mechanism.load(mech_name)
    if mech_name == "li2004":
        case = cases.reactor_batch(mech, 41, seed=3)
    else:
        X = np.zeros(mech.n_spec)
        X[mech.index("H2")], X[mech.index("O2")], X[mech.index("AR")] = 0.2, 0.1, 0.7
        case = cases.reactor(mech, np.linspace(1500.0, 1900.0, 41), 30000.0, X)
    oz, gz = _pair(case)
    for _ in range(40):
        gz.ctx.wu_reaction_step(2e-7 if mech_name == "li2004" else 2e-6, schedule=1)
    for k in ("cv", "bv", "sv"):
        oz[k][:] = gz.get(k)
    oz["reaction_timeScale"][:] = 2 * dt  # one substep
    before = gz.get("sv").copy()
    out = []
    for schedule in (0, 1):
        gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
        gz.ctx.wu_reaction_step(dt, schedule=schedule)
        gz.ctx.sync()
        out.append([gz.get(k).copy() for k in ("cv", "sv", "reaction_timeScale")])
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    ns = oz.reaction_step(dt, want_nsub=True)
    assert np.all(ns == 1)
    assert np.abs(out[0][1] - before).max() > 1e-5  # the step did something
    assert rel_err(out[0][0], oz["cv"]) <= 1e-11
    assert rel_err(out[0][1], oz["sv"], momentum=()) <= 1e-11


@pytest.mark.parametrize("edge", ["t_low", "t_mid", "t_high", "cold"])
def test_states_at_the_edges_of_the_thermo_ranges(edge):
    """Temperatures on and one part in 1e6 around each end of the species' polynomial
    ranges and at 250 to 350 K, with the radicals present or exactly zero."""
    mech = mechanism.load("li2004")
    if edge == "cold":
        T = np.linspace(250.0, 350.0, 21)
    else:
        t = np.unique(np.asarray(getattr(mech, edge), dtype=float))
        T = np.concatenate([t, t * (1 - 1e-6), t * (1 + 1e-6), t * 0.98, t * 1.02])
    T = np.concatenate([T, T])
    X = np.full((T.size, 9), 1e-4)
    X[T.size // 2:] = 0.0
    X[:, mech.index("H2")], X[:, mech.index("O2")], X[:, mech.index("N2")] = 0.3, 0.15, 0.55
    case = cases.reactor(mech, T, 101325.0, X / X.sum(axis=1, keepdims=True))
    oz, gz = _pair(case)
    for step in range(2):
        oz["reaction_timeScale"][:] = 1e-8 / 4.5
        gz.load_from(oz, keys=("cv", "bv", "sv", "reaction_timeScale"))
        gz.ctx.wu_reaction_step(1e-8, schedule=step)
        gz.ctx.sync()
        oz.reaction_step(1e-8)
        assert rel_err(gz.get("cv"), oz["cv"]) <= 1e-12
        assert rel_err(gz.get("bv")[[0, 4, 5]], oz["bv"][[0, 4, 5]], momentum=()) <= 1e-12
        ts = oz["reaction_timeScale"]
        assert np.all(np.abs(gz.get("reaction_timeScale") - ts) <= 1e-11 * np.abs(ts))
