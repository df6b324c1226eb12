"""Boundary faces and the properties shell of blocks around the extents at
which a face's ghost layers stop being shared between threads and its two
faces stop being one launch (ngg + 1 nodes), against the CPU oracle.

The faces copy, average and reflect; cv is then one product and sum a value:
1e-14 of each plane's largest value."""
import dataclasses

import numpy as np
import pytest

import cases
import mechanism
import pyoracle
from gpuzone import GpuZone, rel_err

pytestmark = pytest.mark.gpu

LABELS = {"periodic": [(a, d, 8) for a in range(3) for d in (-1, 1)],
          "outflow": [(a, d, 6) for a in range(3) for d in (-1, 1)],
          "symmetry": [(a, d, 3) for a in range(3) for d in (-1, 1)],
          # the two faces of an axis apart in the list, or of two conditions: a launch each
          "mixed": [(0, -1, 6), (1, -1, 6), (0, 1, 6), (1, 1, 3), (2, -1, 8), (2, 1, 8)]}


def _corner(case, n, ny, nz):
    """The first n x ny x nz nodes of a block, with its padded arrays' values."""
    g = case.ngg

    def cut(a):
        a = a.reshape(a.shape[:-1] + case.shape())[..., : nz + 2 * g, : ny + 2 * g, : n + 2 * g]
        return np.ascontiguousarray(a.reshape(a.shape[:-3] + (-1,)))

    return dataclasses.replace(case, mx=n, my=ny, mz=nz, metric=cut(case.metric), jac=cut(case.jac), bv=cut(case.bv),
                               sv=cut(case.sv) if case.sv.shape[0] else np.zeros((0, cut(case.jac).size)), x=None,
                               xyz=None)


@pytest.mark.parametrize("labels", list(LABELS))
@pytest.mark.parametrize("shape", [(9, 8, 7), (5, 4, 6), (4, 6, 5), (12, 5, 4)])
@pytest.mark.parametrize("viscous", [False, True])
def test_boundary_conditions_of_thin_blocks(labels, shape, viscous):
    case = _corner(cases.perturbed(cases.sine_wave(n=13, ny=9, nz=9, scheme=52, viscous=viscous, amp=0.02), seed=1,
                                   amp=0.05), *shape)
    if labels == "symmetry" and min(shape) < 5:
        pytest.skip("a reflected node of one symmetry face would be the other's")
    case.faces = LABELS[labels]
    oz = pyoracle.OracleZone(case)
    oz.call("orc_compute_cv_from_bv")
    gz = GpuZone(case)
    gz.load_from(oz, keys=("cv", "bv"))
    oz.call("orc_apply_boundary_conditions")
    gz.ctx.boundary_conditions()
    for k in ("bv", "cv"):
        assert rel_err(gz.get(k), oz[k][: gz.t[k].shape[0]], momentum=()) <= 1e-14, k


@pytest.mark.parametrize("shape", [(9, 7, 5), (5, 9, 6), (33, 5, 5)])
def test_properties_shell_covers_what_the_update_leaves(shape):
    """After a step every property of the padded block is that of its final
    state: the update's nodes and the shell's together are all of them."""
    n, ny, nz = shape
    mech = mechanism.load("li2004")
    case = cases.perturbed(cases.mix_wave(mech, n, ny=ny, nz=nz, scheme=52, dt=1e-9), seed=2,
                           amp=1e-3)
    gz = GpuZone(case)
    gz.initialize()
    gz.ctx.rk3_step()
    keys = ("mul", "gamma", "acoustic_speed", "thermal_conductivity", "rho_D")
    out = {k: gz.get(k).copy() for k in keys}
    gz.ctx.properties()
    for k in keys:
        assert np.allclose(out[k], gz.get(k), rtol=1e-14, atol=0), k


THIN = [(5, 9, 8), (6, 9, 8), (9, 5, 8), (9, 6, 8), (9, 8, 5), (9, 8, 6), (5, 5, 5), (4, 5, 6), (6, 4, 5), (5, 6, 4)]


@pytest.mark.parametrize("kind", ["isothermal", "adiabatic", "back_pressure", "symmetry_wall"])
@pytest.mark.parametrize("gas", ["air", "mixture"])
@pytest.mark.parametrize("shape", THIN)
def test_walls_and_back_pressure_of_thin_blocks(kind, gas, shape):
    """The conditions whose ghosts read inner nodes up to ngg away, on blocks
    of ngg, ngg + 1 and ngg + 2 nodes (ngg = 4) along each axis."""
    mech = mechanism.load("li2004")
    if gas == "air":
        case = cases.perturbed(cases.sine_wave(n=13, ny=11, nz=11, scheme=72, viscous=True, amp=0.02), seed=1, amp=0.05)
    else:
        case = cases.perturbed(cases.mix_wave(mech, 13, ny=11, nz=11, scheme=72), seed=1, amp=0.01)
    case = _corner(case, *shape)
    if kind == "back_pressure":
        case.faces = LABELS["outflow"]
        case = cases.with_back_pressure(case, 0.9 * float(case.bv[4].mean()))
    else:
        if kind == "symmetry_wall":
            case.faces = [(0, -1, 3), (1, -1, 2), (0, 1, 2), (1, 1, 3), (2, -1, 2), (2, 1, 2)]
        else:
            case.faces = [(a, d, 2) for a in range(3) for d in (-1, 1)]
        catalytic = gas == "mixture" and kind == "isothermal"
        case = cases.with_walls(case, thermal_type=int(kind == "adiabatic"), faces=(), catalytic_type=int(catalytic),
                                yk=case.sv[:, 0] if catalytic else None)
    oz = pyoracle.OracleZone(case)
    oz.call("orc_compute_cv_from_bv")
    gz = GpuZone(case)
    gz.load_from(oz, keys=("cv", "bv"))
    oz.call("orc_apply_boundary_conditions")
    gz.ctx.boundary_conditions()
    tol = 1e-14 if gas == "air" else 1e-13  # the mixture's energy is a sum over nine species' polynomials
    for k in ("bv", "cv") + (("sv",) if gas == "mixture" else ()):
        assert rel_err(gz.get(k), oz[k][: gz.t[k].shape[0]], momentum=()) <= tol, k


@pytest.mark.parametrize("labels", ["periodic", "outflow"])
@pytest.mark.parametrize("shape", THIN)
def test_mixture_boundary_conditions_of_thin_blocks(labels, shape):
    case = _corner(cases.perturbed(cases.mix_wave(mechanism.load("li2004"), 13, ny=11, nz=11, scheme=72), seed=3,
                                   amp=0.01), *shape)
    case.faces = LABELS[labels]
    oz = pyoracle.OracleZone(case)
    oz.call("orc_compute_cv_from_bv")
    gz = GpuZone(case)
    gz.load_from(oz, keys=("cv", "bv"))
    oz.call("orc_apply_boundary_conditions")
    gz.ctx.boundary_conditions()
    for k in ("bv", "cv", "sv"):
        assert rel_err(gz.get(k), oz[k][: gz.t[k].shape[0]], momentum=()) <= 1e-13, k


@pytest.mark.parametrize("gas", ["air", "mixture"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 3, 3), (2, 3, 9), (9, 2, 3), (3, 9, 2), (9, 7, 5)])
def test_properties_shell_of_the_thinnest_blocks(gas, shape):
    """As above with two and three nodes an axis, where an axis has no or one
    inner node, and for air."""
    if gas == "air":
        case = cases.perturbed(cases.sine_wave(n=13, ny=11, nz=11, scheme=52, viscous=True, amp=0.02), seed=1, amp=0.02)
        keys = ("mul",)
    else:
        case = cases.perturbed(cases.mix_wave(mechanism.load("li2004"), 13, ny=11, nz=11, scheme=52, dt=1e-9), seed=2,
                               amp=1e-3)
        keys = ("mul", "gamma", "acoustic_speed", "thermal_conductivity", "rho_D")
    case = _corner(case, *shape)
    case.faces = LABELS["outflow"]
    gz = GpuZone(case)
    gz.initialize()
    for k in keys:
        gz.t[k].mul_(1 + 1e-6)  # what the step does not write again stays off
    gz.ctx.rk3_step()
    out = {k: gz.get(k).copy() for k in keys}
    gz.ctx.properties()
    for k in keys:
        assert np.all(np.isfinite(out[k])) and np.allclose(out[k], gz.get(k), rtol=1e-14, atol=0), k


@pytest.mark.parametrize("shape", [(1, 1), (7, 5), (128, 3), (121, 17), (3, 300)])
@pytest.mark.parametrize("gas", ["air", "mixture"])
def test_k_copy_of_2d_blocks(gas, shape):
    """Every ghost plane of bv, sv and cv is a copy of plane 0, corners
    included, and plane 0 is left as it is."""
    import torch

    case = cases.sod(12, 7, scheme=52) if gas == "air" else cases.mix_tube(mechanism.load("premix_h2_ar"), 12, 7)
    g, (n, ny) = case.ngg, shape
    P = (n + 2 * g) * (ny + 2 * g) * (1 + 2 * g)
    case = dataclasses.replace(case, mx=n, my=ny, metric=np.ones((9, P)), jac=np.ones(P), bv=np.ones((6, P)),
                               sv=np.ones((case.param["n_scalar"], P)), x=None, xyz=None)
    gz = GpuZone(case)
    gen = torch.Generator(device="cuda:0").manual_seed(1)
    keys = ("bv", "cv") + (("sv",) if gas == "mixture" else ())
    before = {}
    for k in keys:
        gz.t[k].copy_(torch.rand(gz.t[k].shape, generator=gen, device="cuda:0", dtype=torch.float64))
        before[k] = gz.t[k].clone().view(gz.t[k].shape[0], 1 + 2 * g, ny + 2 * g, n + 2 * g)
    gz.ctx.eliminate_k_gradient()
    for k in keys:
        a = gz.t[k].view(before[k].shape)
        assert torch.equal(a, before[k][:, g: g + 1].expand_as(a)), k
