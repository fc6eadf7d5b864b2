"""The fast build's flat-grid kernels and the general kernels at the edges of
their level tiles (16 levels, 32 at p = 1), against the oracle; the flat
reverse of phase 2 against the exact build's general one; the output kernel's
tiles, sub-cell counts and quantity lists.

Tolerances: the tendency's rounding is set by the pressure sums, 2 (p + 1)
terms of 1e5 Pa times derivative coefficients of about 5, each within 2^-53:
1e-10 Pa over a node spacing of some 1e5 m at rho >= 0.01 is 1e-13 m/s^2,
against u, v, w tendencies of 1e-3 and more: 1e-10 of the largest.  The other
fields have no such cancellation: 1e-12."""
import dataclasses

import numpy as np
import pytest

from _cases import make_case, rel_err_per_field

pytestmark = pytest.mark.gpu

CASES = [(3, 4, 2, 0), (3, 4, 15, 1), (2, 4, 16, 2), (3, 4, 17, 4), (2, 4, 33, 1), (2, 4, 64, 0), (3, 3, 16, 1),
         (3, 3, 17, 3), (3, 2, 18, 2), (3, 1, 31, 2), (3, 1, 33, 0)]


def _tol(nv):
    return np.array([1e-12, 1e-10, 1e-10, 1e-10] + [1e-12] * (nv - 4))


def _moving(o, U):
    """The state with vertical motion and seeded winds (no zero mass flux)."""
    rng = np.random.Generator(np.random.PCG64(7))
    U = np.array(U, order="F")
    U[:, :, 1:3] += rng.uniform(-0.5, 0.5, U[:, :, 1:3].shape)
    U[:-1, :, 3] += rng.uniform(-0.01, 0.01, U[:-1, :, 3].shape)
    return U


@pytest.mark.parametrize("case", CASES)
def test_flat_tendency_and_step(oracle_mod, built_lib, cuda_ok, case):
    from cgd_b200 import Dycore
    n, p, nz, nt = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, nt, "quadratic")
    U = _moving(o, U)
    d = Dycore(g, nt, nu)
    assert d.flat_form()
    err = rel_err_per_field(d.fcn(U), o.rhs(U))
    assert (err <= _tol(5 + nt)).all(), err
    V = np.array(U, order="F")
    d.time_stepper(V, 200.0, 2)
    err = rel_err_per_field(V, o.ros_step(U, 200.0, 2))
    assert (err <= 1e-9).all(), err
    d.close()


@pytest.mark.parametrize("case", [(2, 4, 9, 1), (2, 4, 16, 0), (2, 3, 17, 2), (2, 2, 5, 0), (2, 1, 33, 1)])
def test_general_metric(oracle_mod, built_lib, cuda_ok, case):
    """A metric without the flat form (sloping levels, unequal layer nodes):
    both builds run the general kernels; the exact build bit for bit."""
    from cgd_b200 import Dycore
    n, p, nz, nt = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, nt, "quadratic")
    U = _moving(o, U)
    rng = np.random.Generator(np.random.PCG64(11))
    dX = np.asfortranarray(g.dXdxI * (1.0 + 1e-3 * rng.uniform(-1, 1, g.dXdxI.shape)))
    for c in range(2):
        dX[2, c] += 1e-3 * rng.uniform(-1, 1, dX[2, c].shape) * dX[2, 2]
    J = np.asfortranarray(g.J * (1.0 + 1e-3 * rng.uniform(-1, 1, g.J.shape)))
    o.set_metric(dXdxI=dX, J=J)
    g = dataclasses.replace(g, dXdxI=dX, J=J)
    Fo = o.rhs(U)
    for exact in (True, False):
        d = Dycore(g, nt, nu, exact=exact)
        assert not d.flat_form()
        F = d.fcn(U)
        d.close()
        if exact:
            assert np.array_equal(F, Fo)
        else:
            err = rel_err_per_field(F, Fo)
            assert (err <= _tol(5 + nt)).all(), err


@pytest.mark.parametrize("case", [(3, 4, 2), (2, 4, 16), (3, 4, 17), (2, 4, 34), (2, 3, 18), (2, 2, 16), (2, 1, 33)])
def test_flat_adjoint(oracle_mod, built_lib, cuda_ok, case):
    """Both adjoints are of the same map; they differ by rounding."""
    from cgd_b200 import Dycore
    n, p, nz = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, 0, "quadratic")
    U = _moving(o, U)
    rng = np.random.Generator(np.random.PCG64(13))
    L = np.asfortranarray(rng.uniform(-1, 1, U.shape))
    out = []
    for exact in (True, False):
        d = Dycore(g, 0, nu, exact=exact)
        assert d.flat_form() != exact
        out.append(d.fcn_adjoint(U, L))
        d.close()
    err = rel_err_per_field(out[1], out[0])
    assert (err <= 1e-9).all(), err


def test_layers_are_checked(oracle_mod, built_lib, cuda_ok):
    """cgd_set_layers: the grid's own ratios change nothing but rounding, wrong
    ones send the handle to the general kernels, non-positive ones are refused."""
    from cgd_b200 import CgdError, Dycore
    from cgd_b200.grid import layer_ratios
    o, g, U, nu = make_case(oracle_mod, 3, 4, 9, 1, "quadratic")
    U = _moving(o, U)
    Fo = o.rhs(U)
    z = layer_ratios(g)
    F0 = None
    for layers in (None, z, z * 1.01 ** np.arange(9)):
        d = Dycore(dataclasses.replace(g, layers=layers), 1, nu)
        assert d.flat_form() == (layers is None or layers is z)
        F = d.fcn(U)
        d.close()
        assert (rel_err_per_field(F, Fo) <= _tol(6)).all()
        if layers is z:
            assert np.array_equal(F, F0)
        F0 = F if F0 is None else F0
    with pytest.raises(CgdError) as e:
        Dycore(dataclasses.replace(g, layers=0.0 * z), 1, nu)
    assert e.value.code == -1


@pytest.mark.parametrize("case", [(2, 4, 9, 4), (2, 4, 10, 5), (2, 4, 21, 8), (2, 3, 17, 1), (2, 2, 29, 3), (2, 1, 3, 7)])
def test_output_tiles(oracle_mod, built_lib, cuda_ok, case):
    """More quantities than one launch takes, the vorticity twice."""
    from cgd_b200 import Dycore, _lib
    from cgd_b200 import output
    n, p, nz, OP = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, 1, "quadratic")
    U = _moving(o, U)
    d = Dycore(g, 1, nu)
    inter = output.vtk_inter(p, OP, g.xw)
    f = lambda k: np.asfortranarray(U[..., k])
    ref = {_lib.OUT_RHO: o.interpolate(f(0), inter), _lib.OUT_V: o.interpolate(f(2), inter),
           _lib.OUT_WB: o.interpolate_wb(f(1), f(1), f(3), inter), _lib.OUT_PRES: o.interpolate(f(4), inter, kind=1),
           _lib.OUT_VORT: o.interpolate_vort(U, inter), _lib.OUT_TR: o.interpolate(f(5), inter, rhoc=f(0)),
           _lib.OUT_WB_UV: o.interpolate_wb(f(1), f(2), f(3), inter)}
    codes = [_lib.OUT_VORT, _lib.OUT_RHO, _lib.OUT_TR, _lib.OUT_VORT, _lib.OUT_WB, _lib.OUT_PRES]
    codes += [_lib.OUT_V] * 14 + [_lib.OUT_TR, _lib.OUT_WB_UV]
    out = d.output_fields(U, codes, inter)
    for k, c in enumerate(codes):
        assert np.array_equal(out[k].reshape(-1), ref[c].reshape(-1, order="F")), (k, c)
    d.close()


@pytest.mark.parametrize("OP", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("case", [(2, 4, 9), (2, 3, 17), (12, 2, 33), (2, 1, 64)])
def test_output_single_quantities(oracle_mod, built_lib, cuda_ok, case, OP):
    """Every quantity in a call of its own, on grids below and above the size
    at which a thread takes more sub-cells."""
    from cgd_b200 import Dycore, _lib, output
    n, p, nz = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, 1, "quadratic")
    U = _moving(o, U)
    d = Dycore(g, 1, nu)
    inter = output.vtk_inter(p, OP, g.xw)
    f = lambda k: np.asfortranarray(U[..., k])
    ref = {_lib.OUT_RHO: o.interpolate(f(0), inter), _lib.OUT_PRES: o.interpolate(f(4), inter, kind=1),
           _lib.OUT_WB: o.interpolate_wb(f(1), f(1), f(3), inter), _lib.OUT_VORT: o.interpolate_vort(U, inter),
           _lib.OUT_WB_UV: o.interpolate_wb(f(1), f(2), f(3), inter),
           _lib.OUT_TR: o.interpolate(f(5), inter, rhoc=f(0))}
    for c, r in ref.items():
        assert np.array_equal(d.output_fields(U, [c], inter).reshape(-1), r.reshape(-1, order="F")), c
    # formed quantities on both sides of a launch's sixteen
    codes = [_lib.OUT_PRES, _lib.OUT_WB] + [_lib.OUT_RHO] * 14 + [_lib.OUT_VORT, _lib.OUT_WB, _lib.OUT_PRES, _lib.OUT_WB_UV]
    for k, a in enumerate(d.output_fields(U, codes, inter)):
        assert np.array_equal(a.reshape(-1), ref[codes[k]].reshape(-1, order="F")), (k, codes[k])
    d.close()


@pytest.mark.parametrize("OP", [1, 2, 5])
def test_output_quotients_at_the_limits(oracle_mod, built_lib, cuda_ok, OP):
    """c / rho with zeros, infinities, NaN and values whose quotients leave the
    range of the shared reciprocal; weights of any size."""
    from cgd_b200 import Dycore, output
    o, g, U, nu = make_case(oracle_mod, 2, 4, 9, 0, "quadratic")
    d = Dycore(g, 0, nu)
    rng = np.random.Generator(np.random.PCG64(17))
    edge = np.array([0.0, -0.0, 1e-310, 1e-200, 1e-130, 1.0, -3.0, 1e130, 1e200, 1e308, np.inf, np.nan])
    c = np.asfortranarray(rng.uniform(-2, 2, d.shape[:2]))
    r = np.asfortranarray(rng.uniform(0.1, 2, d.shape[:2]))
    at = rng.random(c.shape) < 0.05
    c[at] = rng.choice(edge, at.sum())
    at = rng.random(c.shape) < 0.01
    r[at] = rng.choice(edge, at.sum())
    for scale in (1.0, 1e-120, 1e120):
        inter = np.asfortranarray(output.vtk_inter(4, OP, g.xw) * scale)
        with np.errstate(all="ignore"):
            ref = o.interpolate(c, inter, rhoc=r)
        assert np.array_equal(d.interpolate(c, inter, rhoc=r), ref, equal_nan=True), scale
    d.close()


@pytest.mark.parametrize("case", [(16, 4, 48, 0, False), (25, 4, 32, 2, False), (21, 4, 48, 4, True), (20, 3, 48, 0, False),
                                  (25, 3, 48, 1, True), (26, 2, 48, 0, False), (38, 2, 33, 3, True), (33, 1, 33, 0, False),
                                  (45, 1, 33, 2, True)])
def test_phase2_launch_forms(built_lib, cuda_ok, case):
    """From p2_split_threads threads a role on, a handle runs the roles of phase
    2 in launches of their own, an ensemble always in one: the same bits."""
    import torch
    from cgd_b200 import Dycore, Ensemble, physics
    from cgd_b200 import grid as G
    n, p, nz, nt, mixed = case
    role = 6 * n * n * -(-nz // (32 if p == 1 else 16)) * (32 if p == 1 else 16) * (p + 1) ** 2
    assert role >= (500000 if mixed else 750000) * (2 + nt)
    g = G.init_grid_sphere_device(n, p, G.vertical_quadratic(nz, 30000.0), 30000.0, 6.371e6)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    U = torch.rand((5 + nt, g.NumG, nz), dtype=torch.float64, device="cuda", generator=gen) * 0.01 + 1.0
    U[1:4] = 10.0 * (U[1:4] - 1.005)
    U[4] *= 300.0
    out = []
    for ensemble in (False, True):
        d = Dycore(g, nt, physics.hyperdiffusion(n, p), precision="mixed" if mixed else "fp64")
        assert d.flat_form()
        V = U.clone()
        if ensemble:
            e = Ensemble([d])
            e.step([V], [10.0], 1)
            e.close()
        else:
            d.time_stepper(V, 10.0, 1)
        d.close()
        out.append(V)
    assert bool(torch.isfinite(out[0]).all())
    assert torch.equal(out[0], out[1])


def _workload_grids():
    from cgd_b200 import physics as Ph
    out = {(c.nPanel, c.OrdPoly, c.nz, c.stretch) for c in Ph.CONFIGS.values()}
    out |= {(n, Ph.ENSEMBLE["OrdPoly"], nz, "quadratic") for n, nz in Ph.ENSEMBLE["grids"]}
    return sorted(out | {(12, p, 31, "quadratic") for p in (1, 2, 3)})


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("case", _workload_grids())
def test_workload_grids_are_flat(built_lib, cuda_ok, case, where):
    """The grids of the package's configurations are of the flat form, formed on
    the device or on the host: a set-up that moved their rounding past the check
    (2e-15; uniform levels come near it, and above it at nz 45) would lose the
    flat kernels silently."""
    from cgd_b200 import Dycore
    from cgd_b200 import grid as G
    n, p, nz, stretch = case
    if where == "host" and n > 16:
        pytest.skip("minutes on the host")
    z = G.vertical_uniform(nz, 30000.0) if stretch == "uniform" else G.vertical_quadratic(nz, 30000.0)
    init = G.init_grid_sphere if where == "host" else G.init_grid_sphere_device
    d = Dycore(init(n, p, z, 30000.0, 6.371e6))
    assert d.flat_form()
    d.close()


def test_step_where_rho_theta_is_zero(oracle_mod, built_lib, cuda_ok):
    """dp/d(rho theta) there is 0, as the power gives it, not 0 / 0."""
    from cgd_b200 import Dycore
    o, g, U, nu = make_case(oracle_mod, 3, 4, 9, 1, "quadratic")
    U = _moving(o, U)
    U[3, 10, 4] = U[0, 50, 4] = U[8, 70, 4] = 0.0
    d = Dycore(g, 1, nu)
    V = np.array(U, order="F")
    d.time_stepper(V, 1e-3, 1)
    d.close()
    assert np.isfinite(V).all()
    assert (rel_err_per_field(V, o.ros_step(U, 1e-3, 1)) <= 1e-9).all()
