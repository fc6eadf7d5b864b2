"""Decomposed grid on the GPU: the parts of a 2- and 3-rank element partition
run together in one process (PartGroup: the same pack, exchange and unpack
of contributions as between processes, the transport being device copies)
and must reproduce the single-process tendency and Rosenbrock-W steps bit
for bit on every rank's DOFs - the contributors of a DOF are summed in the
same order whichever rank owns them.  The exact build is also compared with
the oracle."""
import numpy as np
import pytest

from _cases import make_case

pytestmark = pytest.mark.gpu


def _dev(U):
    import torch
    return torch.from_numpy(np.ascontiguousarray(U.transpose(2, 1, 0))).cuda()


def _host(t):
    return t.cpu().numpy().transpose(2, 1, 0)


@pytest.mark.parametrize("nranks", [2, 3])
@pytest.mark.parametrize("variant", ["exact", "fast"])
def test_group_matches_single_process(oracle_mod, built_lib, cuda_ok, nranks, variant):
    import torch
    from cgd_b200 import Dycore, PartGroup
    from cgd_b200.parallel import build_plans, partition_elements
    exact = variant == "exact"
    o, g, U, nu = make_case(oracle_mod, 4, 4, 12, 1, "quadratic")
    whole = Dycore(g, 1, nu, exact=exact)
    plans = build_plans(g, partition_elements(g.NF, nranks))
    parts = [Dycore(P.local_grid(g), 1, nu, exact=exact, halo=P) for P in plans]
    grp = PartGroup(parts)
    # tendency
    F1 = whole.fcn(U)
    Ul = [_dev(P.restrict(U)) for P in plans]
    Fl = [torch.empty_like(u) for u in Ul]
    grp.fcn(Ul, Fl)
    for P, f in zip(plans, Fl):
        assert np.array_equal(_host(f), F1[:, P.dofs, :])
    if exact:
        assert np.array_equal(F1, o.rhs(U))
    # steps
    V = U.copy(order="F")
    whole.time_stepper(V, 300.0, 3)
    grp.time_stepper(Ul, 300.0, 3)
    for P, u in zip(plans, Ul):
        assert np.array_equal(_host(u), V[:, P.dofs, :])
    if exact:
        assert np.array_equal(V, o.ros_step(U, 300.0, 3))
    # the global mass integral: each DOF counted on its owning rank
    m = sum(p.mass_integral(_host(u).copy(order="F")) for p, u in zip(parts, Ul))
    assert abs(m - whole.mass_integral(V)) <= 1e-13 * abs(m)
    for p in parts:
        p.close()
    whole.close()


def test_decomposed_grid_rejects_mixed_form(oracle_mod, built_lib, cuda_ok):
    from cgd_b200 import CgdError, Dycore
    from cgd_b200.parallel import build_plans, partition_elements
    o, g, U, nu = make_case(oracle_mod, 3, 4, 6, 0)
    P = build_plans(g, partition_elements(g.NF, 2))[0]
    with pytest.raises(CgdError) as e:
        Dycore(P.local_grid(g), 0, nu, precision="mixed", halo=P)
    assert e.value.code == -7


def _group_fcn(parts, plans, U):
    import torch
    from cgd_b200 import PartGroup
    Ul = [_dev(P.restrict(U)) for P in plans]
    Fl = [torch.empty_like(u) for u in Ul]
    PartGroup(parts).fcn(Ul, Fl)
    return [_host(f) for f in Fl]


@pytest.mark.parametrize("case", [(3, 4, 17, 1), (4, 3, 16, 0), (4, 2, 18, 2), (5, 1, 33, 0)])
@pytest.mark.parametrize("stretch", ["uniform", "quadratic"])
def test_flat_parts(oracle_mod, built_lib, cuda_ok, case, stretch):
    """The fast build's flat kernels on the parts (layers given) and on the
    whole grid: the same bits, whichever element a part begins with."""
    from cgd_b200 import Dycore
    from cgd_b200.parallel import build_plans, partition_elements
    n, p, nz, nt = case
    o, g, U, nu = make_case(oracle_mod, n, p, nz, nt, stretch)
    whole = Dycore(g, nt, nu)
    assert whole.flat_form()
    F = whole.fcn(U)
    for nranks in (2, 5):
        plans = build_plans(g, partition_elements(g.NF, nranks))
        parts = [Dycore(P.local_grid(g), nt, nu, halo=P) for P in plans]
        assert all(d.flat_form() for d in parts)
        for P, f in zip(plans, _group_fcn(parts, plans, U)):
            assert np.array_equal(f, F[:, P.dofs, :])
        for d in parts:
            d.close()
    whole.close()


def test_one_part_off_the_flat_form(oracle_mod, built_lib, cuda_ok):
    """One element of the last part has a perturbed metric: the whole grid runs
    the general kernels, and so do all parts of the group, bit for bit."""
    import dataclasses
    from cgd_b200 import Dycore
    from cgd_b200.parallel import build_plans, partition_elements
    o, g, U, nu = make_case(oracle_mod, 4, 4, 12, 1, "quadratic")
    dX = np.array(g.dXdxI, order="F")
    dX[..., 5, -1] *= 1.0 + 1e-3   # one level: no product of horizontal and vertical factors
    g = dataclasses.replace(g, dXdxI=dX)
    whole = Dycore(g, 1, nu)
    assert not whole.flat_form()
    plans = build_plans(g, partition_elements(g.NF, 3))
    parts = [Dycore(P.local_grid(g), 1, nu, halo=P) for P in plans]
    before = [d.flat_form() for d in parts]
    assert before[0] and not before[-1]
    F = whole.fcn(U)
    for P, f in zip(plans, _group_fcn(parts, plans, U)):
        assert np.array_equal(f, F[:, P.dofs, :])
    assert [d.flat_form() for d in parts] == before
    # ranks of their own agree with cgd_set_flat_form
    for d in parts:
        d.set_flat_form(False)
        assert not d.flat_form()
        d.set_flat_form(True)
    assert [d.flat_form() for d in parts] == before
    for d in parts + [whole]:
        d.close()


def test_parts_without_layers(oracle_mod, built_lib, cuda_ok):
    """Parts that were not given the whole grid's layers run the general
    kernels: the same bits as a whole grid that does."""
    import dataclasses
    from cgd_b200 import Dycore
    from cgd_b200.parallel import build_plans, partition_elements
    o, g, U, nu = make_case(oracle_mod, 4, 4, 12, 1, "quadratic")
    whole = Dycore(g, 1, nu)
    whole.set_flat_form(False)
    F = whole.fcn(U)
    plans = build_plans(g, partition_elements(g.NF, 3))
    parts = [Dycore(dataclasses.replace(P.local_grid(g), layers=None), 1, nu, halo=P) for P in plans]
    assert not any(d.flat_form() for d in parts)
    for P, f in zip(plans, _group_fcn(parts, plans, U)):
        assert np.array_equal(f, F[:, P.dofs, :])
    for d in parts + [whole]:
        d.close()
