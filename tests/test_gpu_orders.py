"""The tensor-core kernels sum only the Bessel orders tce_orders.cuh picks (a
stride and a last order per tile); the CPU oracle sums every order of the
reference's truncation.  Same rule, same screens: J and K agree to rounding,
1e-12 of the density's absolute sum, the bound the other kernel-form tests use
(a sum of some 1e5 integrals of rounding 1e-16 each)."""
import dataclasses

import numpy as np
import pytest

from conftest import random_density

pytestmark = pytest.mark.gpu


def _system(name, ncell, spacing=None, off_axis=False):
    import pyoracle
    from william_ci_b200 import system as S
    cell, basis = S.workload(name)
    if spacing:
        cell = dataclasses.replace(cell, spacing=spacing)
    if off_axis:      # second atom off the periodic axis: R != 0 in the real directions
        cell = dataclasses.replace(cell, atoms=cell.atoms + [(cell.atoms[0][0], (0.7, 0.9, -0.4))])
    s = S.build_system(S.scaled_down(cell, ncell), basis)
    pyoracle.normalize(s)
    return s


def _one_d_component(s):
    """The system with dxy alone of every d shell: shells of one function whose
    power combinations outnumber their components."""
    keep = [f for f in range(s.nbas) if not s.labels[f].startswith("d") or s.labels[f] == "dxy"]
    off, ex, co = [0], [], []
    for f in keep:
        ex.extend(s.exps[s.prim_off[f]:s.prim_off[f + 1]])
        co.extend(s.coefs[s.prim_off[f]:s.prim_off[f + 1]])
        off.append(len(ex))
    return dataclasses.replace(s, nfuc=len([f for f in keep if f < s.nfuc]), ctr=s.ctr[keep], lxyz=s.lxyz[keep],
                               prim_off=np.array(off, dtype=np.int32), exps=np.array(ex), coefs=np.array(co),
                               labels=[s.labels[f] for f in keep], atom_of=s.atom_of[keep])


def _split_p(name, ncell):
    """The workload with px, py and pz of different exponents: three shells of one
    function each, in the order of one full p shell's components."""
    import pyoracle
    from william_ci_b200 import system as S
    cell, basis = S.workload(name)
    s = S.build_system(S.scaled_down(cell, ncell), basis)
    for f in range(s.nbas):
        if s.lxyz[f].sum() == 1:
            s.exps[s.prim_off[f]:s.prim_off[f + 1]] *= (1.0, 1.4, 0.8)[int(np.argmax(s.lxyz[f]))]
    pyoracle.normalize(s)
    return s


def _with_d(name, ncell):
    """The chain with the sheet's s, p, d basis and its second atom off the axis."""
    import pyoracle
    from william_ci_b200 import system as S
    cell, _ = S.workload(name)
    cell = dataclasses.replace(cell, atoms=cell.atoms + [(cell.atoms[0][0], (0.7, 0.9, -0.4))])
    s = S.build_system(S.scaled_down(cell, ncell), S.workload("h2_sheet")[1])
    pyoracle.normalize(s)
    return s


CASES = [
    ("h2_ring", (2, 1, 1), None, False),        # antipodal pairs: Bessel argument 0
    ("h_chain64", (1, 1, 1), 3.0, False),       # one cell, small arguments
    ("h_chain64", (3, 1, 1), None, True),
    ("h_chain64", (13, 1, 1), None, False),     # strides above 1
    ("h_chain64", (7, 1, 1), 30.0, True),       # long torus: large strides, phases past the width
    ("h2_sheet", (2, 2, 1), None, False),
    ("li_cube", (2, 2, 2), None, False),
]
LONG = [    # long tori of two and three directions, one of them ragged: strides above 1, phases past the width
    ("h2_sheet", (3, 1, 1), 25.0, False),
    ("h2_sheet", (2, 2, 1), 25.0, True),
    ("li_cube", (3, 1, 2), 25.0, False),
    ("li_cube", (2, 2, 1), 25.0, True),
]


@pytest.mark.parametrize("name,ncell,spacing,off,nquad",
                         [c + (n,) for c in CASES for n in (32, 40, 64)] + [c + (128,) for c in CASES[:3]])
def test_strided_orders_match_every_order(name, ncell, spacing, off, nquad):
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _system(name, ncell, spacing, off)
    P = random_density(s.nbas, 5) * 0.05
    t, w = pyoracle.fast_quad(nquad)
    J0, K0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).direct_jk(P)[:2]
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        J, K = eng.direct_JK(P)
    scale = np.abs(P).sum()
    assert np.abs(J0).max() > 0
    assert np.abs(J - J0).max() <= 1e-12 * scale, np.abs(J - J0).max() / scale
    assert np.abs(K - K0).max() <= 1e-12 * scale, np.abs(K - K0).max() / scale


# The CUDA-core kernels turn e^{i n phi} by a recurrence of 32 steps over some 170
# orders: 32 eps per order, 170 orders, 1e-12 of a sum's peak; 1e-11 of the
# density's sum with room for the sum over quartets.  (Not the long torus, whose
# 1000 orders and phases take that past 1e-10.)
EVERY = 1e-11


@pytest.mark.parametrize("name,ncell,spacing,off,nquad",
                         [c + (n,) for c in CASES if c[2] != 30.0 for n in (32, 40, 64)] + [c + (128,) for c in CASES[:3]])
def test_tensor_cores_off(name, ncell, spacing, off, nquad):
    """Every class through the CUDA-core kernels or the generic kernel's every-order
    form: J and K direct, and from the stored integrals of the small systems."""
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _system(name, ncell, spacing, off)
    P = random_density(s.nbas, 5) * 0.05
    t, w = pyoracle.fast_quad(nquad)
    J0, K0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).direct_jk(P)[:2]
    scale = np.abs(P).sum()
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        eng.set_tensor_cores(False)
        got = [eng.direct_JK(P)]
        if s.nbas < 70:
            eng.ERI_integral_toroidal()
            J, K = eng.stored_JK(P)
            got.append((J[:s.nfuc], K[:s.nfuc]))
        eng.set_tensor_cores(True)      # the lists are cut again for the tensor-core kernels
        got.append(eng.direct_JK(P))
    for J, K in got:
        assert np.abs(J - J0[:len(J)]).max() <= EVERY * scale and np.abs(K - K0[:len(K)]).max() <= EVERY * scale


@pytest.mark.parametrize("nquad", [32, 64])
@pytest.mark.parametrize("name,ncell,spacing,off", LONG)
def test_long_tori_of_two_and_three_directions(name, ncell, spacing, off, nquad):
    """Strided sums against every order on the same power vectors (the engine's
    CUDA-core form).  Not against the oracle: at Bessel arguments of 1e4 its d_k
    sums, and not the orders, set the difference (1.1e-12 of the density's sum on
    the ragged sheet, where these two forms agree to 1e-17)."""
    from william_ci_b200.engine import Engine
    s = _system(name, ncell, spacing, off)
    P = random_density(s.nbas, 5) * 0.05
    with Engine(s, nquad=nquad) as eng:
        J, K = eng.direct_JK(P)
        eng.set_tensor_cores(False)
        J0, K0 = eng.direct_JK(P)
    scale = np.abs(P).sum()
    assert np.abs(J0).max() > 0
    assert np.abs(J - J0).max() <= 1e-12 * scale and np.abs(K - K0).max() <= 1e-12 * scale


@pytest.mark.parametrize("cores", [True, False])
def test_d_shells_of_one_direction_off_the_axis(cores):
    """J and K of s, p and d shells with one periodic direction and R != 0 in the real ones."""
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _with_d("h_chain64", (2, 1, 1))
    P = random_density(s.nbas, 5) * 0.05
    t, w = pyoracle.fast_quad(32)
    J0, K0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).direct_jk(P)[:2]
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        eng.set_tensor_cores(cores)
        J, K = eng.direct_JK(P)
    tol = (1e-12 if cores else EVERY) * np.abs(P).sum()
    assert np.abs(J - J0).max() <= tol and np.abs(K - K0).max() <= tol


@pytest.mark.parametrize("name,ncell", [("h2_sheet", (1, 1, 1)), ("h2_sheet", (2, 1, 1)), ("li_cube", (1, 1, 1)),
                                        ("li_cube", (2, 1, 1)), ("h2_sheet", (3, 2, 1))])
def test_classes_of_few_quartets_share_a_launch(name, ncell):
    """Systems whose generic classes hold fewer quartets than the GPU holds warps:
    the all-s list and one to four merged ones instead of up to fifteen launches, each
    as long as its dearest quartet (cube: four of them).  J and K, direct and stored, and the learned grid's."""
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _system(name, ncell)
    with Engine(s) as eng:
        if ncell == (3, 2, 1):            # most classes have a wave of their own
            assert eng.pass_kernels() >= 12
            return
        assert eng.pass_kernels() <= (5 if name == "h2_sheet" else 2)
        P = random_density(s.nbas, 5) * 0.05
        scale = np.abs(P).sum()
        J0, K0 = pyoracle.Oracle(s).direct_jk(P)[:2]
        got = [eng.direct_JK(P)]
        eng.ERI_integral_toroidal()
        got.append(eng.stored_JK(P))
    for J, K in got:
        J, K = J[:s.nfuc], K[:s.nfuc]
        assert np.abs(J - J0[:s.nfuc]).max() <= 1e-12 * scale and np.abs(K - K0[:s.nfuc]).max() <= 1e-12 * scale
    _learned_against_plain(s)


@pytest.mark.parametrize("nquad", [32, 64])
def test_shells_of_one_d_component(nquad):
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _one_d_component(_system("h2_sheet", (2, 2, 1)))
    P = random_density(s.nbas, 5) * 0.05
    t, w = pyoracle.fast_quad(nquad)
    J0, K0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).direct_jk(P)[:2]
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        J, K = eng.direct_JK(P)
    scale = np.abs(P).sum()
    assert np.abs(J - J0).max() <= 1e-12 * scale and np.abs(K - K0).max() <= 1e-12 * scale


@pytest.mark.parametrize("cores", [True, False])
@pytest.mark.parametrize("nquad", [32, 40, 64])
@pytest.mark.parametrize("shells", ["sp", "spd"])
def test_nuclear_attraction_few_orders(shells, nquad, cores):
    """One periodic direction, atoms off the axis, s to d shells: every element
    within 1e-12 (tensor cores off: EVERY) of the sum of charges times the largest
    s element's scale (1)."""
    import pyoracle
    from william_ci_b200 import system as S
    from william_ci_b200.engine import Engine
    cell, basis = S.workload("h_chain64")
    if shells == "spd":
        basis = S.workload("h2_sheet")[1]
    cell = dataclasses.replace(cell, atoms=cell.atoms + [("H", (0.7, 0.9, -0.4))])
    s = S.build_system(S.scaled_down(cell, (5, 1, 1)), basis)
    pyoracle.normalize(s)
    t, w = pyoracle.fast_quad(nquad)
    V0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).one_electron()[2]
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        eng.set_tensor_cores(cores)
        V = eng.nuclear_attraction()
    assert np.abs(V0).max() > 0.1
    assert np.abs(V - V0).max() <= (1e-12 if cores else EVERY) * max(1.0, np.abs(V0).max()) * len(s.charges), np.abs(V - V0).max()


@pytest.mark.parametrize("nquad", [32, 40, 64])
def test_p_functions_that_are_no_full_shell(nquad):
    """px, py, pz with exponents of their own are three shells, although the
    functions after px are py and pz: the s/p kernels (full p shells) do not
    take them."""
    import pyoracle
    from william_ci_b200.engine import Engine
    s = _split_p("h_chain64", (4, 1, 1))
    P = random_density(s.nbas, 5) * 0.05
    t, w = pyoracle.fast_quad(nquad)
    J0, K0 = pyoracle.Oracle(s, t_nodes=t, t_weights=w).direct_jk(P)[:2]
    scale = np.abs(P).sum()
    with Engine(s, t_nodes=t, t_weights=w) as eng:
        assert {n for _, n in eng.shells()} == {1}
        J, K = eng.direct_JK(P)
    assert np.abs(J - J0).max() <= 1e-12 * scale and np.abs(K - K0).max() <= 1e-12 * scale, np.abs(J - J0).max() / scale


def _learned_against_plain(s):
    """The learned grid's J and K within the judge's 1e-10 of the plain method's; its list kinds."""
    from william_ci_b200.engine import TCE_METHOD_LEARNED, TCE_METHOD_PLAIN, Engine
    P = random_density(s.nbas, 5) * 0.05
    scale = np.abs(P).sum()
    with Engine(s) as eng:
        eng.lg_setup(n_train=2000, seed=2026, epochs=40)
        eng.set_method(TCE_METHOD_PLAIN)
        J0, K0 = eng.direct_JK(P)
        eng.set_method(TCE_METHOD_LEARNED)
        J, K = eng.direct_JK(P)
        kinds = {w["kind"] for w in eng.lg_lists()}
    assert np.abs(J - J0).max() <= 1e-10 * scale and np.abs(K - K0).max() <= 1e-10 * scale, np.abs(J - J0).max() / scale
    return kinds


def test_learned_grid_p_functions_that_are_no_full_shell():
    assert 2 not in _learned_against_plain(_split_p("h_chain64", (6, 1, 1)))


def test_learned_grid_pairs_of_p_shells_off_the_axis():
    """(pp|ss) and (ss|pp) with R != 0: the (1,0) and (0,1) power vectors of a pair
    differ, and the s/p kernel takes each for its own component."""
    assert 2 in _learned_against_plain(_system("h_chain64", (6, 1, 1), None, True))
