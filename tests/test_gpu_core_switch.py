"""tce_set_tensor_cores(0) and blocks-only handles: every call runs the FP64
CUDA-core kernels, which sum every Bessel order.

That form takes a quartet's primitive quartets in one fixed order (one 32-node
chunk), whatever else is in the launch, so each entry point is held bitwise to
tce_rule_blocks, or to the unsharded call, on the same handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _some_quartets(eng, n, seed):
    """Shell quartets with the first shell in the unit cell, the largest block among them."""
    sh = eng.shells()
    nuc = eng.info()["nshuc"]
    rng = np.random.default_rng(seed)
    q = [(int(rng.integers(nuc)),) + tuple(int(x) for x in rng.integers(0, len(sh), 3)) for _ in range(n)]
    big = max(range(nuc), key=lambda s: sh[s][1])
    return q + [(big, big, big, big)]


def _check_blocks(eng, seed):
    q = _some_quartets(eng, 24, seed)
    K, _, off = eng.rule_blocks(-1, np.array(q), mode=2)
    assert np.abs(K).max() > 1e-2
    for i, s in enumerate(q):
        ref = K[off[i]:off[i + 1]]
        for call in (eng.ERI_shell_block, eng.ERI_shell_block_noalloc):
            got = call(*s, mode=2).ravel(order="F")
            assert np.array_equal(got, ref), (call.__name__, s, np.abs(got - ref).max())


@pytest.mark.parametrize("name,ncell", [("h_chain64", (6, 1, 1)), ("h2_sheet", (2, 2, 1)), ("li_cube", (2, 2, 2))])
def test_shell_blocks_follow_the_switch(systems, name, ncell):
    from william_ci_b200.engine import Engine
    with Engine(systems(name, ncell)) as eng:
        eng.set_tensor_cores(False)
        _check_blocks(eng, 3)


@pytest.mark.parametrize("name,ncell", [("h_chain64", (6, 1, 1)), ("h2_sheet", (2, 2, 1))])
def test_shell_blocks_of_a_blocks_only_handle(systems, name, ncell):
    from william_ci_b200.engine import Engine
    with Engine(systems(name, ncell), blocks_only=True, prim_screen=False) as eng:
        _check_blocks(eng, 4)


@pytest.mark.parametrize("name,ncell", [("h_chain64", (4, 1, 1)), ("h2_sheet", (2, 2, 1))])
def test_stored_integrals_of_a_shard_follow_the_switch(systems, name, ncell):
    from william_ci_b200.engine import Engine
    with Engine(systems(name, ncell)) as eng:
        eng.set_tensor_cores(False)
        ref = eng.ERI_integral_toroidal()
        assert np.abs(ref).max() > 0.1
        eng.set_shard(1, 2)
        got = eng.ERI_integral_toroidal()
    assert np.array_equal(got, ref), np.abs(got - ref).max()


def test_list_forms_of_each_setting_are_kept_apart(systems):
    """The generic classes are numbered by p and d shells with the tensor cores on, by
    d shells with them off: a form set for one is no form of the other's lists."""
    from william_ci_b200.engine import TCE_METHOD_LEARNED, Engine
    with Engine(systems("h2_sheet", (2, 2, 1))) as eng:
        eng.lg_setup(n_train=1500, seed=2026, epochs=20)
        eng.set_method(TCE_METHOD_LEARNED)
        generic = [i for i, w in enumerate(eng.lg_lists()) if w["kind"] == 0]
        eng.lg_set_list_form(generic[-1], 0)          # kept over the other setting
        chosen = eng.lg_lists()
        assert chosen[generic[-1]]["tc"] == 0
        eng.set_tensor_cores(False)
        for i, w in enumerate(eng.lg_lists()):
            if w["kind"] == 0:
                assert w["cls"] <= 4
                eng.lg_set_list_form(i, 0)
        eng.set_tensor_cores(True)
        assert eng.lg_lists() == chosen
