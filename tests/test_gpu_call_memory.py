"""Device memory of single calls: the workspaces of tce_ao_to_kmo, tce_dfmp2 and
tce_dfmp2_energy come from a pool that all handles share, and a call needs no
more at once than its buffers that live at the same time."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def _chain(n):
    import pyoracle
    from william_ci_b200 import df as DF
    from william_ci_b200 import system as S
    cell, basis = S.workload("h_chain64")
    cell = S.scaled_down(cell, (n, 1, 1))
    s, aux = S.build_system(cell, basis), S.build_system(cell, DF.even_tempered_aux([1]))
    pyoracle.normalize(s)
    pyoracle.normalize(aux)
    return s, aux


def _orbitals(n, nf):
    rng = np.random.default_rng(5)
    C = np.linalg.qr(rng.standard_normal((n, nf, nf)) + 1j * rng.standard_normal((n, nf, nf)))[0]
    eps = np.sort(rng.uniform(0.1, 2.0, (n, nf)), axis=1)
    eps[:, 0] = -0.5
    occ = np.zeros((n, nf), dtype=np.int32)
    occ[:, 0] = 2
    return C, eps, occ


class _Filled:
    """The device with only `room` bytes free."""

    def __init__(self, room):
        self.room = room

    def __enter__(self):
        import torch
        gc.collect()
        torch.cuda.empty_cache()
        self.t = torch.empty(_free() - self.room, dtype=torch.uint8, device="cuda")
        return _free()

    def __exit__(self, *a):
        import torch
        del self.t
        torch.cuda.empty_cache()


def test_handles_share_the_workspaces():
    """Calls on three handles hold no more than calls on one, and nothing when the
    handles are gone (but for what the driver itself keeps, below 64 MB)."""
    from william_ci_b200 import df as DF
    from william_ci_b200.engine import Engine
    s, aux = _chain(20)
    C, eps, occ = _orbitals(20, s.nfuc)
    gc.collect()
    base = _free()
    engs, dfs = [Engine(s) for _ in range(3)], [DF.DeviceDF(s, aux) for _ in range(3)]
    for e in engs:
        e.ERI_integral_toroidal()
    before = _free()

    def calls(e, d):
        out = [e.ao_to_kmo(C, (0, 1), (1, s.nfuc))]
        return out + [d.dfmp2(C, eps, occ, mode=m)["emp2"] for m in (0, 1)]

    ref = calls(engs[0], dfs[0])
    one = _free()
    assert before - one <= 1100 * MB
    for e, d in zip(engs, dfs):
        got = calls(e, d)
        assert np.array_equal(got[0], ref[0]) and abs(got[1] - ref[1]) <= 1e-12 * abs(ref[1])
    assert one - _free() <= 2 * MB
    del e, d, engs, dfs, calls
    gc.collect()
    assert _free() >= base - 64 * MB


def test_dfmp2_peak_memory():
    """96 cells, split-BF16: G takes 354 MB, L 12 MB, the cell sums 170 MB, which
    are gone before G is made: 440 MB do."""
    from william_ci_b200 import df as DF
    s, aux = _chain(8)
    C, eps, occ = _orbitals(8, s.nfuc)
    small = DF.DeviceDF(s, aux)
    small.dfmp2(C, eps, occ, mode=1)               # loads the kernels
    s, aux = _chain(96)
    C, eps, occ = _orbitals(96, s.nfuc)
    d = DF.DeviceDF(s, aux)
    with _Filled(440 * MB) as room:
        assert room < 460 * MB
        tight = d.dfmp2(C, eps, occ, mode=1)["emp2"]
    assert abs(tight - d.dfmp2(C, eps, occ, mode=1)["emp2"]) <= 1e-12 * abs(tight)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("ncl,no,nv,nau,room", [((96, 1, 1), 1, 5, 16, 200), ((3, 3, 3), 2, 3, 7, 8)])
def test_dfmp2_energy_without_room_for_g(ncl, no, nv, nau, room, mode):
    """Where G (354 and 11 MB) does not fit, the FP64 energy comes from the kernel
    that holds no G, and the split-BF16 one is refused with an error."""
    from william_ci_b200.engine import TCEError, dfmp2_energy
    rng = np.random.default_rng(2)
    N = int(np.prod(ncl))
    L = (rng.standard_normal((no, nv, nau, N, N)) + 1j * rng.standard_normal((no, nv, nau, N, N))) * 0.05
    args = (ncl, L, -0.5 - rng.random((N, no)), np.full((N, no), 2, dtype=np.int32), 0.2 + rng.random((N, nv)),
            np.zeros((N, nv), dtype=np.int32))
    args[2][:, 0] = args[4][:, 0] = 0.0                        # zero-gap terms: left out and counted
    args[3][2, no - 1] = 0
    ref = dfmp2_energy(*args, mode=mode)
    assert ref["nzero"] > 0
    with _Filled(room * MB):
        if mode == 0:
            got = dfmp2_energy(*args, mode=0)
            assert abs(got["emp2"] - ref["emp2"]) <= 1e-12 * abs(ref["emp2"]) and got["nzero"] == ref["nzero"]
        else:
            with pytest.raises(TCEError):
                dfmp2_energy(*args, mode=1)
    again = dfmp2_energy(*args, mode=mode)
    assert abs(again["emp2"] - ref["emp2"]) <= 1e-12 * abs(ref["emp2"])


def test_kmo_one_k4_at_a_time_when_memory_is_short():
    """20 cells: four k4 at a time take 70 MB, one at a time 20 MB."""
    from william_ci_b200.engine import Engine
    s, _ = _chain(20)
    C = _orbitals(20, s.nfuc)[0]
    with Engine(s) as e:
        e.ERI_integral_toroidal()
        ref = e.ao_to_kmo(C, (0, 1), (1, s.nfuc))
        with _Filled(48 * MB):
            assert np.array_equal(e.ao_to_kmo(C, (0, 1), (1, s.nfuc)), ref)
