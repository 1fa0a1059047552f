"""Work space of the FP64 three-body kernels: sized by what the handle's structures need, and
never allocated while a stream is being captured."""
import numpy as np
import pytest

import d3_systems as S
from d3_b200 import OPT_PRECISION, D3

pytestmark = pytest.mark.gpu


def box(n, density, seed=3):
    edge = (n / density) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [0.05, -0.1, 1.0]]), seed=seed)


def handle(s, **rc):
    d = D3(s["Z"], len(s["Z"]), **rc)
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    return d


@pytest.mark.parametrize("kind,mib", [("crystal", 96), ("molecule", 32), ("sparse", 64)])
def test_device_memory_of_small_handles(kind, mib):
    """A 16-atom cell with rc_ATM 40 bohr has lists of about 2,000 entries: 148 CTAs of up to
    4,096 entries of 96 bytes and the rows of one of nine splits, 75 MiB."""
    import torch

    if kind == "crystal":
        s, rc = S.gtest_bcc_fe(), dict(rc=95.0, rc_cn=40.0, rc_atm=40.0)
    elif kind == "molecule":
        s, rc = S.gtest_small_system(), dict(rc=46.0, rc_cn=30.0, rc_atm=20.0)
    else:
        s, rc = box(500, 0.005), dict(rc=60.0, rc_cn=30.0, rc_atm=25.0)
    handle(s, **rc).compute()  # the context's own memory
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    d = handle(s, **rc)
    d.compute()
    torch.cuda.synchronize()
    used = (before - torch.cuda.mem_get_info()[0]) / 2 ** 20
    d.close()
    assert used <= mib


def replay(d, s, stream):
    import torch

    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        d.set_positions_device(pos.data_ptr(), stream.cuda_stream)
        assert d.compute_async(stream.cuda_stream) == 0
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    assert d.fetch_status() == 0
    out = d.fetch_results()
    del graph
    return out


@pytest.mark.parametrize("n,rc_atm,shrink", [
    (64, 11.5, 0.985),   # 47 entries expected per list, then 49: on both sides of the rule for block pairs
    (20, 30.0, 0.95),    # lists 17 % longer
    (400, 30.0, 0.95),
])
def test_capture_right_after_a_denser_cell(n, rc_atm, shrink):
    """One evaluation sizes the lists (with their margin); a capture after a smaller cell was
    set runs with the work space there is."""
    import torch

    s = box(n, 0.1)
    rc = dict(rc=40.0, rc_cn=25.0, rc_atm=rc_atm)
    d = handle(s, **rc)
    d.compute()
    dense = dict(s, cell=shrink * s["cell"], pos=shrink * s["pos"])
    d.set_cell(dense["cell"])
    e, f, st = replay(d, dense, torch.cuda.Stream())
    ref = handle(dense, **rc)
    e1, f1, s1 = ref.compute()
    assert abs(e - e1) <= 1e-11 * abs(e1)
    assert np.abs(f - f1).max() <= 1e-9 and np.abs(st - s1).max() <= 1e-11
    ref.close()
    d.close()


def test_capture_right_after_a_change_of_form():
    import torch

    s = box(100, 0.1)
    rc = dict(rc=40.0, rc_cn=25.0, rc_atm=25.0)
    d = handle(s, **rc)
    d.set_option(OPT_PRECISION, 1)
    d.compute()
    d.set_option(OPT_PRECISION, 0)
    e, f, _ = replay(d, s, torch.cuda.Stream())
    ref = handle(s, **rc)
    e1, f1, _ = ref.compute()
    assert abs(e - e1) <= 1e-11 * abs(e1) and np.abs(f - f1).max() <= 1e-9
    ref.close()
    d.close()


@pytest.mark.parametrize("n,pad", [(1500, 30.0), (300, 20.0)])
def test_lists_longer_than_the_room_for_them(n, pad):
    """Clusters in vacuum, whose lists are many times the mean that the room is sized by (weighted
    and weight-free cells): by block pairs or rows, whole or in parts, as the FP64 oracle."""
    import oracle

    s = box(n, 0.1)
    edge = float(s["cell"][0, 0]) + pad
    s = dict(s, cell=np.eye(3) * edge)
    rc = dict(rc=45.0, rc_cn=25.0, rc_atm=40.0)
    d = handle(s, **rc)
    e, f, st = d.compute()
    d.close()
    r = oracle.compute(s["pos"], s["Z"], s["cell"], c6_mode=1, **rc)
    assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
    assert np.abs(f - r["forces"]).max() <= 1e-7
    assert np.abs(st - r["stress"]).max() <= 1e-7
