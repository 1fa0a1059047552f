"""Work counters and per-pass diagnostics describe the last evaluation, whatever is set or
asked for after it, and asking for them leaves the handle as it was."""
import numpy as np
import pytest

import d3_systems as S
from d3_b200 import OPT_ATM_LIST_CAPACITY, OPT_BIN_DIVISOR, OPT_PRECISION, D3

pytestmark = pytest.mark.gpu

RC = dict(rc=40.0, rc_cn=25.0, rc_atm=24.0)


def short_cell(n=24, seed=2):
    """A cell shorter than rc_ATM: lists hold several images of one atom, which the
    reference's enumeration visits more than once."""
    edge = (n / 0.1) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [0.05, -0.1, 1.0]]), seed=seed)


def handle(s, precision=0):
    d = D3(s["Z"], len(s["Z"]), **RC)
    d.set_option(OPT_PRECISION, precision)
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    return d


@pytest.mark.parametrize("precision", [0, 1])
def test_diagnostics_after_the_geometry_changed(precision):
    s = short_cell()
    d = handle(s, precision)
    d.compute()
    _, before = d.pass_times()
    terms = d.pass_terms()
    pairs = d.atm_pairs()
    for change in (lambda: d.set_cell(1.3 * s["cell"]), lambda: d.set_option(OPT_BIN_DIVISOR, 3)):
        d.set_cell(s["cell"])
        d.compute()
        change()
        _, after = d.pass_times()
        assert after.tolist() == before.tolist()
        # FP64 sums of the same terms in another order; the FP32 form's last bits
        np.testing.assert_allclose(d.pass_terms(), terms, rtol=0, atol=1e-12 if precision == 0 else 1e-8)
        rows = d.atm_pairs()
        assert sorted(map(tuple, rows.tolist())) == sorted(map(tuple, pairs.tolist()))
        d.set_option(OPT_BIN_DIVISOR, 6)
    d.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_counters_of_a_replayed_graph(precision):
    import torch

    s = short_cell()
    far = short_cell(seed=9)["pos"]
    d = handle(s, precision)
    d.compute()
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        d.set_positions_device(pos.data_ptr(), stream.cuda_stream)
        d.compute_async(stream.cuda_stream)
    torch.cuda.synchronize()
    d.compute()  # (a capture leaves the timers' events to the next direct evaluation)
    d.pass_times()
    d.pass_terms()
    pos.copy_(torch.tensor(far, dtype=torch.float64))
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.replay()
    torch.cuda.synchronize()
    _, cnt = d.pass_times()
    ref = handle(dict(s, pos=far), precision)
    ref.compute()
    _, want = ref.pass_times()
    assert cnt.tolist() == want.tolist()
    np.testing.assert_allclose(d.pass_terms(), ref.pass_terms(), rtol=0, atol=1e-12 if precision == 0 else 1e-8)
    del graph
    ref.close()
    d.close()


def test_diagnostics_leave_the_lists_and_the_status_alone():
    """The reference's lists hold both (a, T) and (a, -T), so they are longer than the
    evaluation's: with a capacity that just holds the latter, asking for the former must not
    move the evaluation's buffer (a captured graph keeps its address) nor report an overflow."""
    s = short_cell(n=4)
    d = handle(s)
    d.compute()
    rows = d.atm_pairs()
    own = int((rows[:, 0] == rows[:, 1]).sum())  # images of the apex atom itself
    assert own > 0 and own % 2 == 0
    exact = len(rows) - own // 2
    d.set_option(OPT_ATM_LIST_CAPACITY, exact)
    e0 = d.compute()[0]
    assert d.atm_list_capacity() == exact
    d.pass_terms()
    assert d.atm_list_capacity() == exact and d.fetch_status() == 0
    assert len(d.atm_pairs()) == len(rows)
    assert d.atm_list_capacity() == exact and d.fetch_status() == 0
    assert abs(d.compute()[0] - e0) <= 1e-12 * abs(e0)
    d.close()
