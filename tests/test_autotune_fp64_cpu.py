"""The autotuner's FP64 search on the host: the row kernel's default shape is a candidate, a
handle whose lists go to block pairs is left at the defaults, and its options stay."""
import pytest

import d3_autotune
from d3_b200 import OPT_ATM_CTAS_PER_SM, OPT_ATM_SCHEDULE, OPT_ATM_TILE


class Handle:
    def __init__(self, blocks, schedule=0):
        self.blocks, self.options = blocks, {OPT_ATM_SCHEDULE: schedule}
        self.noise = 0.0

    def set_option(self, k, v):
        self.options[k] = v

    def compute(self):
        pass

    def launches_per_eval(self):
        return 22 if self.blocks and self.options[OPT_ATM_SCHEDULE] == 0 else 21

    def pass_times(self):
        o = self.options.get
        if self.blocks and o(OPT_ATM_SCHEDULE) == 0:
            self.noise -= 0.01  # the knobs do nothing: every trial a little faster
            atm = 10.0 + self.noise
        else:  # whole lists in one CTA per SM are the fastest
            atm = 10.0 + (1.0 if o(OPT_ATM_TILE, 0) else 0.0) + (1.0 if o(OPT_ATM_CTAS_PER_SM, 0) > 1 else 0.0)
        return {"bin": 0.0, "cn": 0.0, "twobody": 1.0, "atm_list": 0.0, "atm": atm, "chain": 0.0, "finalize": 0.0}, None


@pytest.mark.parametrize("blocks,schedule", [(False, 0), (True, 0), (True, 1)])
def test_default_shape_is_kept_where_it_is_the_fastest_or_nothing_depends_on_it(blocks, schedule):
    h = Handle(blocks, schedule)
    res = d3_autotune.tune(h, "k|p0", repeats=1, use_cache=False)
    assert (res["atm_tile"], res["atm_ctas_per_sm"]) == (0, 0)
    assert (h.options[OPT_ATM_TILE], h.options[OPT_ATM_CTAS_PER_SM]) == (0, 0)
    assert h.options[OPT_ATM_SCHEDULE] == schedule


def test_entries_of_the_removed_kernel_are_not_reused(monkeypatch):
    monkeypatch.setattr(d3_autotune, "gpu_name", lambda: "gpu")
    key = d3_autotune.workload_key(1000, 1e4, 95.0, 40.0, 40.0, 0)
    assert not key.startswith("v2|") and key.endswith("|p0")
