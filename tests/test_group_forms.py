"""CPU checks of what chooses between the plan group's two forms: the autotuner
searches only options that count in the current form, and bench.py times each
form with the option that selects it, on a stand-in for the device batch."""
import types

import pytest

torch = pytest.importorskip("torch")


class FakeBatch:
    def __init__(self, form):
        self.options = {5: form, 4: 1}
        self.log = []                                   # (what, form, one stream) of each timing
        self.captured = None
        self.applied = None
        self.group = types.SimpleNamespace(set_option=self.options.__setitem__, get_option=self.options.get)
        self.device, self.buckets, self.count, self.plans = "cuda:0", [63, 127], [3, 2], []
        self.Q = self.V = self.R = []

    def apply_options(self, opts):
        self.applied = dict(opts)

    def release_graph(self):
        self.captured = None

    def capture(self):
        self.captured = self.options[5]

    def pair(self):
        self.log.append(("pair", self.options[5], self.options[4]))

    def replay(self):
        self.log.append(("graph", self.captured, self.options[4]))


@pytest.mark.parametrize("form", [0, 1])
def test_autotune_searches_the_options_of_the_current_form(form, tmp_path, monkeypatch):
    from shtns_b200 import batch as B
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "gpu")
    ticks = iter(range(100))
    monkeypatch.setattr(B, "_time", lambda fn, reps: float(next(ticks)))
    path = str(tmp_path / "tune.json")
    rec = B.autotune(FakeBatch(form), cache=path)
    keys = {k for t in rec["trials"] for k in t} - {"ms", "fft_pairs", "ckseg"}
    assert keys == (set() if form else {"order", "ctas_per_sm"})
    # the other form does not take this one's cached choice
    other = FakeBatch(1 - form)
    assert set(B.autotune(other, cache=path)["options"]) != set(rec["options"])
    assert B.autotune(FakeBatch(form), cache=path)["options"] == rec["options"]


@pytest.mark.parametrize("fast", [0, 1])
def test_bench_times_each_form_with_its_own_option(fast):
    import bench
    ub = FakeBatch(1)

    def timed(fn, steps):
        fn()
        what, form, _ = ub.log[-1]
        return 1.0 if form == fast else 2.0
    best, forms = bench.uneven_group_forms(ub, timed, 1, lambda b: {"form": b.options[5]})
    assert ub.log == [("pair", 1, 0), ("pair", 1, 1), ("graph", 1, 1), ("pair", 0, 0), ("pair", 0, 1), ("graph", 0, 1)]
    assert best == ("per_plan" if fast else "persistent")
    # the batch is left in the form that is reported, with that form's options
    assert ub.options[5] == fast and ub.captured == fast and ub.applied == {"form": fast}
    assert forms["per_plan"]["options"] == {"form": 1} and forms["persistent"]["options"] == {"form": 0}
