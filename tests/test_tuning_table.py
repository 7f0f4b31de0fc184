"""The tuner's choice and the committed table, without a GPU."""
import json

import pytest

from duct_b200 import tune


class Recorder:
    def __init__(self):
        self.calls = []

    def set_pass_kernel(self, kernel, size_class=-1):
        self.calls.append(("pass", kernel, size_class))

    def set_rect_fold(self, on):
        self.calls.append(("rect", on))


def test_the_default_stays_unless_beaten_at_every_batch():
    d = {"default": 1.0}
    assert tune.choose({"4": {**d, "a": 0.5}, "64": {**d, "a": 1.1}}) == "default"
    assert tune.choose({"4": {**d, "a": 0.99}, "64": {**d, "a": 0.99}}) == "default"
    assert tune.choose({"4": {**d, "a": 0.9, "b": 0.8}, "64": {**d, "a": 0.9, "b": 0.95}}) == "b"
    assert tune.choose({"4": {**d, "a": 0.5}, "64": d}) == "default"      # refused the larger batch


@pytest.mark.parametrize("m,kernel,size_class", [(66, "default", 0), (67, "parity", 1), (130, "register", 1), (131, "default", 2)])
def test_apply_square(tmp_path, m, kernel, size_class):
    path = tmp_path / "t.json"
    path.write_text(json.dumps({"entries": [{"ny": m, "nz": m, "pass_kernel": kernel}]}))
    ctx = Recorder()
    assert tune.apply(ctx, m, m, str(path))["pass_kernel"] == kernel
    assert ctx.calls == [("pass", tune.FORMS[kernel], size_class)]
    assert tune.apply(ctx, m + 1, m, str(path)) is None


@pytest.mark.parametrize("form,value", [("default", -1), ("full", 0), ("fold", 1), ("fold-one-launch", 2), (1, 1)])
def test_apply_rect(tmp_path, form, value):
    path = tmp_path / "t.json"
    path.write_text(json.dumps({"entries": [{"ny": 33, "nz": 49, "rect_fold": form}]}))
    ctx = Recorder()
    tune.apply(ctx, 33, 49, str(path))
    assert ctx.calls == [("rect", value)]


def test_committed_table_follows_its_own_timings():
    """Every entry is what choose() makes of the timings beside it."""
    with open(tune.TABLE) as f:
        entries = json.load(f)["entries"]
    assert entries
    for e in entries:
        assert e.get("pass_kernel", e.get("rect_fold")) == tune.choose(e["ms_per_batch"])
