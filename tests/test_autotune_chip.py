"""The autotuner and cases that run on chip: the library's own plan is one of its candidates."""
import json
import os
from importlib import import_module

import numpy as np
import pytest


class _FakePkg:
    """A library whose batches run on chip; `win`: the nodes per CTA (None: not set) that is fastest."""
    ARITH_FAST, USED_CHIP = 1, 8
    OPT_THREADS, OPT_CTAS_PER_SM, OPT_NODES_PER_CTA, OPT_L1_LOADS, OPT_STAGED, OPT_ENGINE = range(1, 7)

    def __init__(self, win):
        pkg = self

        class Batch:
            def __init__(self, params, meshes):
                self.n, self.opt = len(params), {}

            def set_option(self, k, v):
                assert k != pkg.OPT_NODES_PER_CTA or v >= 64   # as in the library
                self.opt[k] = v

            def set_state(self, c, st):
                pass

            def run(self, steps, itc):
                win = self.opt.get(pkg.OPT_NODES_PER_CTA) == pkg.win and not self.opt[pkg.OPT_ENGINE]
                return None, np.full((self.n, 1), 10 ** 6 if win else 10), None, None

            def engines_used(self):
                return 2 if self.opt[pkg.OPT_ENGINE] else 8

            def close(self):
                pass

        self.win, self.Batch = win, Batch


@pytest.mark.parametrize("win", [None, 1024])
def test_the_library_s_plan_is_a_candidate(pkg, tmp_path, monkeypatch, win):
    at = import_module(pkg.__name__ + ".autotune")
    monkeypatch.setattr(at, "CACHE_DIR", str(tmp_path))
    items, _ = pkg.configs.cfg_batch(3, seed=5, sizes=(51,))
    old = tmp_path / f"{at._device_name(pkg)}-{at.signature(items)}.json"
    old.write_text(json.dumps({"best": {"threads": 256, "ctas_per_sm": 2, "nodes_per_cta": 8192, "staged": 0, "engine": 0}}))
    fake = _FakePkg(win)
    best = at.tune(fake, items, iters=20)   # not the choice cached for earlier kernels
    assert best["nodes_per_cta"] == (win or 0) and best["engine"] == 0
    new = [f for f in os.listdir(tmp_path) if f != old.name]
    with open(tmp_path / new[0]) as f:
        table = json.load(f)["table"]
    # one row per split, the plan's own first, and the graph engine
    assert [r["nodes_per_cta"] for r in table] == [0] + at.NODES + [4096]
    b = fake.Batch([None], [None])
    at.apply(b, fake, best)
    assert b.opt.get(fake.OPT_NODES_PER_CTA) == win
