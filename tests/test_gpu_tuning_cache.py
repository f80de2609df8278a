"""Tuning decisions kept on disk count for the kernels that they were measured with."""
import json

import numpy as np
import pytest

from novaphy_gb300 import capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernels", [None, "0" * 16, "this"])
def test_decision_of_other_kernels(tmp_path, monkeypatch, kernels):
    cache = tmp_path / "autotune.jsonl"
    monkeypatch.setenv("PBF_AUTOTUNE_CACHE", str(cache))
    w = workloads.dam_break((10, 9, 8), 0.025, (1.0, 1.0, 1.0), dt=1.0 / 120.0, seed=1)
    sc = capi.Scene(capi.default_settings(**w.settings), w.x, w.v, mass=w.mass)
    sc.set_gravity(w.gravity)

    def tuned(steps):
        b = capi.Batch()
        b.set_autotune(True)
        for _ in range(steps):
            b.step([sc], [np.float32(w.dt)])
        out = b.tuning()
        b.close()
        return out

    tuned(6)
    line = json.loads(cache.read_text().splitlines()[0])
    line.update(block=256, persistent=1)
    if kernels is None:
        line.pop("kernels", None)
    elif kernels != "this":
        line["kernels"] = kernels
    cache.write_text(json.dumps(line) + "\n")
    # The first trial, unless the kept decision counts.
    assert tuned(1) == ((256, 1) if kernels == "this" else (128, 0))
    sc.close()
