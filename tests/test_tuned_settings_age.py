"""Tuned settings timed on earlier kernels (tuner 3: conditional refit nodes, a
thread an atom for every list, halfword lists) are not taken from the cache."""
import json

from naivedynamics import dynamics as dyn


class _Ctx:
    handle = None

    def device_name(self):
        return "GB300-test"

    def check(self, st, what):
        raise RuntimeError("timed anew")


def test_settings_of_earlier_kernels_are_timed_anew(nd, tmp_path, monkeypatch):
    import numpy as np
    import pytest
    p = nd.md_params(cutoff=2.5, skin=0.3, box_hi=(17, 17, 17))
    path = tmp_path / "autotune.json"
    monkeypatch.setenv("ND_AUTOTUNE_CACHE", str(path))
    x = np.zeros((8, 3))
    hit = {"params": {k: getattr(p, k) for k in dyn.TUNED_FIELDS}, "seconds_per_step": 1e-5}
    now = json.loads(dyn._tune_key(_Ctx(), p, 8, None, False, False))
    for tuner, cached in ((3, False), (dyn.TUNER_VERSION, True)):
        path.write_text(json.dumps({json.dumps(dict(now, tuner=tuner), sort_keys=True): hit}))
        if cached:
            assert dyn.autotune(p, x, x, ctx=_Ctx())[1] == 1e-5
        else:
            with pytest.raises(RuntimeError):
                dyn.autotune(p, x, x, ctx=_Ctx())
