"""A batch's settings are those that run: its queue has a largest CTA count per SM (fewer on the flux pass than on the
colour passes, which peso other than 1 takes), lsh_batch_set_tune keeps no more than that, and the autotuner times each
launch once."""
import ctypes

import pytest

from landslidehysea_gb300 import scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("peso", [1.0, 0.9])
def test_settings_are_what_runs(gpu_lib, peso):
    from landslidehysea_gb300.solver import Batch, Tune
    sc = scenarios.shelf(n=24, dx=200.0)
    sc.params.peso = peso
    ctas = {}

    def tune(b):
        t = Tune()
        assert gpu_lib.lsh_batch_get_tune(b._b, ctypes.byref(t)) == 0
        return t.ctas_per_sm

    with Batch([sc.params]) as b:
        b.set_state(0, sc.state)
        ctas["default"] = tune(b)
        b.set_tune(ctas_per_sm=20)  # taken, as any number up to 20
        ctas["20"] = most = tune(b)
        b.set_tune(ctas_per_sm=5)
        assert tune(b) == 5
        best = b.autotune(trial_steps=2)
        b.synchronize()
        steps = b.time(0)[2]
    assert most == (12 if peso == 1.0 else 20)
    assert ctas["default"] <= most and best["ctas_per_sm"] <= most
    tried = sum(c <= most for c in (8, 12, 16, 20)) * 4  # four fetch sizes each
    assert steps == tried * 3  # one step to warm up and two timed
