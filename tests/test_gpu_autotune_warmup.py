"""What the autotuner times holds no graph capture (85 us beside trials of some 200): the substeps it takes
before each of its 12 timed trials are of all the kinds that the trial has, a call's first, middle and
last, which are graphs of their own."""
import pytest

from conftest import cuda_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

import crmpm_b200 as cb  # noqa: E402
from crmpm_b200 import scenes  # noqa: E402


@pytest.mark.parametrize("trial", [1, 2, 3, 8])
def test_every_graph_of_a_trial_is_captured_before_it(trial):
    g = cb.DeviceScene(scenes.cube_drop())

    def launches(fn):
        before = cb.kernel_launch_count()
        fn()
        return cb.kernel_launch_count() - before

    kinds = [launches(lambda: g.step(n)) for n in (1, 2, 3, 4)]  # a call's substeps, by its length
    middle = kinds[3] - kinds[2]
    timed = kinds[trial - 1] if trial <= 3 else kinds[2] + (trial - 3) * middle
    warm = kinds[min(trial, 3) - 1]
    states = 1 + 12 * 2 + 1  # the state saved, loaded before the substeps and the trial, and at the end
    assert launches(lambda: g.solver.autotune(trial)) == states + 12 * (warm + timed)
