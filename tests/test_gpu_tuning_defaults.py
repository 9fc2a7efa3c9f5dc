"""set_tuning's defaults are the choices a tracer starts with: naming one knob
leaves the others as they were."""
import pytest

from pfx_b200 import synth
from pfx_b200.trace import Trace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("knob", [{}, {"graphs": False}, {"short_stack": 8}, {"sort_shading": True}])
def test_other_knobs_stay(gpu, knob):
    w = synth.small("plain_512", (16, 16), "sobol")
    trace = Trace(w.scene, w.settings, w.width, w.height)
    start = trace.tuning()
    trace.set_tuning(**knob)
    assert trace.tuning() == {**start, **knob}
