"""The benchmark's choice of attention launches that it times, and what they hold."""
import pytest

import bench


@pytest.mark.parametrize("layers,launches", [(61, 1), (61, 7), (61, 13), (27, 2), (4, 4), (61, 21), (56, 7)])
def test_the_timed_launches_are_every_group_of_a_step(layers, launches):
    """As the library cuts a step: equal groups, the last one what is left.  Over the steps every launch of a step is timed equally
    often, so the layers of the timed launches come to those of whole steps."""
    stride = bench.event_stride(launches)
    assert stride >= bench.MIN_EVENT_STRIDE
    assert sorted(k * stride % launches for k in range(launches)) == list(range(launches))
    assert bench.timed_layers(layers, launches, stride, 3 * launches) == 3 * layers
