"""lst_event_get_launch_shape: the shape that a launch of all the set's slots
takes, set or default, and a set shape is the one that is read."""
import pytest

from tracklooper_b200 import lst

pytestmark = pytest.mark.gpu

PER_EVENT = {"kCreateMD": 2, "kCreateLS": 4, "kCreateT3": 4, "kPixMid<3>": 2}  # blocks per SM, from 16 to 64


@pytest.mark.parametrize("slots", [1, 4, 5, 8, 9, 16, 17])
def test_shape_in_effect(slots):
    es = lst.ES(device=0)
    s = lst.EventSet(es, slots, 4096)
    try:
        shapes = s.launch_shapes()
        for name, (warps, per_sm) in shapes.items():
            assert warps == (8 if name in ("kCreateMD", "kMDDerived") else 4)
            assert per_sm == max(16, min(64, PER_EVENT.get(name, 0) * slots)), name
        for name, shape in shapes.items():  # what was read, set
            s.set_launch_shape(name, *shape)
        assert s.launch_shapes() == shapes
        s.set_launch_shape("kCreateLS", 2, 100)
        assert s.launch_shapes() == {**shapes, "kCreateLS": (2, 100)}
    finally:
        s.close()
        es.close()
