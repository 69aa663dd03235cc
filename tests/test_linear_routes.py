"""Where a linear of a step may take the tensor-core form: the room for normalised rows and the shape of gated results. No GPU needed."""
from types import SimpleNamespace

import pytest
import torch


def test_product_only_where_its_rows_fit():
    from ironpangu_b200.runtime.plan_engine import PlanEngine

    takes = lambda width, normed, units: PlanEngine._takes_product(SimpleNamespace(_norm_rows=torch.empty(8, 64)), width, normed, units)
    assert takes(64, True, 0) and takes(8, True, 16) and takes(4096, False, 0)
    assert not takes(72, True, 0)                  # wider than the rows that are kept
    assert not takes(64, True, 12) and not takes(64, False, 4)


def test_room_of_another_shape_is_refused_before_anything_runs():
    from ironpangu_b200.ops import decode as K

    x, w, gain = (torch.zeros(*s, dtype=torch.bfloat16) for s in ((3, 128), (16, 128), (128,)))
    with pytest.raises(AssertionError):
        K.linear_product(x, w, torch.zeros(3, 16, dtype=torch.bfloat16), norm_w=gain, norm_out=torch.zeros(8, 64, dtype=torch.bfloat16)[:3, :128])
