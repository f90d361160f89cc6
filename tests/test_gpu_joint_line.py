"""Joints at a node on either side of the line between the two forms of their
evaluation (GPU): one launch up to two joints a slot, two launches above."""
import pytest

from test_gpu_joint_forms import test_a_node_with_many_joints as compare_with_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spokes", [2, 3])
def test_either_side_of_the_line(spokes):
    compare_with_the_oracle(spokes)
