"""The line between the resident solve's two forms: a system just past one cluster's
bricks must not take longer an iteration than a larger one on the whole grid. Device
times of the profile, medians of 15; on the cluster the smaller took a fifth more.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_iteration_past_one_round_of_a_cluster():
    from test_gpu_form_lines import _median
    (a, na), (b, nb) = _median(48, "vcycle"), _median(56, "vcycle")  # 116 and 183 domain bricks
    assert na < nb
    print(a, b)
    assert a <= 1.05 * b, (a, b)
