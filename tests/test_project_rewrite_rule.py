"""When the feature gather rewrites a map channels-last first: sizes where
both ways were timed, and the rule's edges (no GPU)."""
import pytest


@pytest.mark.parametrize("n,C,edge,per_pixel,want", [
    (4, 5, 512, 5.0, False), (4, 6, 512, 2.0, False), (4, 6, 512, 3.0, True), (4, 8, 512, 0.9, False),
    (4, 8, 512, 1.0, True), (4, 12, 512, 0.6, False), (4, 12, 512, 1.0, True), (4, 16, 512, 0.45, False),
    (4, 16, 512, 0.5, True), (4, 32, 512, 0.25, False), (4, 32, 512, 0.45, True), (4, 68, 512, 0.25, False),
    (4, 68, 512, 0.5, True),
    (4, 32, 512, 3.0, True),                                                    # a chunk of 16384 rays
    (1, 16, 512, 0.99, False), (1, 16, 512, 1.0, True), (1, 32, 128, 5.0, False), (4, 32, 64, 3.0, False)])
def test_rule(n, C, edge, per_pixel, want):
    from sailor_gb300 import views
    assert views._rewrites(n, C, edge * edge, int(edge * edge * per_pixel)) == want
