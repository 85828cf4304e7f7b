"""Which meshes have their sign spread: closed ones, with enough node-triangle
pairs, no triangle thinner and no coordinate larger than the limits."""
import numpy as np
import pytest

from sdf_gate import sliver, spreads, tilted_box

NODES = 65536


def _sphere():
    from mpm_b200 import scenes
    return scenes.uv_sphere(9.0, (300.0, 310.0, 290.0), 40, 24)


def test_closed_and_open(mpm):
    ball = _sphere()
    assert spreads(mpm, ball, NODES)
    assert not spreads(mpm, ball[:-1], NODES)
    assert not spreads(mpm, ball[:700], NODES)  # fewer than 5e7 pairs
    turned = ball.copy()
    turned[5] = turned[5][[0, 1, 2, 6, 7, 8, 3, 4, 5]]
    assert not spreads(mpm, turned, NODES)


@pytest.mark.parametrize("width, inside", [(90.0, True), (88.0, True), (85.0, False), (61.0, False)])
def test_slivers(mpm, width, inside):
    tris = np.concatenate([tilted_box((517.0, width, width), (0.01, 0.02), (20.0, 20.0, 20.0)), _sphere()])
    assert (sliver(tris) < 2e4) == inside
    assert spreads(mpm, tris, NODES) == inside


@pytest.mark.parametrize("top, inside", [(1024.0, True), (1024.0625, False)])
def test_coordinates(mpm, top, inside):
    ball = _sphere()
    ball = (ball.reshape(-1, 3) + (np.float32(top) - ball.reshape(-1, 3)[:, 2].max()) * np.array([0, 0, 1], np.float32)).reshape(-1, 9)
    assert ball.max() == top
    assert spreads(mpm, ball, NODES) == inside
    assert spreads(mpm, ball * np.float32(-1.0), NODES) == inside
    ball[3, 4] = np.nan
    assert not spreads(mpm, ball, NODES)
