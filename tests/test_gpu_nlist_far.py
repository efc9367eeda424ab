"""The list of particles tens and hundreds of boxes away: an FP32 coordinate there is
coarse, but the pair set of those coordinates is still exact. Particles whose
cell differs when it is taken from the coordinate itself in FP32 (whose sum with
half a box rounds across a cell face), each with a partner just inside the list
radius on the far side of that face, among a random fluid."""
import numpy as np
import pytest

from helpers import f32, kdtree_reference_pairs
from sucrose_gb300 import GpuSystem

pytestmark = pytest.mark.gpu

SIDE, SHORT, CUTOFF, SKIN = 73.05, 10.9, 1.8, 0.2
CELLS = 36   # floor(73.05 / 2.0002); CELLS * (1 / SIDE) rounds to 6e-8 of itself in FP32
# the search's own slack: half the FP64 band, 1e-4 of the radius squared, and some 1e-5
# of radius and 1e-6 of side besides; pairs further than this from the face test it
SLACK = 3e-4


def across_a_face(boxes):
    """FP32 coordinates near the cell faces, `boxes` boxes out, whose FP32 cell and
    whose image's cell differ; (coordinate, image, +1 or -1: the image's side)."""
    L, out = np.float32(SIDE), []
    for face in range(1, CELLS):
        at = face * SIDE / CELLS - SIDE / 2
        x0 = np.float32(boxes * SIDE + at)
        x = x0 + np.arange(-6, 7) * np.spacing(x0)
        image = x.astype(np.float64) - boxes * SIDE
        cell = np.floor((x + np.float32(0.5) * L) * (np.float32(CELLS) * np.float32(1.0 / SIDE)))
        cell = cell.astype(np.int64) % CELLS
        side = np.where(image >= at, 1, -1)
        wrong = ((cell == face) != (side == 1)) & (np.abs(image - at) > SLACK)
        out += list(zip(x[wrong], image[wrong], side[wrong]))
    return out


@pytest.mark.parametrize("boxes", [range(60, 100), range(-100, -60), range(300, 400)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_pairs_across_cell_faces(lib, axis, boxes):
    rng = np.random.default_rng(abs(boxes[0]))
    far = [f for b in boxes for f in across_a_face(b)]
    far = [far[k] for k in rng.permutation(len(far))]
    assert len(far) >= 20
    box = np.full(3, SHORT)
    box[axis] = SIDE
    r = rng.uniform(-0.5, 0.5, (4000, 3)) * box
    for k in range(100):
        x, image, side = far[k % len(far)]
        r[2 * k + 1] = r[2 * k]
        r[2 * k, axis] = x
        r[2 * k + 1, axis] = image + side * (CUTOFF + SKIN) * (1 - 3e-6)
    r = f32(r[rng.permutation(len(r))])
    g = GpuSystem(len(r), box)
    g.upload(r=r)
    g.init_nlist(SKIN, CUTOFF)
    want, got = kdtree_reference_pairs(r, box, CUTOFF, SKIN), g.pairs()
    assert len(want[0]) == len(got[0])
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
