"""Cells of a 4x4x2 sub-block that lie outside the grid take no evidence and leave their neighbours'
alone (csrc/evidence.cu, Cols): grid sizes of every remainder, rays along the axes through the last
cells included, to the tolerance of the other evidence checks."""
import numpy as np
import pytest

from test_gpu_evidence_batches import check, scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,Gz", [(13, 5), (14, 6), (15, 7), (16, 9), (1, 1), (3, 2)])
def test_cells_outside_the_grid(G, Gz):
    res = 0.2
    axes = np.eye(3, dtype=np.float32) * np.float32(0.45 * G * res)
    pts = np.concatenate([scan(300, G, 0.6 * G * res), axes, -axes]).astype(np.float32)
    check(G, Gz, res, 0.5, 0.1, pts)
    check(G, Gz, res, 0.5, 0.1, pts, tuning=(2, 512))
