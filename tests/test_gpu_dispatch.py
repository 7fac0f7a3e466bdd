"""Edges of the sizes at which the device path changes kernels or splits, against the oracle."""
import numpy as np
import pytest
import torch

from fourierd3_b200 import neighbour_list
from oracle.neighbours import neighbour_list_cells

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_atoms", [1, 33, 250, 264, 2300])
def test_neighbours_of_bins_from_one_to_hundreds_of_atoms(cuda_device, n_atoms):
    # 2 x 2 x 2 bins of 6.05 A: segments of the counting sort below, at and far beyond one warp
    rng = np.random.default_rng(n_atoms)
    cell = np.diag([12.1, 12.1, 12.1])
    pos = rng.random((n_atoms, 3)) @ cell
    i, j, s = neighbour_list(torch.tensor(pos, device=cuda_device), cell, 6.0)
    got = torch.cat((i[:, None], j[:, None], s.to(torch.int64)), 1).cpu().numpy()
    ri, rj, rs = neighbour_list_cells(pos, cell, 6.0)
    want = np.concatenate((ri[:, None], rj[:, None], rs), 1)
    assert np.all(np.diff(got[:, 0]) >= 0)
    assert np.array_equal(got[np.lexsort(got.T[::-1])], want[np.lexsort(want.T[::-1])])
