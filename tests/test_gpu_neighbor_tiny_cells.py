"""Cells whose vectors are far shorter than the cutoff: more images than a 32-bit walk holds are
refused, whichever direction they come from."""
import pytest
import torch

from matpl_gb300 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("edges", [(4e-9, 30.0, 30.0), (30.0, 4e-9, 30.0), (30.0, 30.0, 4e-9), (4e-9, 4e-9, 4e-9),
                                   (0.003, 0.003, 0.003), (1e-4, 1e-4, 30.0)])
def test_too_many_images_are_refused(edges):
    lat = torch.diag(torch.tensor(edges, dtype=torch.float64, device=DEV))
    frac = torch.tensor([[0.1, 0.2, 0.3], [0.6, 0.7, 0.8]], dtype=torch.float64, device=DEV)
    with pytest.raises(_lib.MatplError, match="images"):
        ops.find_neighbore(torch.zeros(2, dtype=torch.int32, device=DEV), frac, lat, 1, 100, 6.0, 6.0)
