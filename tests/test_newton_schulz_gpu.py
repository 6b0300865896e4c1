"""The one-launch Newton-Schulz iteration issues the arithmetic of the separate products: the same bits."""
import pytest
import torch

from chaoscontrol_b200.ops import _lib
from chaoscontrol_b200.optim import muon as M

pytestmark = pytest.mark.gpu


# one, two, four and eight tiles; ragged rows, columns and contraction (tall and wide); several clusters to an SM group
@pytest.mark.parametrize("G,r,c", [(1, 8, 8), (3, 64, 128), (2, 72, 200), (1, 136, 128), (5, 200, 72), (16, 256, 256),
                                   (3, 256, 504), (4, 512, 256), (70, 256, 256), (1, 128, 1024), (1, 1024, 120)])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_one_launch_matches_separate_products(G, r, c, steps):
    g = torch.Generator(device="cuda").manual_seed(G + r + c)
    X = torch.randn(G, r, c, generator=g, device="cuda")
    X = (X / X.norm(dim=(1, 2), keepdim=True)).bfloat16()
    n0 = _lib.launch_count()
    got = M._ns_kernels(X.clone(), steps)
    assert _lib.launch_count() - n0 == 1
    k = min(r, c)
    A = torch.empty(2, G, k, k, dtype=torch.bfloat16, device="cuda")
    want = M._ns_products(X.clone(), torch.empty_like(X), A[0], A[1], steps)
    _lib.assert_ok()
    assert torch.equal(got, want)


def test_larger_matrices_take_the_separate_products():
    X = torch.randn(1, 512, 512, device="cuda")
    X = (X / X.norm()).bfloat16()
    n0 = _lib.launch_count()
    M._ns_kernels(X, 5)
    assert _lib.launch_count() - n0 == 15
