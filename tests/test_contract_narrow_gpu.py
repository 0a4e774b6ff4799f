"""The contraction in tiles of 128 columns (results no wider): one column, the edges of the epilogue's 64-column
groups, several tiles of rows, one and two sources, operands in blocks of 64 rows. Bounds as for the wider tiles."""

import pytest

import test_contract_tiles_gpu as tiles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_i,n_j,n_k,n_src", [(1, 1, 1, 1), (77, 77, 77, 1), (128, 63, 64, 2), (129, 65, 130, 1), (300, 128, 200, 1)])
@pytest.mark.parametrize("running", [False, True])
def test_contract(cuda_device, n_i, n_j, n_k, n_src, running):
    tiles.test_contract(cuda_device, n_i, n_j, n_k, n_src, running)


@pytest.mark.parametrize("n_i,n_j,n_src", [(128, 128, 1), (97, 104, 2), (203, 120, 1), (65, 72, 1)])
def test_contract_in_blocks_of_64_rows(cuda_device, n_i, n_j, n_src):
    tiles.test_contract_in_blocks_of_64_rows(cuda_device, n_i, n_j, n_src)
