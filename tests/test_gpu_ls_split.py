"""The Gram matrix's last wave split along K (k_gram_dmma, k_gram_sum in fp_ls.cu):
a closed body by least squares against the oracle, as the tests of test_gpu_ls.py."""
import numpy as np
import pytest

from test_gpu_ls import _check, freestream

pytestmark = pytest.mark.gpu


# 480 panels: 15 slices of K, none split; 512: two pieces of 8; 1,100: 45 tiles, 3 pieces
# of 12, 12 and 11 slices; 2,200: 171 tiles, the last 23 in 6 pieces
@pytest.mark.parametrize("nx,nt", [(30, 16), (32, 16), (44, 25), (55, 40)])
def test_split_tiles(fp, O, nx, nt):
    m = fp.meshes.prolate_ellipsoid(4.0, 0.5, nx, nt, tail=1.0)
    body = fp.RigidWakeBody(m, watertight=True)
    U = np.tile(freestream(5.0), (m.npanels, 1))
    fp.solve(body, U, np.zeros((0, 3)), np.zeros((0, 3)))
    _check(fp, O, body, U, np.zeros((0, 3)), [(0, 0.0)], body.strength)
