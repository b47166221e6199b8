"""Device memory of a network's first gradient: activations, gelu' and gradients
of every layer (3 x 512 bytes a row and layer) and one set of weight-gradient
partials per 512 rows and layer, but not the 64 sets of the per-tile kernels."""
import numpy as np
import pytest

import gpueularsolver2d_gb300 as e2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,nhidden", [(2048, 3), (4096, 8), (16384, 5)])
def test_first_gradient(lib, batch, nhidden):
    import torch
    x, t = np.zeros((batch, 32), np.float32), np.zeros((batch, 4), np.float32)
    used = []
    for _ in range(2):  # the first loads the kernels
        net = e2d.MLP(nhidden=nhidden, batch=batch)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        net.gradient(x, t)
        used.append(free - torch.cuda.mem_get_info()[0])
        net.close()
    need = nhidden * (3 * 512 * batch + batch // 512 * 256 * 257 * 4) + batch * 512
    # allocations come in pieces of 2 MB: one more for each of three buffers a layer and some others
    assert used[1] < need + (2 * nhidden + 8) * (2 << 20), (used[1], need)
