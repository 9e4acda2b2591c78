"""Weight gradients by kernel rows (k_conv3_wgrad_row in csrc/dn.cu): image
sizes whose levels take it (whole groups of 32 pixels), mix it with the general
kernel (12 x 12), and whose rows are shorter than a group.  Tolerances as the
batched gradients' against the same oracle (tests/test_gpu_denoiser_tcb.py)."""
import numpy as np
import pytest

import dn_oracle as D
from test_gpu_denoiser_tcb import _net, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,nb,seed", [(64, 64, 3, 21), (96, 96, 2, 22), (128, 64, 2, 23), (64, 128, 1, 24)])
def test_weight_gradients_against_oracle(h, w, nb, seed):
    import torch
    net, p, x, t, xd, td = _net(h, w, nb, seed)
    net.set_batch_tensor_cores(True)
    out = torch.empty_like(xd)
    loss, g = net.gradients(xd.data_ptr(), td.data_ptr(), nb, out.data_ptr())
    loss_o, g_o, y_o = D.loss_and_grads(p.astype(np.float64), x, t, tf32_operands=True)
    convs, ow, ob, n = D.layout()
    assert abs(loss - loss_o) <= 1e-3 * abs(loss_o)
    for wo, bo, ci, co in convs:
        assert rel(g[wo:wo + ci * co * 9], g_o[wo:wo + ci * co * 9]) <= 2e-2, (ci, co)
        assert rel(g[bo:bo + co], g_o[bo:bo + co]) <= 2e-2, (ci, co)
    assert net.tensor_errors() == 0
