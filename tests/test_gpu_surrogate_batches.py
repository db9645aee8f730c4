"""The training gradient at batch sizes around a block's turn of 128 samples,
and with weights that are not 16-byte aligned, against FP64 autograd on the
same BF16 weights."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(net, x, y):
    import torch
    from alya_sma_b200 import surrogate as S
    w = torch.as_tensor(net.params_bf16(), dtype=torch.float64, device="cuda").requires_grad_()
    st = torch.as_tensor(net.stats_array(), device="cuda")
    z = torch.nn.functional.pad((x.double() - st[:14]) / st[14:28], (0, 2))
    for k, (i, o) in enumerate(((16, 64), (64, 64), (64, 64), (64, 64), (64, 16)), 1):
        a, b = S.OFF["W%d" % k], S.OFF["b%d" % k]
        z = z @ w[a:a + i * o].reshape(o, i).T + w[b:b + o]
        if k < 5:
            z = z * torch.sigmoid(z)
    ((z[:, :13] - (y.double() - st[28:41]) / st[41:54]) ** 2).mean().backward()
    return w.grad


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 148 * 128 + 5])
@pytest.mark.parametrize("aligned", [True, False])
def test_gradient_of_ragged_batches(n, aligned):
    import torch
    from alya_sma_b200 import _check, lib
    from alya_sma_b200 import problem as P
    from alya_sma_b200 import surrogate as S
    x, y = S.generate(P.nitinol_props(**P.NITI), P.NITI_E_MART, 256, nstep=256, seed=9, inactive_only=True)
    net = S.Surrogate(seed=2)
    net.fit_stats(x, y)
    net.w[S.OFF["b2"]:S.OFF["b2"] + 64] = 0.1                # some biases that are not zero
    net.pack()
    x, y = x[:n].contiguous(), y[:n].contiguous()
    wb = torch.zeros(S.NPARAM + 8, dtype=torch.int16, device="cuda")
    off = 0 if aligned else 1
    wb[off:off + S.NPARAM] = net.wb
    grad = torch.zeros(S.NPARAM, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    _check(lib().sma_sur_train_step(C.c_void_p(wb.data_ptr() + 2 * off), C.c_void_p(net.w.data_ptr()),
                                    C.c_void_p(net.stats.data_ptr()), C.c_int64(n), C.c_void_p(x.data_ptr()),
                                    C.c_void_p(y.data_ptr()), C.c_void_p(grad.data_ptr()),
                                    C.c_void_p(loss.data_ptr()), C.c_void_p(net._s)))
    torch.cuda.synchronize()
    ref = _reference(net, x, y)
    # activations and deltas carry BF16 rounding (2^-9) through five layers
    # forward and back; few samples average little of it out
    assert float((grad.double() - ref).norm() / ref.norm()) < 10 * 2.0 ** -9
    assert np.isfinite(float(loss))
    pad = grad[:1024].reshape(64, 16)[:, 14:]
    assert float(pad.abs().max()) == 0.0                     # padding inputs get no gradient
