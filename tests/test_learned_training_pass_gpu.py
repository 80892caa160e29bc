"""The learned estimator's training passes (all layers in one launch each) against a chain of single
convolution layers through the public entries, around the window sizes of the fused kernel (200 exact
rows per one-tile window, 456 per two-tile window) and the 128-row tiles of the weight gradients: the
output equals the chain's bit for bit (same products in the same order), the gradients to the
rounding of their FP32 sums."""
import ctypes

import numpy as np
import pytest

from pusch_b200 import learned
from pusch_b200 import tclayout as tl

pytestmark = pytest.mark.gpu


def chain(ctx, params, x, dy, valid, rows):
    """Outputs and gradients layer by layer (device tensors in the library's layout)."""
    import torch
    lib, st = ctx.lib, torch.cuda.current_stream().cuda_stream
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws, o = [], 0
    for cin, cout in learned.LAYERS:
        w = params[o:o + 5 * cin * cout].reshape(5, cin, cout).transpose(2, 1, 0)     # [co][ci][t]
        b = torch.from_numpy(params[o + 5 * cin * cout:o + 5 * cin * cout + cout].copy()).cuda()
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda()
        ws.append((dev(tl.pack_weights(w)), dev(tl.pack_weights_t(w)), b))
        o += 5 * cin * cout + cout
    new = lambda c: torch.zeros((c // 8, rows, 8), dtype=torch.int16, device="cuda")
    ins, outs, a, skip = [], [], x, None
    for i, (cin, cout) in enumerate(learned.LAYERS):
        y = new(cout)
        second = 0 < i < 13 and i % 2 == 0
        ctx.check(lib.pg_conv1d_forward_device(ctx.handle, cin, cout, a.data_ptr(), ws[i][0].data_ptr(), ws[i][2].data_ptr(),
                                               skip.data_ptr() if second else None, y.data_ptr(), valid.data_ptr(), rows,
                                               int(i < 13), err.data_ptr(), st))
        ins.append(a)
        outs.append(y)
        a = y
        if i % 2 == 0:
            skip = y
    grads, g, passed = [None] * 14, dy, None
    for i in reversed(range(14)):
        cin, cout = learned.LAYERS[i]
        dw = torch.zeros(5 * cin * cout, dtype=torch.float32, device="cuda")
        db = torch.zeros(cout, dtype=torch.float32, device="cuda")
        ctx.check(lib.pg_conv1d_backward_weights_device(ctx.handle, cin, cout, ins[i].data_ptr(), g.data_ptr(), rows,
                                                        dw.data_ptr(), db.data_ptr(), err.data_ptr(), st))
        grads[i] = torch.cat([dw, db])
        if i == 0:
            break
        dx = new(cin)
        first = i % 2 == 1 and i < 13            # first layer of a block: the gradient that passed by it
        ctx.check(lib.pg_conv1d_backward_data_device(ctx.handle, cin, cout, g.data_ptr(), ws[i][1].data_ptr(),
                                                     passed.data_ptr() if first else None, outs[i - 1].data_ptr(),
                                                     dx.data_ptr(), valid.data_ptr(), rows, err.data_ptr(), st))
        g = dx
        if i % 2 == 1:
            passed = dx
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return outs[-1].cpu().numpy(), torch.cat(grads).cpu().numpy()


@pytest.mark.parametrize("rows", [1, 127, 200, 201, 456, 457, 1025, 70001])
def test_training_pass_equals_layer_chain(ctx, rows):
    import torch
    rng = np.random.default_rng(rows)
    valid = np.ones(rows, np.uint8)
    valid[rng.integers(0, rows, rows // 40)] = 0
    params = learned.init_params(3)
    params[-16 - 5 * 64 * 16:] *= 50.0
    bf = lambda a: tl.to_chunked(tl.bf16_round(a.astype(np.float32))).view(np.int16)
    x = torch.from_numpy(bf(rng.standard_normal((rows, 16)) * valid[:, None])).cuda()
    dy = torch.from_numpy(bf(rng.standard_normal((rows, 16)) * valid[:, None])).cuda()
    v = torch.from_numpy(valid).cuda()
    net = learned.LearnedEstimator(ctx, rows + 50, params=params)
    y = torch.zeros((2, rows, 8), dtype=torch.int16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    net.forward(x.data_ptr(), v.data_ptr(), rows, y.data_ptr(), st)
    net.backward(dy.data_ptr(), rows, st)
    g = net.grads()
    net.status()
    net.close()
    want_y, want_g = chain(ctx, params, x, dy, v, rows)
    assert np.array_equal(y.cpu().numpy(), want_y)
    # Sums of at most 70,001 products and partial sums in FP32 in another order.
    assert np.linalg.norm(g - want_g) <= 2e-6 * np.linalg.norm(want_g)
