"""Weights that are infinite (a diverged training run) act in the training passes as in a chain of single layers:
infinities and NaN in the same places, through the layers, the ReLU and the gradients."""
import numpy as np
import pytest

from pusch_b200 import learned
from pusch_b200 import tclayout as tl
from test_learned_training_pass_gpu import chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer,tap,value", [(0, 3, np.inf), (0, 4, -np.inf), (5, 2, np.inf), (5, 4, np.inf),
                                            (6, 0, -np.inf), (13, 3, np.inf), (13, 1, np.inf)])
def test_infinite_weight(ctx, layer, tap, value):
    import torch
    rows = 457
    rng = np.random.default_rng(layer)
    params = learned.init_params(3)
    params[-16 - 5 * 64 * 16:] *= 50.0
    cin, cout = learned.LAYERS[layer]
    at = sum(5 * a * b + b for a, b in learned.LAYERS[:layer])
    params[at + (tap * cin + 3) * cout + 7] = value  # input channel 3, output channel 7
    valid = np.ones(rows, np.uint8)
    valid[rng.integers(0, rows, rows // 40)] = 0
    bf = lambda a: torch.from_numpy(tl.to_chunked(tl.bf16_round(a.astype(np.float32))).view(np.int16)).cuda()
    x, dy = (bf(rng.standard_normal((rows, 16)) * valid[:, None]) for _ in range(2))
    v = torch.from_numpy(valid).cuda()
    net = learned.LearnedEstimator(ctx, rows, params=params)
    y = torch.zeros((2, rows, 8), dtype=torch.int16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    net.forward(x.data_ptr(), v.data_ptr(), rows, y.data_ptr(), st)
    net.backward(dy.data_ptr(), rows, st)
    g = net.grads()
    net.status()
    net.close()
    want_y, want_g = chain(ctx, params, x, dy, v, rows)
    f32 = lambda b: (b.view(np.uint16).astype(np.uint32) << 16).view(np.float32)
    got, want = f32(y.cpu().numpy()), f32(want_y)
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.isnan(g), np.isnan(want_g)) and np.array_equal(np.isinf(g), np.isinf(want_g))
    ok = np.isfinite(want_g)
    assert np.linalg.norm(g[ok] - want_g[ok]) <= 2e-6 * np.linalg.norm(want_g[ok])
