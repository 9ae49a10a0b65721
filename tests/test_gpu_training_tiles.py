"""The training gradient at the edges of its tiles: sample counts around a warp's 16 and a block's 64,
and more tiles than blocks, for both networks, against the float64 restatement. Operands are BF16
(8-bit significands, four roundings in a row from input to weight gradient: 4 * 2^-9 of each product,
at most about 1% of a block's norm with the approximate tanh), so a parameter block may be 3% off."""
import numpy as np
import pytest

from itsu import capi, prefilter

pytestmark = pytest.mark.gpu
HIDDEN = {"pair": 64, "gate": 16}


@pytest.mark.parametrize("net", ["pair", "gate"])
@pytest.mark.parametrize("n", [1, 15, 17, 63, 64, 65, 130, 296 * 64 + 33])
def test_gradient_at_tile_edges(net, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    ctx = capi.Context()
    try:
        if net == "pair":
            model = capi.prefilter_load(prefilter.CHECKPOINTS["pbpb"])
            ctx.prefilter_set_model(model)
        else:
            model = capi.gate_load(prefilter.GATE_CHECKPOINTS["pbpb"])
            ctx.gate_set_model(model)
        mean, inv_std = np.array(list(model.mean)), np.array(list(model.inv_std))
        features = (mean + rng.normal(0.0, 1.0, (n, 8)) / inv_std).astype(np.float32)
        labels = (rng.uniform(0.0, 1.0, n) < 0.3).astype(np.uint8)
        on_device = torch.from_numpy(features).cuda(), torch.from_numpy(labels).cuda()
        gradient = ctx.prefilter_gradient if net == "pair" else ctx.gate_gradient
        got, loss = gradient(on_device[0].data_ptr(), on_device[1].data_ptr(), n, 1.5)
        want, want_loss = prefilter.mlp_gradient(model.arrays(), features, labels, 1.5, **({} if net == "pair" else {"act": "relu"}))
    finally:
        ctx.close()
    assert abs(loss - want_loss) <= 1e-2 * max(1.0, abs(want_loss))
    h = HIDDEN[net]
    bounds = np.cumsum([0, 8 * h, h, h * h, h, h, 1])
    for a, b in zip(bounds[:-1], bounds[1:]):
        assert np.linalg.norm(got[a:b] - want[a:b]) <= 0.03 * np.linalg.norm(want[a:b]) + 1e-6, (a, b)
