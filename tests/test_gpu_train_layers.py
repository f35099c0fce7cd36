"""The proposal network's layer kernels at the edges of their tiles: 16-row tiles, stages of 1, 4,
16 and 64 samples, one partial per CTA, against the float64 oracle with the same BF16 points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 15, 17, 64, 65, 153, 161])
def test_gradient_at_tile_edges(dic, n):
    torch = pytest.importorskip("torch")
    from fasticgn_gb300.proposal import ProposalNet, init_params
    from oracle import cnn_oracle as O
    rng = np.random.default_rng(n)
    params = init_params(3) + rng.normal(0, 0.02, O.PARAM_COUNT).astype(np.float32)   # biases too
    x = rng.normal(0, 1, (n, 31, 31, 2)).astype(np.float32)
    t = rng.normal(0, 1, (n, 6)).astype(np.float32) * np.array([2, 2, .01, .01, .01, .01], np.float32)
    want_loss, want, want_out = O.loss_and_grad(params, O.bf16(x), t)
    net = ProposalNet(0, params)
    flat = torch.from_numpy(x).to(torch.bfloat16).reshape(-1).cuda()
    shifted = torch.empty(flat.numel() + 1, dtype=torch.bfloat16, device="cuda")      # starts between two pixels
    shifted[1:] = flat
    td = torch.from_numpy(t).cuda()
    got = []
    for xd in (flat.view(n, 31, 31, 2), shifted[1:].view(n, 31, 31, 2)):
        out = net.forward(xd).cpu().numpy()[:, :6]
        loss, grad = net.gradient(xd, td)
        got.append((out, loss, grad.cpu().numpy()))
    net.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    out, loss, grad = got[0]
    # FP32 accumulation order can move an activation by one BF16 step (2^-9 of its size); each
    # such step passes through at most 288 products of the next layer
    assert np.linalg.norm(out - want_out) <= 4e-3 * np.linalg.norm(want_out)
    assert abs(loss - want_loss) <= 8e-3 * want_loss
    for name, (o, size) in O.LAYOUT.items():
        w = want[o:o + size]
        assert np.linalg.norm(grad[o:o + size] - w) <= 2e-2 * np.linalg.norm(w), name
