"""The training kernel at the edges of its tiles: one row, around one tile of 16
rows, and around one tile per CTA of the largest grid (608), against the FP64
oracle with the proposer's tolerances (2e-4 of the largest gradient entry, 1e-5
of the loss); the same bits on a second call."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 608 * 16 - 1, 608 * 16 + 1, 3 * 608 * 16 + 5])
def test_gradient_at_tile_edges(rg, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    bits = mo.bf16_bits(rng.normal(0, 0.3, mo.NPARAM).astype(np.float32))
    xn = rng.normal(0, 1, (n, mo.NFEAT)).astype(np.float32)
    tn = rng.normal(0, 1, n).astype(np.float32)
    w, X, T = (torch.from_numpy(a).cuda() for a in (bits.view(np.int16), xn, tn))
    got = []
    for _ in range(2):
        grad = torch.full((mo.NPARAM,), float("nan"), dtype=torch.float32, device="cuda")
        loss = torch.full((1,), float("nan"), dtype=torch.float32, device="cuda")
        rg.lib.mlp_grad(w.data_ptr(), X.data_ptr(), T.data_ptr(), n, grad.data_ptr(), loss.data_ptr())
        torch.cuda.synchronize()
        got.append((grad, loss))
    ref_loss, ref = mo.loss_and_grad(mo.bf16_value(bits), xn, tn)
    g, loss = got[0][0].cpu().numpy(), got[0][1].item()
    assert abs(loss - ref_loss) <= 1e-5 * ref_loss
    assert np.abs(g - ref).max() <= 2e-4 * np.abs(ref).max()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
