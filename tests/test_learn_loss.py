"""The loss kernel around its blocks of 256 values: the loss against float64 (a sum
of N terms of one sign is off by at most (N + 8) 2^-24 of itself), its gradient
to one rounding of each operand, masked rows and padding columns zero."""
import pytest
import torch

import sources_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,ld", [(1, 4), (63, 4), (64, 4), (65, 4), (2, 128), (1025, 128)])
@pytest.mark.parametrize("delta", [0.0, 0.7])
def test_loss_and_gradient(cuda_ok, rows, ld, delta):
    lib, nout = sources_b200.load(), 3
    g = torch.Generator().manual_seed(rows + ld)
    pred, target = torch.randn(rows, ld, generator=g).cuda(), torch.randn(rows, nout, generator=g).cuda()
    mask = (torch.rand(rows, generator=g) < 0.7).float()
    mask[0] = 1.0
    mask = mask.cuda()
    loss, dpred = torch.full((1,), 2.0, device="cuda"), torch.full_like(pred, 9.0)
    rc = lib.sphg_gnn_mse(pred.data_ptr(), ld, target.data_ptr(), nout, mask.data_ptr(), rows, 1.0 / 16, delta,
                          dpred.data_ptr(), loss.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    d = (pred[:, :nout] - target).double() * mask[:, None].double()     # the kernel's own FP32 difference
    big = (d.abs() > delta) if delta > 0 else torch.zeros_like(d, dtype=torch.bool)
    dl = torch.tensor(delta, dtype=torch.float32).double().item()
    want = torch.where(big, dl * (2 * d.abs() - dl), d * d).sum().item() / 16
    n = rows * nout
    assert abs(loss.item() - 2.0 - want) <= (n + 8) * 2.0 ** -24 * (2.0 + want)   # added to what was there
    grad = torch.where(big, 2 * dl * d.sign(), 2 * d) / 16
    assert (dpred[:, :nout].double() - grad).abs().max().item() <= 4 * 2.0 ** -24 * max(grad.abs().max().item(), 1e-30)
    assert dpred[:, nout:].abs().max().item() == 0.0 if ld > nout else True
    assert (dpred[mask == 0] == 0).all()
