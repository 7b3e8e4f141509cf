"""Entry points of the network's C interface that the package itself no longer calls
(its backward pass runs fused forms): against plain torch."""
import pytest
import torch

import sources_b200

pytestmark = pytest.mark.gpu


@pytest.fixture
def env(cuda_ok):
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    return sources_b200.load(), torch.cuda.current_stream().cuda_stream, lambda *s: torch.randn(s, device="cuda", generator=g)


@pytest.mark.parametrize("rows,cols", [(1, 4), (33, 64), (700, 128), (5001, 256)])
@pytest.mark.parametrize("f32", [0, 1])
def test_transpose(env, rows, cols, f32):
    lib, s, randn = env
    x = randn(rows, cols) if f32 else randn(rows, cols).to(torch.bfloat16)
    out = torch.zeros((cols, rows), dtype=torch.bfloat16, device="cuda")
    assert lib.sphg_gnn_transpose(x.data_ptr(), f32, out.data_ptr(), rows, cols, s) == 0
    assert torch.equal(out, x.to(torch.bfloat16).t())


@pytest.mark.parametrize("n", [4, 1020, 128 * 4099])
def test_f32_to_bf16(env, n):
    lib, s, randn = env
    x, y = randn(n), torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    assert lib.sphg_gnn_f32_to_bf16(x.data_ptr(), y.data_ptr(), n, s) == 0
    assert torch.equal(y, x.to(torch.bfloat16))
    assert lib.sphg_gnn_f32_to_bf16(x.data_ptr(), y.data_ptr(), 3, s) == 4


@pytest.mark.parametrize("rows,cols", [(1, 128), (513, 128), (5001, 256)])
def test_colsum(env, rows, cols):
    """Added to out: N terms and what was there, one rounding each."""
    lib, s, randn = env
    x, out = randn(rows, cols), torch.ones(cols, device="cuda")
    assert lib.sphg_gnn_colsum(x.data_ptr(), rows, cols, out.data_ptr(), s) == 0
    d = x.double()
    assert ((out.double() - 1 - d.sum(0)).abs() <= 2.0 ** -24 * (rows + 1) * (d.abs().sum(0) + 1)).all()


def test_relu_bwd(env):
    lib, s, randn = env
    n = 128 * 333
    dh, z = randn(n), randn(n)
    z[::7] = 0.0
    dz, dzb = torch.full_like(dh, 9.0), torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    assert lib.sphg_gnn_relu_bwd(dh.data_ptr(), z.data_ptr(), dz.data_ptr(), dzb.data_ptr(), n, s) == 0
    want = torch.where(z > 0, dh, torch.zeros((), device="cuda"))
    assert torch.equal(dz, want) and torch.equal(dzb, want.to(torch.bfloat16))


@pytest.mark.parametrize("ne", [1, 40, 7003])
def test_segsum_bwd(env, ne):
    """de += scale dagg[dst]: a product and a sum, at most two roundings."""
    lib, s, randn = env
    nn = ne // 9 + 3
    dagg, de = randn(nn, 128), randn(ne, 128)
    dst = torch.sort(torch.randint(0, nn, (ne,), device="cuda", dtype=torch.int32))[0].contiguous()
    add = dagg[dst.long()].double() * 0.125
    want = de.double() + add
    assert lib.sphg_gnn_segsum_bwd(dagg.data_ptr(), dst.data_ptr(), de.data_ptr(), ne, 128, 0.125, s) == 0
    assert ((de.double() - want).abs() <= 2.0 ** -23 * (want.abs() + add.abs())).all()
    assert lib.sphg_gnn_segsum_bwd(dagg.data_ptr(), dst.data_ptr(), de.data_ptr(), ne, 64, 0.125, s) == 4
