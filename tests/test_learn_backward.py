"""The backward pass's fused kernels against FP64 numpy: the weight-gradient
GEMM (MN-major operands straight from row-major rows), the bf16 cast with column
sums, the edge-gradient pass, the ReLU-backward GEMM epilogue and the one-launch
Adam step."""
import ctypes as C

import numpy as np
import pytest

from sources_b200 import learn, load

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    return load()


def bf(a):
    import torch
    t = torch.from_numpy(a.astype(np.float32)).cuda().to(torch.bfloat16)
    return t, t.float().cpu().numpy().astype(np.float64)


# one row block; a lone and a ragged split over CTAs; more blocks than 4 x 148 CTAs hold evenly
@pytest.mark.parametrize("rows", [128, 384, 4992, 128 * 301])
@pytest.mark.parametrize("out,inn", [(128, 64), (128, 128), (128, 256), (256, 128)])
def test_wgrad_matches_fp64(cuda_ok, lib, out, inn, rows):
    import torch
    g = np.random.default_rng(rows + out + inn)
    Y, y = bf(g.normal(size=(rows, out)))
    X, x = bf(g.normal(size=(rows, inn)))
    G0 = g.normal(size=(out, inn)).astype(np.float32)
    G = torch.from_numpy(G0).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = lib.sphg_gnn_wgrad(Y.data_ptr(), X.data_ptr(), G.data_ptr(), rows, out, inn, err.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    # exact products; one fp32 rounding of the running sum per 16 rows, per CTA's share and for G itself
    tol = 2.0 ** -23 * (rows / 16 + 160) * (np.abs(y).T @ np.abs(x) + np.abs(G0))
    e = np.abs(G.cpu().numpy() - (y.T @ x + G0))
    assert (e <= tol).all(), float((e / tol).max())


def test_wgrad_rejects_bad_arguments(lib):
    f = lib.sphg_gnn_wgrad
    p = C.c_void_p(256)
    assert f(None, p, p, 128, 128, 128, p, None) == 4
    assert f(p, p, p, 100, 128, 128, p, None) == 4
    assert f(p, p, p, 0, 128, 128, p, None) == 4
    assert f(p, C.c_void_p(264), p, 128, 128, 128, p, None) == 4
    assert f(p, p, p, 128, 256, 256, p, None) == 8


@pytest.mark.parametrize("rows", [1, 7, 128, 70001])
@pytest.mark.parametrize("cols,c0", [(128, 0), (256, 128), (256, 0)])
def test_cast_colsum(cuda_ok, lib, rows, cols, c0):
    import torch
    g = np.random.default_rng(rows + cols)
    x = torch.from_numpy(g.normal(size=(rows, cols)).astype(np.float32)).cuda()
    y = torch.zeros((rows, cols), dtype=torch.bfloat16, device="cuda")
    out = torch.ones(128, dtype=torch.float32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    assert lib.sphg_gnn_cast_colsum(x.data_ptr(), y.data_ptr(), rows, cols, c0, out.data_ptr(), s) == 0
    assert torch.equal(y, x.to(torch.bfloat16))
    a = x.double()[:, c0:c0 + 128]
    tol = 2.0 ** -24 * (rows / 8 + 1200) * (a.abs().sum(0) + 1)
    assert ((out.double() - 1 - a.sum(0)).abs() <= tol).all()
    assert lib.sphg_gnn_cast_colsum(x.data_ptr(), None, rows, cols, c0, None, s) == 0


@pytest.mark.parametrize("init", [0, 1])
@pytest.mark.parametrize("ne,npad", [(1, 128), (128, 128), (1000, 1024), (70000, 70016)])
def test_edge_grad(cuda_ok, lib, ne, npad, init):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(ne)
    nn = ne // 9 + 3
    dagg = torch.randn((nn, 128), device="cuda", generator=g)
    dst = torch.sort(torch.randint(0, nn, (ne,), device="cuda", generator=g, dtype=torch.int32))[0].contiguous()
    de = torch.randn((npad, 128), device="cuda", generator=g)
    de[ne:] = 0
    want = (torch.zeros_like(de) if init else de.clone())
    want[:ne] += dagg[dst.long()] * learn.AGG_SCALE
    deb = torch.empty((npad, 128), dtype=torch.bfloat16, device="cuda")
    gb = torch.zeros(128, device="cuda")
    if init:
        de.fill_(float("nan"))   # not read
    s = torch.cuda.current_stream().cuda_stream
    assert lib.sphg_gnn_edge_grad(dagg.data_ptr(), dst.data_ptr(), de.data_ptr(), deb.data_ptr(), gb.data_ptr(), ne, npad,
                                  learn.AGG_SCALE, init, s) == 0
    assert ((de - want).abs() <= 2.0 ** -23 * want.abs().clamp(min=1)).all()   # an add, perhaps fused with the scaling
    assert torch.equal(deb, de.to(torch.bfloat16))
    tol = 2.0 ** -24 * (ne / 8 + 1200) * (de.double().abs().sum(0) + 1)
    assert ((gb.double() - de.double().sum(0)).abs() <= tol).all()


@pytest.mark.parametrize("M", [128, 640, 128 * 301])
@pytest.mark.parametrize("keep", [True, False])
def test_relu_bwd_epilogue(cuda_ok, lib, M, keep):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    A = torch.randn((M, 128), device="cuda", generator=g).to(torch.bfloat16)
    W = torch.randn((128, 128), device="cuda", generator=g).to(torch.bfloat16)
    P = torch.randn((M, 128), device="cuda", generator=g)
    P[::5] = 0.0
    z = torch.empty((M, 128), device="cuda")
    h = torch.empty((M, 128), dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    e = learn.GemmEpi(learn.EPI_RELU_BWD, 0, None, z.data_ptr() if keep else None, h.data_ptr(), P.data_ptr(), None, None, 0)
    assert lib.sphg_gemm_bf16_ws(A.data_ptr(), W.data_ptr(), M, 128, 128, C.addressof(e), err.data_ptr(),
                                 torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    want = torch.where(P > 0, A.double() @ W.double().t(), torch.zeros((), dtype=torch.float64, device="cuda"))
    tol = 2.0 ** -23 * 16 * (A.double().abs() @ W.double().abs().t())
    if keep:
        assert ((z.double() - want).abs() <= tol).all()
        assert torch.equal(h, z.to(torch.bfloat16))
    assert ((h.double() - want).abs() <= tol + 2.0 ** -8 * want.abs()).all()
    assert (h[P <= 0] == 0).all()
    bad = learn.GemmEpi(learn.EPI_RELU_BWD, 0, None, None, h.data_ptr(), None, None, None, 0)
    assert lib.sphg_gemm_bf16_ws(A.data_ptr(), W.data_ptr(), M, 128, 128, C.addressof(bad), err.data_ptr(), None) == 4


def test_adam_all_equals_adam(cuda_ok, lib):
    """One launch for every tensor: the same values as one launch each."""
    import torch
    net, ref = learn.MPNet(seed=3), learn.MPNet(seed=3)
    g = torch.Generator(device="cuda")
    for step in range(1, 4):
        g.manual_seed(step)
        net.grads.copy_(torch.randn(net.grads.shape, device="cuda", generator=g))
        net.adam(1e-3)
        s = torch.cuda.current_stream().cuda_stream
        for d, r in zip(list(net.W.values()) + list(net.B.values()), list(ref.W.values()) + list(ref.B.values())):
            p = lambda k: r[k].data_ptr() if k in r else None  # noqa: E731
            assert lib.sphg_gnn_adam(p("w"), d["g"].data_ptr(), p("m"), p("v"), p("wb"), p("wt"), r["rows"],
                                     r.get("cols", 1), 1e-3, 0.9, 0.999, 1e-8, step, r["lim"], s) == 0
    for d, r in zip(list(net.W.values()) + list(net.B.values()), list(ref.W.values()) + list(ref.B.values())):
        for k in ("w", "m", "v", "wb", "wt"):
            if k in d:
                assert torch.equal(d[k], r[k]), k
