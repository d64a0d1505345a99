"""The network's fused products (w2b_mlp_ops) on the B200 against FP64 products of the same BF16 values: every pair of
operand orders at the edges of the tiles (64 or 128 rows by 32) and of the 256-wide K chunk, and each epilogue against its definition
applied to the product the plain epilogue gives."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(*ops):
    import torch

    from wadi2d_b200 import _lib

    arr = (_lib.MlpOp * len(ops))()
    for o, given in zip(arr, ops, strict=True):
        for name, v in given.items():
            setattr(o, name, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("w2b_mlp_ops", arr, len(ops), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(status.item()) == 0


def _operands(rng, m, n, k):
    import torch

    make = lambda shape: torch.as_tensor(rng.standard_normal(shape), dtype=torch.float32).to(torch.bfloat16).cuda()  # noqa: E731
    return make((m, k)), make((n, k))


@pytest.mark.parametrize("m,n,k", [(16, 16, 16), (128, 32, 256), (144, 48, 272), (304, 256, 512), (256, 16, 1040), (2400, 256, 272)])
@pytest.mark.parametrize("a_mn", [0, 1])
@pytest.mark.parametrize("b_mn", [0, 1])
def test_products_in_every_order(m, n, k, a_mn, b_mn):
    import torch

    rng = np.random.default_rng(m + 3 * n + 7 * k)
    a, b = _operands(rng, m, n, k)
    c = torch.full((m, n), np.nan, device="cuda")
    gb = torch.full((m,), np.nan, device="cuda")
    op = dict(a=a.T.contiguous() if a_mn else a, b=b.T.contiguous() if b_mn else b, m=m, n=n, k=k, a_mn=a_mn, b_mn=b_mn,
              c=c)  # fmt: skip
    if a_mn:
        op["gb"] = gb
    _run(op)
    want = a.double() @ b.double().T
    tol = k * 2.0**-24 * float((a.double().abs() @ b.double().abs().T).max())  # k FP32 additions of exact products
    assert float((c.double() - want).abs().max()) <= tol
    if a_mn:
        serial = torch.zeros(m, device="cuda")
        for r in range(k):
            serial = serial + a[:, r].float()
        assert torch.equal(gb, serial)


def test_epilogues():
    import torch

    rng = np.random.default_rng(4)
    m, n, k, valid = 144, 48, 32, 139
    x = torch.as_tensor(rng.standard_normal((200, k)), dtype=torch.float32, device="cuda")
    rows = torch.as_tensor(np.stack([rng.permutation(200)[:valid] for _ in range(3)]), device="cuda")
    step = torch.full((1,), 2, dtype=torch.int64, device="cuda")
    _, b = _operands(rng, m, n, k)
    bias = torch.as_tensor(rng.standard_normal(n), dtype=torch.float32, device="cuda")
    pick = dict(x=x, rows=rows, step=step, batch=valid, valid=valid)
    f32 = lambda *s: torch.full(s, np.nan, device="cuda")  # noqa: E731
    bf = lambda *s: torch.full(s, np.nan, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    c, h, h0 = f32(m, n), bf(m, n), bf(m, k)
    _run(dict(pick, b=b, m=m, n=n, k=k, bias=bias, c=c, h=h, h0=h0))
    a = torch.zeros((m, k), dtype=torch.bfloat16, device="cuda")
    a[:valid] = x[rows[2]].to(torch.bfloat16)
    plain = f32(m, n)
    _run(dict(a=a, b=b, m=m, n=n, k=k, bias=bias, c=plain))
    assert torch.equal(h0, a) and torch.equal(c, plain)
    assert torch.equal(h, torch.relu(plain).to(torch.bfloat16))
    # behind an activation
    z = torch.as_tensor(rng.standard_normal((m, n)), dtype=torch.float32, device="cuda")
    _run(dict(a=a, b=b, m=m, n=n, k=k, bias=bias, z=z, h=h))
    assert torch.equal(h, torch.where(z > 0, plain, torch.zeros_like(plain)).to(torch.bfloat16))
    # the loss and its gradient
    t = torch.as_tensor(rng.standard_normal((200, n)), dtype=torch.float32, device="cuda")
    partial = torch.full((6,), np.nan, dtype=torch.float64, device="cuda")
    _run(dict(pick, b=b, m=m, n=n, k=k, bias=bias, t=t, scale=0.25, h=h, partial=partial))
    off = torch.zeros_like(plain)
    off[:valid] = plain[:valid] - t[rows[2]]
    assert torch.equal(h, (0.25 * off).to(torch.bfloat16))
    assert float(partial.sum()) == pytest.approx(float((off.double() ** 2).sum()), rel=1e-12)
    # Adam of two layers in one launch, against the products' gradients through w2b_adam
    from wadi2d_b200 import _lib

    layers, lr = [], torch.as_tensor(np.float32([0.1, 0.2, 1e-3]), device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for out, inp, batch in ((16, 256, 272), (256, 16, 272)):
        dz, hh = _operands(rng, out, inp, batch)
        dz, hh = dz.T.contiguous(), hh.T.contiguous()
        w, mw, vw = (torch.rand((out, inp), device="cuda") for _ in range(3))
        bb, mb, vb = (torch.rand(out, device="cuda") for _ in range(3))
        g, gb, wb = f32(out, inp), f32(out), bf(out, inp)
        base = dict(a=dz, b=hh, m=out, n=inp, k=batch, a_mn=1, b_mn=1)
        _run(dict(base, c=g, gb=gb))
        want = [v.clone() for v in (w, mw, vw, bb, mb, vb)]
        wantb = bf(out, inp)
        for (p, q, r), grad, to in ((want[:3], g, wantb), (want[3:], gb, None)):
            _lib.call("w2b_adam", p.data_ptr(), grad.data_ptr(), q.data_ptr(), r.data_ptr(), p.numel(),
                      float(np.float32(1e-3)), 0.9, 0.999, 1e-8, None if to is None else to.data_ptr(), s)  # fmt: skip
        op = dict(base, w=w, mw=mw, vw=vw, wb=wb, gb=bb, mb=mb, vb=vb, lr_table=lr, step=step, b1=0.9, b2=0.999, eps=1e-8)
        layers.append((op, (w, mw, vw, bb, mb, vb, wb), want + [wantb]))
    _run(*(op for op, _, _ in layers))
    for _, got, want in layers:
        for p, q in zip(got, want, strict=True):
            assert torch.equal(p, q)


@pytest.mark.parametrize("dims,iters,batch", [((16, 16), 2, 1), ((16, 48, 16), 513, 40), ((16,) + (32,) * 7 + (16,), 5, 144)])
def test_training_in_one_launch(dims, iters, batch):
    """Steps of a fit in the cooperative launch (one layer; more steps than a launch takes) and, with more products than
    it takes, launched one by one, against the host's step after step: losses, weights and biases bit for bit."""
    from wadi2d_b200.surrogate import Network

    rng = np.random.default_rng(11)
    x, t = (rng.standard_normal((150, 16)).astype(np.float32) for _ in range(2))
    nets = [Network(dims=dims, seed=4), Network(dims=dims, seed=4)]
    losses = [net.fit(x, t, iters=iters, batch=batch, seed=6, graph=graph) for net, graph in zip(nets, (True, False), strict=True)]
    assert losses[0] == losses[1]
    for (wa, ba), (wb, bb) in zip(nets[0].weights(), nets[1].weights(), strict=True):
        assert np.array_equal(wa, wb) and np.array_equal(ba, bb)
