"""w2b_mlp_train through its own interface, against the same products launched one by one (w2b_mlp_ops, w2b_mlp_tick), bit for
bit: a draw of rows that is the same every step (no step counter), a step counter that is not the call's, and a loss that
the last launch of a step writes."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BATCH, WIDTH, ITERS = 200, 16, 6


def _structs(ops):
    import torch

    from wadi2d_b200 import _lib

    arr = (_lib.MlpOp * len(ops))()
    for o, given in zip(arr, ops, strict=True):
        for name, v in given.items():
            setattr(o, name, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    return arr


class Layer:
    """One layer of WIDTH trained on BATCH of 300 rows: the products of a step, in launches."""

    def __init__(self, step: str, train: bool = True) -> None:
        import torch

        rng = np.random.default_rng(5)
        f32 = lambda a: torch.as_tensor(np.asarray(a, np.float32), device="cuda")  # noqa: E731
        pad = (BATCH + 15) // 16 * 16
        self.x, self.t = f32(rng.standard_normal((300, WIDTH))), f32(rng.standard_normal((300, WIDTH)))
        # a draw for every step and more: a read past the first stays in the array
        self.rows = torch.as_tensor(np.stack([rng.permutation(300)[:BATCH] for _ in range(2 * ITERS)]), device="cuda")
        self.step = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.other = torch.full((1,), 2, dtype=torch.int64, device="cuda")
        self.w, self.b = f32(rng.standard_normal((WIDTH, WIDTH))), f32(rng.standard_normal(WIDTH))
        self.wb = self.w.to(torch.bfloat16)
        self.moments = [torch.zeros_like(v) for v in (self.w, self.w, self.b, self.b)]
        self.dz = torch.zeros((pad, WIDTH), dtype=torch.bfloat16, device="cuda")
        self.h0 = torch.zeros((pad, WIDTH), dtype=torch.bfloat16, device="cuda")
        self.partial = torch.full(((pad + 63) // 64,), np.nan, dtype=torch.float64, device="cuda")
        self.loss = torch.full((ITERS,), np.nan, dtype=torch.float64, device="cuda")
        self.status = torch.zeros(3, dtype=torch.int32, device="cuda")
        pick = {"none": {}, "own": dict(step=self.step), "other": dict(step=self.other)}[step]
        forward = dict(x=self.x, rows=self.rows, batch=BATCH, valid=BATCH, h0=self.h0, b=self.wb, m=pad, n=WIDTH, k=WIDTH,
                       bias=self.b, t=self.t, scale=2.0 / (BATCH * WIDTH), h=self.dz, partial=self.partial, **pick)  # fmt: skip
        mw, vw, mb, vb = self.moments
        end = dict(a=self.dz, b=self.h0, m=WIDTH, n=WIDTH, k=pad, a_mn=1, b_mn=1, w=self.w, mw=mw, vw=vw, wb=self.wb,
                   gb=self.b, mb=mb, vb=vb, lr=0.05, b1=0.9, b2=0.999, eps=1e-8)  # fmt: skip
        self.launches = [[forward], [end]] if train else [[forward]]

    def fit(self, one_call: bool):
        import torch

        from wadi2d_b200 import _lib

        s = torch.cuda.current_stream().cuda_stream
        count = float(BATCH * WIDTH)
        if one_call:
            sizes = np.array([len(g) for g in self.launches], np.int32)
            _lib.call("w2b_mlp_train", _structs([op for g in self.launches for op in g]), sizes.ctypes.data, sizes.size, ITERS,
                      self.partial.data_ptr(), self.partial.numel(), count, self.loss.data_ptr(), self.step.data_ptr(),
                      self.status.data_ptr(), s)  # fmt: skip
        else:
            for _ in range(ITERS):
                for g in self.launches:
                    _lib.call("w2b_mlp_ops", _structs(g), len(g), self.status.data_ptr(), s)
                _lib.call("w2b_mlp_tick", self.partial.data_ptr(), self.partial.numel(), count, self.loss.data_ptr(),
                          self.step.data_ptr(), s)  # fmt: skip
        torch.cuda.synchronize()
        assert int(self.step.item()) == ITERS and not self.status.any()
        return [self.loss, self.w, self.b, self.wb, *self.moments, self.h0, self.dz]


@pytest.mark.parametrize("step", ["none", "own", "other"])
def test_rows_are_the_step_counters(step):
    import torch

    for a, b in zip(Layer(step).fit(False), Layer(step).fit(True), strict=True):
        assert torch.equal(a, b)


def test_a_loss_that_the_last_launch_writes():
    import torch

    a, b = Layer("own", train=False).fit(False), Layer("own", train=False).fit(True)
    assert len(set(a[0].tolist())) == ITERS
    for p, q in zip(a, b, strict=True):
        assert torch.equal(p, q)
