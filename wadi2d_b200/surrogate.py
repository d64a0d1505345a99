"""The storm-sweep surrogate: a small fully connected network, 16 -> 256 -> 256 -> 256 -> 16 with ReLU between, that
maps a storm's descriptors to the peak flow and time to peak at the design points. It is trained and run on the
device by this package's own kernels: every product on the tensor cores (w2b_mlp_ops: BF16 operands, FP32
accumulation), with the activations and their gradients, the loss gradient, bias sums and Adam in the products'
epilogues.

Numbers: FP32 master weights, BF16 copies for the products; activations stored in BF16 between layers, the
pre-activations in FP32; gradients w.r.t. pre-activations rounded to BF16 before their products; bias gradients and
Adam in FP32. Inputs and targets are standardised by the caller's statistics (``Scaler``).
"""

from __future__ import annotations

from dataclasses import dataclass

import numpy as np

from wadi2d_b200 import _lib

DIMS = (16, 256, 256, 256, 16)


def _pad16(n: int) -> int:
    return (n + 15) // 16 * 16


@dataclass
class Scaler:
    """Per-column standardisation: (x - mean) / std."""

    mean: np.ndarray
    std: np.ndarray

    @classmethod
    def fit(cls, x: np.ndarray) -> Scaler:
        x = np.asarray(x, np.float64)
        return cls(x.mean(0), np.where(x.std(0) > 1e-12, x.std(0), 1.0))

    def to(self, x):
        return (np.asarray(x, np.float64) - self.mean) / self.std

    def back(self, z):
        return np.asarray(z, np.float64) * self.std + self.mean


class Network:
    """The network's weights on the device and its forward pass, gradients and Adam steps."""

    def __init__(self, dims=DIMS, seed: int = 0, device="cuda", lr: float = 1e-3) -> None:
        import torch

        self.torch = torch
        self.dims = tuple(int(d) for d in dims)
        for d in self.dims[1:]:
            if d % 16 or not 16 <= d <= 256:
                raise ValueError("layer widths must be multiples of 16 between 16 and 256")
        if self.dims[0] % 16:
            raise ValueError("the input width must be a multiple of 16")
        self.device = torch.device(device)
        rng = np.random.default_rng(seed)
        dev = self.device
        self.W, self.b, self.Wb = [], [], []
        self.mW, self.vW, self.mb, self.vb = [], [], [], []
        for fan_in, fan_out in zip(self.dims[:-1], self.dims[1:], strict=True):
            w = rng.standard_normal((fan_out, fan_in)) * np.sqrt(2.0 / fan_in)  # He initialisation
            self.W.append(torch.as_tensor(w, dtype=torch.float32, device=dev))
            self.b.append(torch.zeros(fan_out, dtype=torch.float32, device=dev))
            self.Wb.append(torch.empty((fan_out, fan_in), dtype=torch.bfloat16, device=dev))
            for lst, shape in ((self.mW, (fan_out, fan_in)), (self.vW, (fan_out, fan_in)), (self.mb, (fan_out,)),
                               (self.vb, (fan_out,))):  # fmt: skip
                lst.append(torch.zeros(shape, dtype=torch.float32, device=dev))
        for i in range(len(self.W)):
            self._sync(i)
        self.lr = lr
        self.t = 0
        self.status = torch.zeros(3, dtype=torch.int32, device=dev)  # the status, and w2b_mlp_train's barrier

    # ------------------------------------------------------------------ plumbing

    def _s(self) -> int:
        return self.torch.cuda.current_stream(self.device).cuda_stream

    def _sync(self, i: int) -> None:
        """The BF16 copy of layer i's weights."""
        W = self.W[i]
        _lib.call("w2b_bf16_act", W.data_ptr(), W.numel(), 0, self.Wb[i].data_ptr(), self._s())

    def _ops(self, *ops) -> None:
        """Products in one launch (w2b_mlp_ops): each a dict of W2BMlpOp's fields, tensors by reference."""
        _lib.call("w2b_mlp_ops", self._structs(ops), len(ops), self.status.data_ptr(), self._s())

    def _structs(self, ops):
        arr = (_lib.MlpOp * len(ops))()
        for o, given in zip(arr, ops, strict=True):
            for name, v in given.items():
                setattr(o, name, v.data_ptr() if isinstance(v, self.torch.Tensor) else v)
        return arr

    def _rows(self, x, width: int, n: int | None = None):
        """x (host array, or a device tensor) as contiguous FP32 rows on the device, 16-byte aligned: as many as x has,
        or n."""
        torch = self.torch
        if not (isinstance(x, torch.Tensor) and x.is_cuda):
            x = torch.as_tensor(np.asarray(x, np.float32), device=self.device)
        x = x.to(device=self.device, dtype=torch.float32)
        n = x.shape[0] if n is None else n
        while x.dim() > 2 and x.shape[0] == 1:  # leading dimensions of one, as an assignment takes them
            x = x[0]
        x = torch.broadcast_to(x, (n, width)).contiguous()
        if n == 0:
            return torch.zeros((1, width), dtype=torch.float32, device=self.device), 0
        return (x.clone() if x.data_ptr() % 16 else x), n

    # ------------------------------------------------------------------ passes

    def _forward(self, x, n: int, keep: bool, loss=None, pick=None):
        """The products of a forward pass over n rows of x padded to npad, one a launch, with the layers'
        pre-activations (FP32) and with ``keep`` their inputs (BF16) that they write. ``loss``: the last product's
        further fields (targets, scale, dy, partials); ``pick``: the fields that draw the rows from the data set x."""
        torch, dev = self.torch, self.device
        npad, L = _pad16(max(n, 1)), len(self.W)

        def bf16(width):
            return torch.empty((npad, width), dtype=torch.bfloat16, device=dev)

        first = dict(x=x, valid=n, **(pick or {}))
        hs = [bf16(self.dims[0])] if keep else []
        if keep:
            first["h0"] = hs[0]
        zs, h, ops = [], None, []
        for i in range(L):
            out, inp = self.W[i].shape
            op = dict(b=self.Wb[i], m=npad, n=out, k=inp, bias=self.b[i], b_early=int(i > 0))
            op.update(first if i == 0 else dict(a=h))
            if keep or i == L - 1:
                zs.append(torch.empty((npad, out), dtype=torch.float32, device=dev))
                op["c"] = zs[-1]
            if i < L - 1:
                h = op["h"] = bf16(out)
                if keep:
                    hs.append(h)
            elif loss is not None:
                op.update(loss)
            ops.append(op)
        return npad, hs, zs, ops

    def forward(self, x, keep: bool = False):
        """Outputs (n x dims[-1], FP32 on the device) of standardised inputs x; with ``keep``, also the layers'
        inputs (BF16) and pre-activations (FP32) for the backward pass."""
        x, n = self._rows(x, self.dims[0])
        npad, hs, zs, ops = self._forward(x, n, keep)
        for op in ops:
            self._ops(op)
        return (zs[-1][:n], (n, npad, hs, zs)) if keep else zs[-1][:n]

    def _backward(self, x, t, n: int, pick=None):
        """The products of a forward and backward pass, one a launch, the loss's partial sums that they write, and the
        products of the weights' and biases' gradients (dz^T h, dz's column sums), to which the caller adds where they
        go: they come after all the others, which read the weights."""
        torch, dev = self.torch, self.device
        npad, nout = _pad16(max(n, 1)), self.dims[-1]
        dz = torch.empty((npad, nout), dtype=torch.bfloat16, device=dev)
        tiles = ((npad + 63) // 64) * ((nout + 31) // 32)
        partial = torch.empty(tiles, dtype=torch.float64, device=dev)
        loss = dict(t=t, valid=n, scale=2.0 / (n * nout), h=dz, partial=partial, **(pick or {}))
        npad, hs, zs, ops = self._forward(x, n, True, loss, pick)
        ends = []
        for i in range(len(self.W) - 1, -1, -1):
            out, inp = self.W[i].shape
            ends.append(dict(a=dz, b=hs[i], m=out, n=inp, k=npad, a_mn=1, b_mn=1, b_early=int(len(self.W) > 1)))
            if i > 0:
                back = torch.empty((npad, inp), dtype=torch.bfloat16, device=dev)
                ops.append(dict(a=dz, b=self.Wb[i], m=npad, n=inp, k=out, b_mn=1, z=zs[i - 1], h=back,
                                b_early=1))  # fmt: skip
                dz = back
        return ops, partial, ends[::-1]

    def gradients(self, x, t):
        """Mean-square error of the standardised targets t and the gradients of the weights and biases (FP32)."""
        torch = self.torch
        x, n = self._rows(x, self.dims[0])
        t, _ = self._rows(t, self.dims[-1], n)
        ops, partial, ends = self._backward(x, t, n)
        gW = [torch.empty_like(w) for w in self.W]
        gb = [torch.empty_like(b) for b in self.b]
        for op in ops:
            self._ops(op)
        for at in range(0, len(ends), _lib.MLP_OPS_MAX):
            part = slice(at, at + _lib.MLP_OPS_MAX)
            self._ops(*(dict(e, c=w, gb=b) for e, w, b in zip(ends[part], gW[part], gb[part], strict=True)))
        loss = torch.empty(1, dtype=torch.float64, device=self.device)
        at0 = torch.zeros(1, dtype=torch.int64, device=self.device)
        _lib.call("w2b_mlp_tick", partial.data_ptr(), partial.numel(), float(n * self.dims[-1]), loss.data_ptr(),
                  at0.data_ptr(), self._s())  # fmt: skip
        return loss[0], gW, gb

    def _lr(self, t: int, b1: float = 0.9, b2: float = 0.999) -> float:
        """Adam's bias-corrected step size at step t."""
        return float(self.lr * np.sqrt(1.0 - b2**t) / (1.0 - b1**t))

    def _adam(self, gW, gb, lr_t: float, b1: float = 0.9, b2: float = 0.999, eps: float = 1e-8):
        """Adam on every layer with step size lr_t."""
        for i in range(len(self.W)):
            for w, g, m, v in ((self.W[i], gW[i], self.mW[i], self.vW[i]), (self.b[i], gb[i], self.mb[i], self.vb[i])):
                _lib.call("w2b_adam", w.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), w.numel(), lr_t, b1,
                          b2, eps, None, self._s())  # fmt: skip
            self._sync(i)

    def _check(self) -> None:
        status = int(self.status[0].item())
        if status != 0:
            raise _lib.W2BError(status, "w2b_mlp_ops")

    def step(self, x, t):
        """One Adam step on the batch (x, t); returns the loss before the step (a device scalar)."""
        loss, gW, gb = self.gradients(x, t)
        self.t += 1
        self._adam(gW, gb, self._lr(self.t))
        self._check()
        return loss

    def fit(self, x, t, iters: int = 2000, batch: int = 256, seed: int = 0, graph: bool = True) -> list[float]:
        """Adam over random batches of (x, t), standardised; returns the loss every 100 steps.

        With ``graph`` (the default) the batches are drawn up front (the same draws, in the same order, as one step
        at a time draws them), the training set goes to the device once, and the library takes every step (gather,
        forward, backward, Adam with the step's own size, all read on the device) in one launch: the same arithmetic on
        the same data in the same order as stepping from the host, without a host round trip a step."""
        rng = np.random.default_rng(seed)
        x, t = np.asarray(x, np.float32), np.asarray(t, np.float32)
        bs = min(batch, x.shape[0])
        draws = [rng.choice(x.shape[0], size=bs, replace=False) for _ in range(iters)]
        if not graph or iters < 2:
            losses = []
            for it in range(iters):
                loss = self.step(x[draws[it]], t[draws[it]])
                if it % 100 == 0 or it == iters - 1:
                    losses.append(float(loss))
            return losses
        torch, dev = self.torch, self.device
        X, T = self._rows(x, self.dims[0])[0], self._rows(t, self.dims[-1])[0]
        if t.shape[0] < x.shape[0]:
            raise IndexError(f"{t.shape[0]} targets for {x.shape[0]} rows")
        idx = torch.as_tensor(np.stack(draws).astype(np.int64), device=dev)
        lr = torch.as_tensor(np.array([self._lr(self.t + s) for s in range(1, iters + 1)], np.float32), device=dev)
        k = torch.zeros(1, dtype=torch.int64, device=dev)
        loss_at = torch.zeros(iters, dtype=torch.float64, device=dev)
        pick = dict(rows=idx, step=k, batch=bs)
        ops, partial, ends = self._backward(X, T, bs, pick)
        launches = [[op] for op in ops]
        ends = [dict(end, w=self.W[i], mw=self.mW[i], vw=self.vW[i], wb=self.Wb[i], gb=self.b[i], mb=self.mb[i],
                     vb=self.vb[i], lr_table=lr, step=k, b1=0.9, b2=0.999, eps=1e-8)
                for i, end in enumerate(ends)]  # fmt: skip
        launches += [ends[at : at + _lib.MLP_OPS_MAX] for at in range(0, len(ends), _lib.MLP_OPS_MAX)]
        sizes = np.array([len(group) for group in launches], np.int32)
        _lib.call("w2b_mlp_train", self._structs([op for group in launches for op in group]), sizes.ctypes.data,
                  sizes.size, iters, partial.data_ptr(), partial.numel(), float(bs * self.dims[-1]), loss_at.data_ptr(),
                  k.data_ptr(), self.status.data_ptr(), self._s())  # fmt: skip
        self.t += iters
        self._check()
        out = loss_at.cpu().numpy()
        return [float(out[it]) for it in range(iters) if it % 100 == 0 or it == iters - 1]

    def predict(self, x) -> np.ndarray:
        return self.forward(x).cpu().numpy().astype(np.float64)

    def weights(self) -> list[tuple[np.ndarray, np.ndarray]]:
        return [(w.cpu().numpy().astype(np.float64), b.cpu().numpy().astype(np.float64)) for w, b in zip(self.W, self.b)]
