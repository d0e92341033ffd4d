"""Weight and bias gradients of the guess network at the edges of their split
over a cluster (1, 2, 4 and 8 ranges of samples, uneven last ranges) and of the
64 x 64 tiles, against the float64 oracle.  Tolerance as for the other FP32
kernels: 2e-5 of the largest magnitude (sums of at most 4097 products, each
rounded to 6e-8)."""

import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m,dims', [(255, [64, 65, 63]), (256, [65, 64, 128]), (511, [7, 130, 1]), (512, [134, 128, 196]),
                                    (1023, [1, 64, 64]), (1024, [63, 33, 129]), (4097, [134, 128, 196])])
def test_split_gradients(m, dims):
    import torch
    from veloxchem_b200.guess_net import GuessMLP
    net = GuessMLP(dims[0], dims[-1], width=dims[1], depth=2, seed=3)
    layers = [(w.double().cpu().numpy(), b.double().cpu().numpy(), i == 0)
              for i, (w, b) in enumerate(zip(net.W, net.b))]
    rng = np.random.default_rng(m)
    x, dy = (rng.standard_normal((m, n)).astype(np.float32) for n in (dims[0], dims[-1]))
    y, cache = net.forward(torch.tensor(x, device=net.dev), keep=True)
    grads = net.backward(torch.tensor(dy, device=net.dev), cache)
    again = net.backward(torch.tensor(dy, device=net.dev), cache)
    expect = mo.backward(dy.astype(np.float64), layers, mo.forward(x.astype(np.float64), layers)[1])
    for (dw, db), (dw2, db2), (ew, eb) in zip(grads, again, expect):
        assert torch.equal(dw, dw2) and torch.equal(db, db2)  # the ranges are added in a fixed order
        for got, want in ((dw, ew), (db, eb)):
            assert np.max(np.abs(got.double().cpu().numpy() - want)) < 2e-5 * np.max(np.abs(want))


@pytest.mark.parametrize('m,n', [(64, 64), (300, 130), (4096, 128)])
@pytest.mark.parametrize('where', ['dY', 'Z'])
def test_input_gradient_in_place(m, n, where):
    """dX in the memory of dY or Z (square layers): equal to dX in its own."""
    import ctypes
    import torch
    from veloxchem_b200 import _native as nat
    gen = torch.Generator('cuda').manual_seed(m + n)
    x, z, dy = (torch.randn(m, n, device='cuda', generator=gen) for _ in range(3))
    w = torch.randn(n, n, device='cuda', generator=gen)

    def backward(dx, z, dy):
        dz, dw, db = torch.empty_like(dy), torch.empty_like(w), torch.empty(n, device='cuda')
        p = [ctypes.c_void_p(t.data_ptr()) for t in (x, w, z, dy, dz, dx, dw, db)]
        nat.check(nat.lib().vlx_b200_mlp_linear_backward(*p, m, n, n, 1,
                                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), 'backward')
        return dx, dw, db

    apart = backward(torch.empty_like(x), z, dy)
    buf = (dy if where == 'dY' else z).clone()
    inside = backward(buf, buf if where == 'Z' else z, buf if where == 'dY' else dy)
    assert all(torch.equal(a, b) for a, b in zip(apart, inside))
