"""The network's kernels at the sizes where they can go wrong: both tile sizes of
the BF16 product with every operand layout, partial tiles and odd strides;
forward and backward of odd widths and row counts; column sums; Adam on
several tensors.

Tolerances: the product accumulates K terms in FP32, as the existing test's
(rtol 1e-5, atol 1e-4 sqrt(K)); predictions and gradients those of the
existing network test (2e-2, 3e-2 normwise: BF16 operands); column sums of R
values of order one 1e-6 R; Adam against the one-tensor entry point, without
tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run_gemm(A, B, ta, tb, pad):
    """C = relu(A B) through ps_gemm_bf16 with A stored transposed if ta, B if
    tb, rows padded by `pad` elements; returns C (FP32) and its BF16 copy."""
    import ctypes as C

    import torch
    from ps_claude_opt_b200 import native

    def store(x, t):
        x = (x.T if t else x).contiguous()
        y = torch.zeros((x.shape[0], x.shape[1] + pad), dtype=torch.bfloat16, device="cuda")
        y[:, :x.shape[1]] = x
        return y

    M, K = A.shape
    N = B.shape[1]
    a, b = store(A, ta), store(B, tb)
    sa, sb = a.shape[1], b.shape[1]
    c = torch.empty((M, N), dtype=torch.float32, device="cuda")
    cb = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    native._check(native.lib().ps_gemm_bf16(M, N, K, p(a), 1 if ta else sa, sa if ta else 1, p(b), 1 if tb else sb,
                                            sb if tb else 1, p(c), N, 0, None, 1, p(cb), N, None))
    torch.cuda.synchronize()
    return c, cb


@pytest.mark.parametrize("M,N,K", [(2000, 300, 200), (2049, 257, 17), (33, 31, 129), (256, 256, 1000), (1, 300, 64)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad", [0, 3])
def test_gemm_tiles(M, N, K, ta, tb, pad):
    import torch

    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn((M, K), generator=g).to(torch.bfloat16).cuda()
    B = torch.randn((K, N), generator=g).to(torch.bfloat16).cuda()
    c, cb = _run_gemm(A, B, ta, tb, pad)
    want = torch.relu(A.double() @ B.double())
    assert torch.allclose(c.double(), want, rtol=1e-5, atol=1e-4 * np.sqrt(K))
    assert torch.equal(cb, c.to(torch.bfloat16))


@pytest.mark.parametrize("sizes,rows", [((88, 256, 256, 256, 1), 1), ((88, 256, 256, 256, 1), 1025), ((7, 33, 5, 1), 130),
                                        ((16, 1), 64), ((24, 300, 1), 4097)])
def test_forward_and_backward(sizes, rows):
    import torch
    from oracle import screen_ref
    from ps_claude_opt_b200 import screen

    rng = np.random.default_rng(rows)
    net = screen.Mlp(sizes=sizes, seed=2)
    x = rng.standard_normal((rows, sizes[0])).astype(np.float32)
    y = rng.standard_normal(rows).astype(np.float32)
    W, b = [w.cpu().numpy() for w in net.W], [v.cpu().numpy().astype(np.float64) for v in net.b]
    yhat = net.forward(torch.from_numpy(x).cuda().to(torch.bfloat16))
    diff = yhat - torch.from_numpy(y).cuda()
    gW, gb = net.backward((2.0 / rows) * diff)
    _, yref, gWr, gbr = screen_ref.mlp_forward_backward(x, y.astype(np.float64), W, b)
    assert np.allclose(yhat.cpu().numpy(), yref, rtol=2e-2, atol=2e-2)
    for g, r in zip(gW + gb, gWr + gbr):
        assert np.linalg.norm(g.cpu().numpy() - r) <= 3e-2 * np.linalg.norm(r)


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (1024, 256), (5000, 1)])
def test_column_sums(rows, cols):
    import ctypes as C

    import torch
    from ps_claude_opt_b200 import native

    x = torch.randn((rows, cols), generator=torch.Generator().manual_seed(3)).cuda()
    out = torch.empty(cols, device="cuda")
    native._check(native.lib().ps_column_sum(rows, cols, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    assert torch.allclose(out.double(), x.double().sum(0), rtol=0, atol=1e-6 * rows)


def test_adam_on_several_tensors_equals_one_by_one():
    import ctypes as C

    import torch
    from ps_claude_opt_b200 import native, screen

    a, b = screen.Mlp(sizes=(9, 257, 3, 1), seed=1), screen.Mlp(sizes=(9, 257, 3, 1), seed=1)
    g = torch.Generator().manual_seed(8)
    gW = [torch.randn(w.shape, generator=g).cuda() for w in a.W]
    gb = [torch.randn(v.shape, generator=g).cuda() for v in a.b]
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    for step in (1, 2):
        a.adam(gW, gb)
        for w, gr, m, v, wb in zip(b.W + b.b, gW + gb, b.mW + b.mb, b.vW + b.vb, b.Wb + [None] * len(b.b)):
            native._check(native.lib().ps_adam_step(w.numel(), p(w), p(gr), p(m), p(v), 1e-3, 0.9, 0.999, 1e-8, step,
                                                    p(wb), None))
    torch.cuda.synchronize()
    for x, y in zip(a.W + a.b + a.mW + a.vb + a.Wb, b.W + b.b + b.mW + b.vb + b.Wb):
        assert torch.equal(x, y)
