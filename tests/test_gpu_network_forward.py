"""The one-launch forward pass against the layers' single products, which sum
each result in the same chain: bit for bit, for FP32 and BF16 activations.  Row
counts around the 16-row blocks and the steps in rows per CTA (148 CTAs of 16,
32, 48 and 64 rows), widths at the tile's edges, and networks that go layer by
layer (too wide, a width that is no multiple of 8, an unaligned input)."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

NET = (88, 256, 256, 256, 1)


@pytest.mark.parametrize("sizes,rows,shift", [
    (NET, 1, 0), (NET, 15, 0), (NET, 17, 0), (NET, 2368, 0), (NET, 2369, 0), (NET, 4737, 0), (NET, 7105, 0),
    (NET, 9473, 0), (NET, 100, 1), ((8, 24, 40, 3), 33, 0), ((64, 256), 50, 0), ((256, 8, 256, 2), 130, 0),
    ((16,) + (64,) * 7 + (5,), 70, 0), ((16,) + (64,) * 8 + (5,), 70, 0), ((88, 264, 16, 1), 40, 0),
    ((88, 20, 33, 1), 40, 0)])
def test_forward_is_the_layers_one_by_one(sizes, rows, shift):
    import torch
    from ps_claude_opt_b200 import native

    g = torch.Generator().manual_seed(rows + len(sizes))
    L = len(sizes) - 1
    w = [torch.randn((n, k), generator=g).mul(k ** -0.5).to(torch.bfloat16).cuda() for k, n in zip(sizes, sizes[1:])]
    b = [torch.randn(n, generator=g).mul(0.1).cuda() for n in sizes[1:]]
    store = torch.randn(rows * sizes[0] + shift, generator=g).to(torch.bfloat16).cuda()
    x = store[shift:].view(rows, sizes[0])

    def buffers():
        return ([x] + [torch.zeros((rows, n), dtype=torch.bfloat16, device="cuda") for n in sizes[1:-1]],
                [torch.zeros((rows, n), dtype=torch.float32, device="cuda") for n in sizes[1:]])

    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    ptrs = lambda ts: (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])  # noqa: E731
    h, hf = buffers()
    lib = native.lib()
    native._check(lib.ps_mlp_forward(L, (C.c_int32 * (L + 1))(*sizes), rows, ptrs(w), ptrs(b), ptrs(h), ptrs(hf), None))
    h1, hf1 = buffers()
    for l, (k, n) in enumerate(zip(sizes, sizes[1:])):
        last = l == L - 1
        native._check(lib.ps_gemm_bf16(rows, n, k, p(h1[l]), k, 1, p(w[l]), 1, k, p(hf1[l]), n, 0, p(b[l]),
                                       0 if last else 1, None if last else p(h1[l + 1]), n, None))
    torch.cuda.synchronize()
    for l in range(L):
        assert torch.equal(hf[l], hf1[l])
        if l:
            assert torch.equal(h[l], h1[l])
