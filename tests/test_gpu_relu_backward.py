"""ps_relu_backward: dz = dh where z > 0, else 0 (a NaN of z gives 0), as FP32 and
BF16; either output may be left out, and neither is refused."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 100_003])
def test_relu_backward(n):
    import torch
    from ps_claude_opt_b200 import native

    g = torch.Generator().manual_seed(n)
    dh, z = (torch.randn(n, generator=g).cuda() for _ in range(2))
    z[::7] = 0.0
    z[::11] = float("nan")
    want = torch.where(z > 0, dh, torch.zeros_like(dh))
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for with_f, with_b in ((True, True), (True, False), (False, True)):
        dz = torch.full_like(dh, 7.0) if with_f else None
        dzb = torch.full_like(dh, 7.0, dtype=torch.bfloat16) if with_b else None
        native._check(native.lib().ps_relu_backward(n, ptr(dh), ptr(z), ptr(dz), ptr(dzb), stream))
        assert dz is None or torch.equal(dz, want)
        assert dzb is None or torch.equal(dzb, want.to(torch.bfloat16))
    with pytest.raises(native.PsError):
        native._check(native.lib().ps_relu_backward(n, ptr(dh), ptr(z), None, None, stream))
