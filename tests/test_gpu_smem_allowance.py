"""The shared memory that the fit kernels are allowed belongs to the kernel, not to
a handle: after a small object has used a kernel, a large one of the same
coefficient count still finds its allowance, so that a thread with the one
cannot have a launch of a thread with the other refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class FuncAttributes(C.Structure):  # the head of cudaFuncAttributes
    _fields_ = [("shared", C.c_size_t), ("const", C.c_size_t), ("local", C.c_size_t), ("threads", C.c_int),
                ("regs", C.c_int), ("ptx", C.c_int), ("binary", C.c_int), ("cache", C.c_int), ("dynamic", C.c_int),
                ("rest", C.c_int * 64)]


def _allowed(lib, name):
    kernel = getattr(lib, name)
    kernel.restype = C.c_void_p
    rt = C.CDLL(next(l.split()[-1] for l in open("/proc/self/maps") if "libcudart.so" in l))
    a = FuncAttributes()
    assert rt.cudaFuncGetAttributes(C.byref(a), C.c_void_p(kernel())) == 0
    return a.dynamic


def _object(curves, rows):
    from ps_claude_opt_b200 import objects, synth

    cfg = synth.SynthConfig(l_max=6, m_max=6, nrows=rows, n_dense=curves, dense_pts=(12, 20), n_freq=20,
                            truth_grid=(30, 60))
    return objects.parse_input(synth.generate(cfg, 7)[0])


@pytest.mark.parametrize("precision", [0, 1])
def test_a_small_object_takes_nothing_from_a_large_one(precision):
    import dataclasses
    from ps_claude_opt_b200 import native

    lib = native.lib()
    small, large = _object(3, 5), _object(60, 8)
    need = getattr(lib, "_ZN3psb14fit_smem_bytesEiiiiiiii")
    need.restype = C.c_size_t
    kernels = ["_ZN3psb17fit_kernel_ptr_56Ev", "_ZN3psb22fit_kernel_team_ptr_56Ev"]
    if precision:
        kernels = ["_ZN3psb23fit_kernel_mixed_ptr_56Ev", "_ZN3psb28fit_kernel_mixed_team_ptr_56Ev"]

    def fits(obj):
        with native.Engine(obj) as eng:
            eng.set_precision(precision)
            eng.configure(stop_condition=2.0)
            n = int(np.prod(eng.occupancy())) + 10
            eng.fit_items(np.ones(n, dtype=np.int32), np.arange(n, dtype=np.int32) % 10)
            eng.eval(np.zeros(large.ma + 1) + 0.1)

    fits(large)
    fits(small)
    if not precision:
        kernels.append("_ZN3psb23fit_kernel_batch_ptr_56Ev")
        native.scan_batch([dataclasses.replace(small, stop_condition=2.0)], max_freq=1)
    nc = large.n_coef
    bytes_large = need(large.n_fac, large.mfit, (nc + 7) // 8 * 8, large.n_curves, (nc + 10) & ~1, 32, 1, precision)
    bytes_small = need(small.n_fac, small.mfit, (nc + 7) // 8 * 8, small.n_curves, (nc + 10) & ~1, 32, 1, precision)
    assert bytes_small < bytes_large <= 232448
    for name in kernels:
        assert _allowed(lib, name) >= bytes_large - 1120  # what is counted for static shared memory
