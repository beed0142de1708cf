"""A handle that has run a whole wave of fits allocates no more, whatever number of
fits comes next, and one that has run fewer none for fewer still: free device
memory stays, and calls that put teams beside whole waves can be captured and
replayed."""
import numpy as np
import pytest

from conftest import prepared

pytestmark = pytest.mark.gpu


def _items(n):
    k = np.arange(n, dtype=np.int32)
    return 1 + k // 10 % 3, k % 10


def test_no_allocation_after_a_wave():
    import torch
    from ps_claude_opt_b200 import native

    torch.zeros(1, device="cuda")
    obj = prepared("c2")
    with native.Engine(obj) as eng:
        eng.configure(stop_condition=2.0)
        per_sm, n_sm = eng.occupancy()
        wave = per_sm * n_sm
        eng.fit_items(*_items(wave))
        eng.fit_items(*_items(2 * wave + 80))  # items and results grow with the number of fits
        free = torch.cuda.mem_get_info()[0]
        for n in (10, wave + 13, wave + 70, 2 * wave + 36):
            eng.fit_items(*_items(n))
            assert torch.cuda.mem_get_info()[0] == free
    nf, pl = _items(wave + 80)
    items = torch.from_numpy(np.stack([nf, pl], axis=1).astype(np.int32)).cuda()
    out = torch.zeros((len(nf), 56), dtype=torch.uint8, device="cuda")  # ps_fit_result
    torch.cuda.synchronize()
    with native.Engine(obj) as eng:
        eng.configure(stop_condition=2.0)
        eng.fit_items_device(wave, items.data_ptr(), out.data_ptr())
        free = torch.cuda.mem_get_info()[0]
        for n in (10, 36, 70, wave - 1, wave + 13, wave + 70):
            eng.fit_items_device(n, items.data_ptr(), out.data_ptr())
            assert torch.cuda.mem_get_info()[0] == free
        eng.status()  # waits for the handle's stream


def test_no_allocation_for_fewer_fits():
    import torch
    from ps_claude_opt_b200 import native

    obj = prepared("c1")  # a kernel no other test here has loaded
    nf, pl = _items(100)
    items = torch.from_numpy(np.stack([nf, pl], axis=1).astype(np.int32)).cuda()
    out = torch.zeros((len(nf), 56), dtype=torch.uint8, device="cuda")  # ps_fit_result
    torch.cuda.synchronize()
    with native.Engine(obj) as eng:
        eng.configure(stop_condition=2.0)
        eng.fit_items_device(100, items.data_ptr(), out.data_ptr())
        free = torch.cuda.mem_get_info()[0]
        for n in (74, 36, 18, 1):
            eng.fit_items_device(n, items.data_ptr(), out.data_ptr())
            assert torch.cuda.mem_get_info()[0] == free
        eng.status()  # waits for the handle's stream


@pytest.mark.parametrize("more", [13, 30, 70])
def test_teams_beside_a_wave_can_be_captured(more):
    import torch
    from ps_claude_opt_b200 import native

    obj = prepared("mixed")
    with native.Engine(obj) as eng:
        eng.configure(stop_condition=4.0)
        per_sm, n_sm = eng.occupancy()
        n = per_sm * n_sm + more
        nf, pl = _items(n)
        items = torch.from_numpy(np.stack([nf, pl], axis=1).astype(np.int32)).cuda()
        out = torch.zeros((n, 56), dtype=torch.uint8, device="cuda")  # ps_fit_result
        stream = torch.cuda.ExternalStream(eng.stream)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            eng.fit_items_device(n - more, items.data_ptr(), out.data_ptr())  # warm: one wave
        torch.cuda.synchronize()
        out.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            eng.fit_items_device(n, items.data_ptr(), out.data_ptr())
        want, it, st = eng.fit_items(nf, pl)  # another call between capture and replay
        for _ in range(2):
            out.zero_()
            g.replay()
            torch.cuda.synchronize()
            got = out.cpu().numpy()
            assert np.array_equal(got[:, :48].copy().view(np.float64), want, equal_nan=True)
            assert np.array_equal(got[:, 48:52].copy().view(np.int32)[:, 0], it)
            assert np.array_equal(got[:, 52:56].copy().view(np.int32)[:, 0], st)
        del g
