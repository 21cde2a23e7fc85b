"""What the server charges a sweep against its budget is what the sweep takes of
the device's memory, but for the margin it states (16 MiB) and the allocator's
rounding: a sweep that fits is not refused."""
import pytest

pytestmark = pytest.mark.gpu

MARGIN = 16 << 20


@pytest.mark.parametrize("h,w", [(1030, 1064), (2162, 2068)])
def test_sweep_bytes_are_the_bytes_taken(h, w):
    import torch
    from sfgb import serve
    srv = serve.Server(hbm_budget=1 << 40, max_batch=4, ring=8)
    first = srv.open_sweep(h, w)  # kernels, graphs and the shape's group
    torch.cuda.synchronize()
    free, used = torch.cuda.mem_get_info()[0], srv.used_bytes
    second = srv.open_sweep(h, w)
    torch.cuda.synchronize()
    taken, charged = free - torch.cuda.mem_get_info()[0], srv.used_bytes - used
    srv.close_sweep(second)
    srv.close_sweep(first)
    srv.close()
    assert charged == serve_bytes(h, w)
    assert taken <= charged, (taken, charged)
    assert charged - MARGIN <= 1.03 * taken, (taken, charged)


def serve_bytes(h, w):
    from sfgb import serve
    srv = serve.Server(hbm_budget=1 << 40, max_batch=4, ring=8)
    n = srv.sweep_bytes(h, w)
    srv.close()
    return n
