"""Device memory of destroyed NMHs: aur_nmh_destroy gives back what its
context's pool does not keep (256 MiB) before it returns, so that an
allocation of another kind right after it finds it."""
import pytest

from aurora_gb300 import api

pytestmark = pytest.mark.gpu

POOL = 256 << 20


def test_destroy_gives_memory_back_at_once():
    import torch
    ctx = api.Context(0)
    n = 8 << 20                       # about 1 GB of records, treelets and vertices
    V = torch.rand((n, 9), device="cuda").reshape(-1)
    api.Nmh(ctx, V, count=n).close()  # the context's build scratch stays from here on
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    nmh = api.Nmh(ctx, V, count=n)
    used = before - torch.cuda.mem_get_info()[0]
    assert used > POOL + (256 << 20)
    nmh.close()
    after = torch.cuda.mem_get_info()[0]
    assert after >= before - POOL - (64 << 20), "%.0f MiB still held" % ((before - after) / 2 ** 20)
    ctx.close()
