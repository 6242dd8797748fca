"""The contact form's scratch pool on the device: memory that it keeps for later
calls is there for any other allocation, the library's also while calls that
use it are still queued, and the host program's (PyTorch here) once they ended."""
import ctypes as ct

import pytest
import torch

import mcpi_b200 as mc

pytestmark = pytest.mark.gpu
MORE = 128 << 20                         # beyond what is free; the pool keeps 248 MB at N=16, M=10


def test_the_pool_gives_way():
    sp = mc.FockSpace(16, 10)
    sp.set_integrals(*mc.lieb_integrals(10, 1.0))
    x = torch.ones(sp.nc, dtype=torch.complex128, device="cuda")
    y = sp.apply_h(x)
    ref = y.clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    L, p = mc.lib(), ct.c_void_p()
    for _ in range(50):                  # their scratch is freed on the stream, the host has not seen it
        sp.apply_h(x, y)
    rc = L.mcpi_alloc(ct.c_void_p(sp._h.value), ct.c_size_t(free + MORE), ct.byref(p))
    assert rc == 0, L.mcpi_last_error()
    assert L.mcpi_free(ct.c_void_p(sp._h.value), p) == 0
    assert torch.equal(y, ref)
    sp.apply_h(x, y)                     # holds scratch again
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    t = torch.empty(free + MORE, dtype=torch.uint8, device="cuda")
    del t
    torch.cuda.empty_cache()
    assert torch.equal(sp.apply_h(x), ref)
    sp.close()
