"""A call that fails after it has begun to copy from pinned memory (here because
the device memory is nearly all taken) returns with no copy under way, so that
the caller may free or reuse its arrays."""
import ctypes as C

import pytest

import signed_triangle_counting_b200 as stc
from signed_triangle_counting_b200 import _capi

pytestmark = pytest.mark.gpu


def test_no_copy_in_flight_after_a_failed_call():
    import torch
    m = 100_000_000  # 500 MB to copy, then 800 MB of keys that do not fit
    edges = torch.zeros(m, dtype=torch.int32).pin_memory()
    signs = torch.zeros(m, dtype=torch.int8).pin_memory()
    offsets = torch.tensor([0, m], dtype=torch.int64).pin_memory()
    rank = torch.zeros(1, dtype=torch.int32).pin_memory()
    csr = _capi.stc_forward_csr()
    csr.n, csr.m = 1, m
    csr.offsets = C.cast(offsets.data_ptr(), _capi.u64p)
    csr.edges = C.cast(edges.data_ptr(), _capi.u32p)
    csr.signs = C.cast(signs.data_ptr(), _capi.i8p)
    csr.rank = C.cast(rank.data_ptr(), _capi.u32p)
    stream, out = torch.cuda.Stream(), _capi.stc_counts()
    with stc.Context(0) as c:
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (760 << 20), dtype=torch.int8, device="cuda")
        try:
            o = c._opts(stream=stream.cuda_stream)
            rc = _capi.lib().stc_count_forward_csr(c._h, C.byref(csr), C.byref(o), C.byref(out))
            done = stream.query()
        finally:
            torch.cuda.synchronize()
            del fill
            torch.cuda.empty_cache()
        assert rc == _capi.STC_ERR_OUT_OF_MEMORY
        assert done
