"""Conversion of several arrays in one launch, against torch's own conversion."""
import ctypes as C

import pytest
import torch

from megafold_b200 import _lib

pytestmark = pytest.mark.gpu
DTYPES = (torch.float32, torch.bfloat16, torch.float16)


@pytest.mark.parametrize("sizes", [(1,), (7, 2048, 2049), (8, 1, 4095, 4096, 100003, 3, 2047, 64)])
@pytest.mark.parametrize("offset", [0, 1])          # 1: neither end is 16-byte aligned
def test_cast_batch(sizes, offset):
    g = torch.Generator(device="cuda").manual_seed(sum(sizes))
    items = (_lib.CastItem * len(sizes))()
    pairs = []
    for i, n in enumerate(sizes):
        src = (torch.randn(n + offset, device="cuda", generator=g) * 10).to(DTYPES[i % 3])[offset:]
        dst = torch.zeros(n + offset, device="cuda", dtype=DTYPES[(i // 3 + i + 1) % 3])[offset:]
        items[i].src, items[i].dst, items[i].n = src.data_ptr(), dst.data_ptr(), n
        items[i].src_dtype, items[i].dst_dtype = _lib.dtype_code(src.dtype), _lib.dtype_code(dst.dtype)
        pairs.append((src, dst))
    _lib.check(_lib.lib().mf_cast_batch(items, len(sizes), _lib.stream_ptr("cuda")), "mf_cast_batch")
    for src, dst in pairs:
        assert torch.equal(dst, src.to(dst.dtype))
    assert _lib.lib().mf_cast_batch(items, 9, None) == -1           # more than MF_CAST_MAX
