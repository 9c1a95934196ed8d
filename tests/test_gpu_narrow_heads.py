"""Heads of up to 64 columns leave the zero columns out of both products; the zeros add nothing, so
the call equals the one on rows padded with zeros to 128 columns bit for bit."""
import pytest
import torch

from sageattention import _native
from sageattention import b200_backend as be

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [1, 2])
@pytest.mark.parametrize("d,dtype,causal,int8,smooth_v", [
    (8, torch.float16, False, None, False), (40, torch.bfloat16, True, None, True), (64, torch.float16, True, None, False),
    (64, torch.float16, False, False, True), (64, torch.bfloat16, False, None, False), (72, torch.float16, False, None, False),
])
def test_equals_zero_padded_rows(shape, d, dtype, causal, int8, smooth_v):
    lib = _native.load()
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn(2, h, 1155, d, generator=g, device="cuda").to(dtype) for h in (4, 2, 2))
    v += 2.0
    pad = lambda t: torch.nn.functional.pad(t, (0, 128 - d))
    kw = dict(is_causal=causal, int8=int8, smooth_v=smooth_v, sm_scale=d ** -0.5, return_lse=True)
    lib.sage_debug_skip_threshold(0.0)                         # the kernels without the negligible-tile tests
    lib.sage_debug_tiles_per_cta(shape)
    try:
        out, lse = be.sage_call(q, k, v, **kw)
        wide, wide_lse = be.sage_call(pad(q), pad(k), pad(v), **kw)
    finally:
        lib.sage_debug_tiles_per_cta(0)
        lib.sage_debug_skip_threshold(-1.0)
    torch.cuda.synchronize()
    assert be.last_status(q, 2, 4, 1155, 2, 1155) == 0
    assert torch.equal(out, wide[..., :d]) and torch.equal(lse, wide_lse)
