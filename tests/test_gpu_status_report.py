"""A failed call's status word reaches a word of pinned host memory without a copy behind the call.
No wait is made to run out: the status word is set before the launch, so that every CTA of the
attention kernel leaves at once, as it does when an earlier one has reported a failure."""
import ctypes

import pytest
import torch

from sageattention import _native
from sageattention import b200_backend as be

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [1, 2])
@pytest.mark.parametrize("causal", [False, True])
def test_the_status_word_is_reported_to_the_host(shape, causal):
    lib = _native.load()
    b, h, n = 1, 2, 300
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(b, h, n, 128, generator=g, device="cuda").half() for _ in range(3))
    pq = be.quant_qkv(q, k, v)
    out = torch.full_like(q, 7.0)
    host = torch.zeros(1, dtype=torch.int32).pin_memory()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    st3 = _native.strides3(*out.stride()[:3])

    def launch():
        lib.sage_debug_tiles_per_cta(shape)
        try:
            rc = lib.sage_attn_fwd_reported(
                *(pq[x].data_ptr() for x in ("q8", "sq", "k8", "sk", "v8t", "svp", "S")), out.data_ptr(), None, None, None,
                b, h, h, n, n, pq["n_pad"], 128, st3, int(causal), 128 ** -0.5, 0, 0, status.data_ptr(), host.data_ptr(),
                torch.cuda.current_stream().cuda_stream)
        finally:
            lib.sage_debug_tiles_per_cta(0)
        assert rc == 0
        torch.cuda.synchronize()

    status.fill_(2)
    launch()
    assert host.item() == 2 and (out == 7.0).all()             # reported, nothing computed
    host.zero_()
    status.zero_()
    launch()
    assert host.item() == 0 and status.item() == 0 and torch.isfinite(out).all() and not (out == 7.0).any()


def test_a_failure_is_reported_once():
    """The host clears its word when it raises, possibly before the last CTAs of the failed call have
    started: those see the status word that the first ones left and do not report it again."""
    lib = _native.load()
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(1, 2, 300, 128, generator=g, device="cuda").half() for _ in range(3))
    pq = be.quant_qkv(q, k, v)
    out = torch.full_like(q, 7.0)
    host = torch.zeros(1, dtype=torch.int32).pin_memory()
    status = torch.full((1,), 2, dtype=torch.int32, device="cuda")
    for expected in (2, 0):                                    # the CTAs that come first, and those that come late
        host.zero_()
        assert lib.sage_attn_fwd_reported(
            *(pq[x].data_ptr() for x in ("q8", "sq", "k8", "sk", "v8t", "svp", "S")), out.data_ptr(), None, None, None,
            1, 2, 2, 300, 300, pq["n_pad"], 128, _native.strides3(*out.stride()[:3]), 0, 128 ** -0.5, 0, 0,
            status.data_ptr(), host.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert host.item() == expected
        assert status.item() == 2 | _native.SAGE_STATUS_REPORTED and (out == 7.0).all()


def test_status_host_must_be_aligned():
    lib = _native.load()
    buf = (ctypes.c_char * 4096)()
    p = ctypes.c_void_p((ctypes.addressof(buf) + 255) // 256 * 256)
    s3 = _native.strides3(1024, 512, 128)
    rc = lib.sage_attention_reported(p, p, p, p, None, p, 1 << 40, 1, 2, 2, 16, 16, 128, s3, s3, s3, s3, 0, -1, 0, 1, 0, 0.1,
                                     ctypes.c_void_p(p.value + 2), None)
    assert rc == _native.SAGE_E_ARG and b"status_host" in lib.sage_last_error()
