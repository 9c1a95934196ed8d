"""Calls with few queries split their keys over CTAs and merge the shares; grouped heads of calls
without a causal mask share query tiles.  A share starts from the running maxima of the keys before
it, so P has the codes of one walk over all keys and a split call differs from the unsplit kernel
only by the order of fp32 sums (2^-24 each, below 1e-5 of the result) and the rounding of the output
to 16 bits (2^-11 or 2^-8 of a value: one step where the sums straddle a boundary)."""
import pytest
import torch

from oracle import ref_numerics as R
from sageattention import _native
from sageattention import b200_backend as be
from test_call_forms import form

pytestmark = pytest.mark.gpu


def _inputs(b, hq, hkv, nq, nk, d, dtype, layout="HND"):
    g = torch.Generator(device="cuda").manual_seed(nq * 7 + nk)
    mk = lambda h, n: torch.randn(b, h, n, d, generator=g, device="cuda")
    q, k, v = mk(hq, nq), mk(hkv, nk) + 0.5 * torch.randn(1, hkv, 1, d, generator=g, device="cuda"), mk(hkv, nk)
    q, k, v = (t.to(dtype) for t in (q, k, v))
    return tuple(t.transpose(1, 2).contiguous() for t in (q, k, v)) if layout == "NHD" else (q, k, v)


@pytest.mark.parametrize("b,hq,hkv,nq,nk,d,dtype,layout,smooth_v,splits", [
    (1, 1, 1, 1, 3072, 128, torch.float16, "HND", False, True),      # one row, the shortest key range that it splits
    (2, 8, 2, 4, 16384, 128, torch.float16, "HND", False, True),     # folded heads, many shares
    (1, 4, 1, 33, 3073, 128, torch.bfloat16, "NHD", False, True),    # folded rows in two tiles; one key in the last tile
    (1, 12, 4, 128, 5000, 96, torch.bfloat16, "NHD", True, True),    # narrow heads, smooth_v, ragged shares
    (3, 5, 5, 128, 4321, 64, torch.float16, "HND", True, True),
    (1, 37, 37, 32, 2304, 128, torch.float16, "HND", False, True),   # two shares
    (1, 98, 98, 17, 4100, 128, torch.bfloat16, "HND", False, True),  # three shares, two CTAs to an SM
    (1, 1, 1, 1, 2048, 128, torch.float16, "HND", False, False),     # sizes at which one pass is faster
    (1, 4, 1, 33, 2049, 128, torch.bfloat16, "NHD", False, False),
    (1, 147, 147, 17, 2300, 128, torch.float16, "HND", False, False),
])
def test_split_keys(b, hq, hkv, nq, nk, d, dtype, layout, smooth_v, splits):
    lib = _native.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (form(b, hq, hkv, nq, nk, sms=sms)[1] > 1) == splits
    q, k, v = _inputs(b, hq, hkv, nq, nk, d, dtype, layout)
    kw = dict(tensor_layout=layout, return_lse=True, smooth_v=smooth_v)
    out, lse = be.sage_call(q, k, v, **kw)
    torch.cuda.synchronize()
    assert be.last_status(q, b, hq, nq, hkv, nk) == 0
    lib.sage_debug_tiles_per_cta(1)                            # a forced shape never splits
    try:
        one, one_lse = be.sage_call(q, k, v, **kw)
    finally:
        lib.sage_debug_tiles_per_cta(0)
    hnd = (lambda t: t.transpose(1, 2)) if layout == "NHD" else (lambda t: t)
    want = R.sdpa_fp32(hnd(q), hnd(k), hnd(v))
    out, one = hnd(out).float(), hnd(one).float()
    step = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    assert ((out - one).abs() <= step * one.abs() + 1e-4 * one.std()).all()
    assert R.rel_l1(out, one) <= step / 8
    assert R.rel_rms(out, want) <= 1.001 * R.rel_rms(one, want)
    # natural-log sums of about nk terms: fp32 sums in another order, 2^-24 x a few of their size
    assert (lse - one_lse).abs().max().item() <= 4e-6 * one_lse.abs().max().item() + 4e-6


def _close(out, one, dtype):
    """The stated distance of two calls that split the keys differently (see the top of the file)."""
    step = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    out, one = out.float(), one.float()
    assert ((out - one).abs() <= step * one.abs() + 1e-4 * one.std()).all()
    assert R.rel_l1(out, one) <= step / 8


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_packed_batch_against_calls_that_split(dtype):
    """A packed batch never splits: its sequences equal the unsplit calls bit for bit, and the calls
    that a program would make, which split, up to the order of fp32 sums."""
    lib = _native.load()
    hq, hkv, nq, nk = 4, 2, (4, 128, 1, 60), (4200, 5000, 4097, 4500)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert all(form(1, hq, hkv, a, b, sms=sms)[1] > 1 for a, b in zip(nq, nk))
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(sum(n), h, 128, generator=g, device="cuda").to(dtype) for n, h in ((nq, hq), (nk, hkv), (nk, hkv)))
    cu = lambda n: torch.tensor([sum(n[:i]) for i in range(len(n) + 1)], dtype=torch.int32, device="cuda")
    out = be.sage_call_varlen(q, k, v, cu(nq), cu(nk), max(nq), max(nk))
    a = b = 0
    for n, m in zip(nq, nk):
        args = (q[None, a:a + n], k[None, b:b + m], v[None, b:b + m], "NHD")
        lib.sage_debug_tiles_per_cta(1)                        # a forced shape never splits
        try:
            assert torch.equal(out[a:a + n], be.sage_call(*args)[0])
        finally:
            lib.sage_debug_tiles_per_cta(0)
        _close(be.sage_call(*args)[0], out[a:a + n], dtype)
        a, b = a + n, b + m


def test_units_of_a_split_call_one_by_one():
    """The number of shares follows from the number of (batch, K/V head) units, so a unit computed
    alone agrees with the whole call up to the order of fp32 sums."""
    b, hq, hkv, nq, nk = 2, 80, 40, 8, 6000
    q, k, v = _inputs(b, hq, hkv, nq, nk, 128, torch.float16)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert form(b, hq, hkv, nq, nk, sms=sms)[1] != form(1, 2, 1, nq, nk, sms=sms)[1]
    whole = be.sage_call(q, k, v)
    for i, h in ((0, 0), (0, 39), (1, 17)):
        one = be.sage_call(q[i:i + 1, 2 * h:2 * h + 2], k[i:i + 1, h:h + 1], v[i:i + 1, h:h + 1])
        _close(one, whole[i:i + 1, 2 * h:2 * h + 2], torch.float16)


def test_a_workspace_without_the_scratch_is_still_accepted():
    """The C entry point takes a workspace that only lacks the shares' scratch, and does not split."""
    lib = _native.load()
    b, hq, hkv, nq, nk = 1, 4, 2, 8, 4096
    q, k, v = _inputs(b, hq, hkv, nq, nk, 128, torch.float16)
    shares = min(2 * 160 // (b * hkv), nk // 128 // 8)
    scratch = (shares * b * hq * nq * 524 + 255) // 256 * 256      # 131 floats per row and share
    ws = torch.empty(lib.sage_workspace_bytes_ex(b, hq, hkv, nq, nk) - scratch, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(q)
    st3 = lambda t: _native.strides3(*t.stride()[:3])
    args = lambda w: (q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, w.data_ptr(), w.numel(), b, hq, hkv,
                      nq, nk, 128, st3(q), st3(k), st3(v), st3(out), 0, -1, 0, 1, 0, 128 ** -0.5,
                      torch.cuda.current_stream().cuda_stream)
    assert lib.sage_attention_ex(*args(ws)) == 0
    lib.sage_debug_tiles_per_cta(1)
    try:
        one = be.sage_call(q, k, v)
    finally:
        lib.sage_debug_tiles_per_cta(0)
    torch.cuda.synchronize()
    assert torch.equal(out, one)
    assert lib.sage_attention_ex(*args(ws[:-512])) == _native.SAGE_E_WORKSPACE


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hq,hkv,nq,nk", [(4, 4, 288, 288), (4, 2, 16, 300), (8, 1, 17, 515), (6, 2, 129, 1000), (2, 2, 1, 1)])
def test_mostly_empty_query_tiles(dtype, hq, hkv, nq, nk):
    """Folding heads and leaving out warps without rows does not change a row: the call equals the
    one on the kernels that do neither (a forced shape), bit for bit."""
    lib = _native.load()
    q, k, v = _inputs(2, hq, hkv, nq, nk, 96, dtype)
    rep = lambda t: t.repeat_interleave(hq // hkv, 1)
    lib.sage_debug_skip_threshold(0.0)                         # the kernels without the negligible-tile tests
    try:
        a, la = be.sage_call(q, k, v, return_lse=True)
        lib.sage_debug_tiles_per_cta(2)
        c, lc = be.sage_call(q, rep(k), rep(v), return_lse=True)
    finally:
        lib.sage_debug_tiles_per_cta(0)
        lib.sage_debug_skip_threshold(-1.0)
    assert torch.equal(a, c) and torch.equal(la, lc)
    out = torch.empty_like(q.transpose(1, 2)).transpose(1, 2)  # another layout of the output
    lib.sage_debug_skip_threshold(0.0)
    try:
        be.sage_call(q, k, v, out=out)
    finally:
        lib.sage_debug_skip_threshold(-1.0)
    assert torch.equal(out, a)
