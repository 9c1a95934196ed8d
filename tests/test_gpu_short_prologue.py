"""The one-launch prologue of short calls against the oracle, bit for bit: cluster sizes from one CTA
to the largest, ragged and full last tiles, grouped heads, narrow heads, options, and the sizes
next to which the launch gives way to the three-launch form."""
import pytest
import torch

from oracle import ref_numerics as R
from sageattention import b200_backend as be
from test_gpu_prologue import _check_against

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("smooth_k", [True, False])
@pytest.mark.parametrize("b,h,n", [(1, 1, 1), (2, 3, 127), (1, 2, 128), (1, 3, 129), (1, 2, 1000), (2, 2, 1025),
                                   (1, 1, 2048), (1, 1, 2049), (1, 150, 500), (2, 240, 100), (3, 165, 100), (1, 500, 100)])
def test_bytes_and_scales(b, h, n, smooth_k, dtype):
    q, k, v = R.make_inputs(b, h, n, 128, dtype, seed=n + h, k_bias_std=0.5)
    v[:, :, : n // 2] *= 600.0                                  # V scales above one: S is not its floor
    ref = R.prologue(q, k, v, smooth_k=smooth_k, pad_multiple=128)
    pq = be.quant_qkv(q.cuda(), k.cuda(), v.cuda(), smooth_k=smooth_k)
    torch.cuda.synchronize()
    _check_against(pq, ref, n, smooth_k)
    # Which form ran: the one-launch form leaves the number of its tiles in the work counter, the
    # persistent quantiser has drawn that many, the fold items and one item more per CTA.
    tiles = 3 * b * h * ((n + 127) // 128)
    counter = pq["ctrl"].view(torch.int32)[4 * b * h + 2].item()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    short = n <= 16 * 128 and (tiles + 1) // 2 <= 5 * sms        # K and V tiles share a CTA, and Q tiles in twos
    assert counter == tiles if short else counter > tiles


@pytest.mark.parametrize("hq,hkv,nq,nk,d,lse,smooth_v", [
    (4, 2, 300, 700, 128, True, False),      # Q tiles follow in a launch of their own
    (6, 3, 64, 1500, 64, False, True),       # two means
    (2, 1, 1000, 40, 96, True, True),
])
def test_whole_calls(hq, hkv, nq, nk, d, lse, smooth_v):
    g = torch.Generator().manual_seed(nq)
    q, k, v = (torch.randn(2, h, n, d, generator=g).half() for h, n in ((hq, nq), (hkv, nk), (hkv, nk)))
    v = (v + 2.0 * torch.randn(1, hkv, 1, d, generator=g)).half() if smooth_v else v
    nhd = [t.transpose(1, 2).contiguous().cuda() for t in (q, k, v)]
    res = be.sage_call(*nhd, "NHD", return_lse=lse, smooth_v=smooth_v)
    out = (res[0] if lse else res).transpose(1, 2)
    torch.cuda.synchronize()
    want = R.sageattn_oracle(q, k, v, tile=128, return_lse=lse, smooth_v=smooth_v)
    assert R.rel_l1(out.cpu(), want[0] if lse else want) <= 5e-3        # the bound of every call against the oracle
    if lse:
        assert (res[1].cpu() - want[1].reshape(res[1].shape)).abs().max().item() <= 1e-3
