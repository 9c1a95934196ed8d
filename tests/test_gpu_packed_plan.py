"""The work list of a packed batch: orders, prefix sums and the searches in them, against one call
per sequence, bit for bit (the kernels quantise and attend every sequence on its own)."""
import random

import pytest
import torch

import sageattention
from sageattention import _native
from sageattention import b200_backend as be

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [0, 2])
@pytest.mark.parametrize("n_seq,hq,hkv,causal,longest", [
    (2, 3, 1, False, 1500), (33, 2, 2, True, 300), (64, 4, 2, False, 129),
    (512, 2, 1, False, 140), (513, 2, 1, True, 140),           # the longest list and the first batch without one
])
def test_work_list_against_single_calls(shape, n_seq, hq, hkv, causal, longest):
    rng = random.Random(n_seq)
    lens = [rng.choice([0, 1, 127, 128, 129, rng.randint(1, longest)]) for _ in range(n_seq)]
    lens = [min(n, longest) for n in lens]
    lens[rng.randrange(n_seq)] = longest
    total = sum(lens)
    g = torch.Generator(device="cuda").manual_seed(n_seq)
    q, k, v = (torch.randn(total, h, 128, generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    k += torch.randn(1, hkv, 128, generator=g, device="cuda").half()
    cu = torch.tensor([sum(lens[:i]) for i in range(n_seq + 1)], dtype=torch.int32, device="cuda")
    _native.load().sage_debug_tiles_per_cta(shape)             # 2: pairs of query tiles
    try:
        out = sageattention.sageattn_varlen(q, k, v, cu, cu, longest, longest, is_causal=causal)
    finally:
        _native.load().sage_debug_tiles_per_cta(0)
    torch.cuda.synchronize()
    be.check()
    at = 0
    for n in lens:
        if n:
            one = be.sage_call(q[None, at:at + n], k[None, at:at + n], v[None, at:at + n], "NHD", causal)
            assert torch.equal(out[at:at + n], one[0]), (at, n)
        at += n
