"""Which form of the attention kernel a call takes: `sage_attention_form` is the function the launch asks."""
import ctypes

import pytest

from sageattention import _native


def form(b, hq, hkv, nq, nk, packed_q=0, causal=0, plain=1, sms=148):
    out = (ctypes.c_int * 4)()
    assert _native.load().sage_attention_form(b, hq, hkv, nq, nk, packed_q, causal, plain, sms, out) == 4
    return tuple(out)                      # query tiles per CTA, shares of the keys, folded heads, tests


@pytest.mark.parametrize("call,want", [
    ((1, 48, 48, 47520, 47520), (2, 1, 1, 0)),       # the headline call
    ((1, 48, 48, 4096, 4096), (1, 1, 1, 0)),
    # up to eight key tiles: one query tile per CTA, whatever the rounds rule says of the queries
    ((1, 48, 48, 288, 288), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 512), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 1024), (1, 1, 1, 0)),
    ((1, 40, 40, 16384, 1025), (2, 1, 1, 0)),
    # heads of a group share query tiles where those are mostly empty
    ((2, 8, 2, 4, 300), (1, 1, 4, 0)),
    ((1, 8, 2, 128, 300), (1, 1, 1, 0)),             # full tiles
])
def test_fixed_length_calls(call, want):
    assert form(*call) == want


def test_negligible_tile_tests():
    assert form(1, 48, 48, 4096, 4096, plain=0)[3] == 1
    assert form(1, 48, 48, 4096, 1024, plain=0)[3] == 0              # short key loops have none
    assert form(4, 48, 48, 4096, 4096, packed_q=9000, plain=0)[3] == 0
    assert form(1, 48, 48, 4096, 4096, causal=1, plain=0)[3] == 1


@pytest.mark.parametrize("n_seq,longest,tokens,heads,causal,keys,tiles", [
    # batches on which both shapes were timed on a 148-SM part, whole call, one / two tiles per CTA in us
    (64, 128, 64 * 128, 92, 0, 128, 1),              # 430 / 626: the second tile of every CTA would be empty
    (128, 300, 128 * 300, 20, 0, 300, 1),            # 603 / 754
    (32, 512, 32 * 512, 46, 0, 512, 1),              # 491 / 532
    (16, 1024, 16 * 1024, 46, 0, 1024, 1),           # 644 / 680
    (12, 1200, 12 * 1200, 53, 0, 1200, 1),           # 789 / 830
    (16, 2000, 8944, 96, 0, 2000, 1),                # 887 / 940: ragged, 559 tokens on average
    (8, 3100, 8 * 3100, 48, 0, 3100, 1),             # 2280 / 2283: 25 tiles each
    (6, 3300, 6 * 3300, 40, 0, 3300, 2),             # 1554 / 1521: 26 tiles each
    (11, 8192, 36124, 48, 0, 8192, 2),               # 4364 / 4276
    (8, 6000, 22496, 48, 0, 6000, 2),                # 2826 / 2783
    (16, 8192, 37280, 48, 0, 8192, 2),               # 3880 / 3802
    (16, 4000, 22976, 48, 0, 4000, 1),               # 1730 / 1718, 1648 / 1694 in bursts: ragged, 1 436 on average
    (2, 8192, 2 * 8192, 48, 0, 8192, 2),             # 3155 / 3025
    (5, 8192, 26705, 32, 0, 8192, 2),                # 2682 / 2616
    (3, 8192, 3 * 8192, 8, 0, 8192, 1),              # 792 / 831: five rounds
    (11, 8192, 36124, 48, 1, 8192, 1),               # 2674 / 2723
    (4, 8192, 16792, 48, 1, 8192, 1),                # 1697 / 1696
    (2, 8192, 2 * 8192, 48, 1, 8192, 2),             # 1837 / 1810
    (2, 8192, 2 * 8192, 48, 0, 1024, 1),             # short key loops take one tile as in every other call
])
def test_packed_batches(n_seq, longest, tokens, heads, causal, keys, tiles):
    assert form(n_seq, heads, heads, longest, keys, packed_q=tokens, causal=causal) == (tiles, 1, 1, 0)


def test_packed_batches_without_a_work_list_take_one_tile():
    assert form(512, 96, 96, 8192, 8192, packed_q=512 * 8192)[0] == 2
    assert form(513, 96, 96, 8192, 8192, packed_q=513 * 8192)[0] == 1


@pytest.mark.parametrize("units,tiles,rows,shares", [
    # calls timed both ways on a 148-SM part: whole call, split / one pass over the keys, in us
    (1, 32, 4, 4), (74, 32, 128, 4), (50, 32, 128, 4), (16, 128, 128, 16), (37, 40, 64, 5),      # all gain
    (98, 32, 16, 3),          # 129.5 / 133.8
    (80, 32, 32, 3),          # 119.0 / 129.1
    (49, 24, 128, 3),         # 77.9 / 82.8
    (64, 24, 128, 1),         # 98.0 / 92.9
    (75, 32, 128, 1),         # 129.9 / 126.1
    (96, 32, 128, 1),         # 146.9 / 139.9
    (80, 48, 96, 3),          # 175.2 / 179.6
    (96, 48, 128, 1),         # 197.8 / 195.5
    (96, 96, 128, 3),         # 351.8 / 360.0
    (128, 16, 4, 1),          # 95.2 / 89.6
    (16, 16, 4, 1),           # 39.0 / 37.7
    (100, 16, 128, 1),        # 101.5 / 83.3
    (100, 64, 128, 1),        # 287.5 / 259.9
    (147, 128, 128, 1),       # 684 / 636
    (37, 18, 32, 2),          # 58.4 / 61.3
    (147, 16, 32, 1),
    (99, 128, 32, 2),         # 467.4 / 487.8
    (110, 256, 4, 2),         # 929 / 945
    (148, 256, 4, 1),         # a unit for every SM
    (16, 15, 4, 1),
])
def test_shares_of_the_keys(units, tiles, rows, shares):
    assert form(1, units, units, rows, tiles * 128)[1] == shares
    if rows % 4 == 0:         # the rows of a K/V head count, whether they are queries or heads of its group
        assert form(1, 4 * units, units, rows // 4, tiles * 128)[1] == shares


def test_the_workspace_holds_the_shares_of_every_device():
    """Its size is fixed without a device; no SM count up to the one it is sized for needs more."""
    lib = _native.load()
    offs = (ctypes.c_size_t * 13)()
    for units in (1, 7, 36, 48, 49, 53, 54, 64, 74, 80, 96, 100, 120, 147, 159):
        for nq in (1, 16, 17, 32, 33, 96, 97, 128):
            for tiles in (16, 23, 24, 31, 32, 47, 48, 96, 128, 256):
                nk = 128 * tiles - 5
                assert lib.sage_workspace_layout_ex(1, units, units, nq, nk, offs) == 13
                room = lib.sage_workspace_bytes_ex(1, units, units, nq, nk) - (offs[12] + units * 512)
                for sms in (64, 100, 132, 144, 148, 152, 160, 200):
                    n = form(1, units, units, nq, nk, sms=sms)[1]
                    assert n == 1 or n * units * nq * 131 * 4 <= room, (units, nq, tiles, sms)


def test_bad_arguments():
    out = (ctypes.c_int * 4)()
    f = _native.load().sage_attention_form
    assert f(1, 3, 2, 8, 8, 0, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 0, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, -1, 0, 0, 148, out) == _native.SAGE_E_ARG
    assert f(1, 2, 2, 8, 8, 0, 0, 0, 148, None) == _native.SAGE_E_ARG
