"""Which way an attention forward goes, by host arithmetic (no GPU: 148 SMs are assumed)."""
import ctypes as C
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lact_b200", "csrc", "lact_b200.cu")


def _ceil_div(a, b):
    return -(-a // b)


def _span():
    """The bound on an item's key tiles, as the source has it: a function of (queries, band)."""
    with open(SRC) as f:
        text = f.read()
    behind = re.search(r"int64_t swa_behind\(.*?\) \{ return (.*?); \}", text)
    span = re.search(r"const int64_t span = causal \? std::min<int64_t>(\(.*?\)) : ceil_div", text).group(1)
    return lambda l, band: min(*eval(span, {"l": l, "ceil_div": _ceil_div, "band": band, "behind": behind and eval(
        behind.group(1), {"ceil_div": _ceil_div, "swa_band": lambda *_: band, "l": l, "window": band})}))


def _key_tiles(l, band):
    """Key tiles of every pair of query tiles: those that hold a key which one of its queries sees."""
    return [_ceil_div(min(q0 + 256, l), 128) - max(q0 - (band - 1), 0) // 128 for q0 in range(0, l, 256)]


def test_no_item_has_more_key_tiles_than_it_is_given_room_for():
    span = _span()
    for l in [*range(1, 1200, 7), 1280, 1536, 2048, 2303, 2304, 2305, 4096, 8192]:
        for band in {1, 2, 127, 128, 129, 130, 255, 256, 257, 383, 384, 385, 1000, 1024, 1025, 2048, l} & set(range(1, l + 1)):
            most = max(_key_tiles(l, band))
            assert most <= span(l, band)
            if l >= band + 512 and l % 256 == 0:   # a pair past the sequence's start, with both tiles: no tile more
                assert most == span(l, band), (l, band)


def _scratch(b, l, lk, h, d, window):
    from lact_b200 import _lib, build
    build.build()
    need, words = C.c_size_t(0), C.c_int64(0)
    assert _lib.lib().lact_swa_fwd_split_bytes(b, l, lk, h, d, window, C.byref(need), C.byref(words)) == 0
    return need.value, words.value


# pairs, the last of them cut (the pieces take a second launch and no counters); single tiles, the last of them cut
@pytest.mark.parametrize("b,l,lk,h,d,window,pairs", [(1, 1560, 4680, 12, 128, -1, True), (1, 1300, 4500, 30, 64, -1, True),
                                                     (1, 2600, 2500, 14, 128, -1, True), (2, 1900, 2600, 10, 64, -1, True),
                                                     (1, 4680, 4681, 5, 128, -1, True), (1, 2305, 2305, 8, 128, 2048, False), (1, 100, 4581, 4, 128, -1, False),
                                                     (2, 300, 5384, 4, 64, -1, False), (1, 777, 2777, 8, 64, -1, False)])
def test_what_is_cut(b, l, lk, h, d, window, pairs):
    need, words = _scratch(b, l, lk, h, d, window)
    assert need > 0 and (words == 0) == pairs
