"""How the latent decode kernel cuts contexts into chunks (the rule runs on the device; the library exports it for the host)."""
import ctypes as C

import numpy as np
import pytest

import candle_vllm_b200 as pkg

PLACES = 296                       # 148 SMs, two CTAs each


def _chunk(lens, heads, window=0):
    a = np.asarray(lens, np.uint32)
    return pkg.lib().mla_decode_chunk_tokens(a.ctypes.data_as(C.c_void_p), C.c_int32(len(lens)), C.c_int32(heads), C.c_int32(window), C.c_int32(PLACES))


@pytest.mark.parametrize("lens,heads", [
    ([20000] + [250] * 71, 128),                  # one long context among many short ones: in one piece it would be 625 tiles in a row
    ([20000] + [250] * 35, 128),                  # the same with every sequence on a place of its own
    ([20000] + [250] * 63, 64),
    ([280] * 128, 64),                            # 512 (sequence, head group) pairs on 296 places
    ([500] * 73, 128),
    ([4096] * 128, 16),                           # rounds enough
    ([16] * 32, 16), ([4096], 16), ([300] * 200, 16),
])
def test_short_chunks(lens, heads):
    assert _chunk(lens, heads) == 256


@pytest.mark.parametrize("lens,heads,window", [
    ([4096 - 40 * i for i in range(32)], 16, 0), ([4096 - 40 * i for i in range(32)], 32, 0), ([1000] * 36, 128, 0), ([200000], 16, 0),
    ([100000] * 32, 16, 4096),                    # a windowed row has its window to read, not its context
])
def test_one_round_where_it_pays(lens, heads, window):
    c, groups = _chunk(lens, heads, window), -(-heads // 16)
    seen = [min(n, window + 32) if window else n for n in lens]
    assert c > 256 and c % 32 == 0
    assert sum(-(-n // c) for n in seen) * groups <= 1.05 * PLACES        # a round, or a little more (contexts of one length can all end just past a chunk)
    assert min(c, max(seen)) * PLACES <= 1.45 * sum(seen) * groups        # no chunk far above the even share
