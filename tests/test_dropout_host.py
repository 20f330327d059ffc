"""The dropout generator as the host compiles it (no GPU needed)."""
import ctypes

import pytest

from allie_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib.have_cuda_lib(), reason="kernel library not built")


def _draws(seed: int, stream: int, group: int) -> list[int]:
    """Philox4x32 with seven rounds (Salmon et al. 2011): sixteen bits for each of a group's eight elements."""
    c = [group & 0xffffffff, group >> 32, stream, 0x9E3779B9]
    k = [seed & 0xffffffff, seed >> 32]
    for _ in range(7):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(p1 >> 32) ^ c[1] ^ k[0], p1 & 0xffffffff, (p0 >> 32) ^ c[3] ^ k[1], p0 & 0xffffffff]
        k = [(k[0] + 0x9E3779B9) & 0xffffffff, (k[1] + 0xBB67AE85) & 0xffffffff]
    return [c[j // 2] >> (16 * (j % 2)) & 0xffff for j in range(8)]


@pytest.mark.parametrize("thr16", [0, 1, 6554, 32768, 65535, 65536])
def test_an_element_is_kept_where_its_draw_reaches_the_threshold(thr16):
    seed, stream, groups = 0x123456789ABCDEF, 7, 4096
    out = (ctypes.c_ubyte * (8 * groups))()
    assert _lib.cuda().ab_dropout_mask_host(ctypes.c_ulonglong(seed), ctypes.c_uint(stream), ctypes.c_longlong(8 * groups),
                                            ctypes.c_uint(thr16), out) == 0
    assert list(out) == [int(x >= thr16) for g in range(groups) for x in _draws(seed, stream, g)]
