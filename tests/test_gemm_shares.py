"""How the CTA pairs share an accumulation (host rule of the GEMM library, no GPU needed)."""
import ctypes

import pytest

from allie_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib.have_cuda_lib(), reason="kernel library not built")


@pytest.mark.parametrize("pairs", [1, 2, 7, 37, 73, 74])
def test_shares_cover_every_step_once(pairs):
    """Every step of every output tile in one unit, and nobody with more than the busiest of equal parts has."""
    room = 4096
    buf, lib, shared = (ctypes.c_int * (4 * room))(), _lib.cuda(), 0
    for tiles in list(range(1, 80)) + [100, 150, 256, 301]:
        for steps in (1, 7, 8, 9, 33, 64, 190, 256, 512):
            n = lib.ab_gemm_even_units(tiles, steps, pairs, buf, room)
            if n < 0:                       # equal parts, the kernel's other way
                assert 1 <= -n <= 32
                continue
            assert 0 < n <= room
            shared += 1
            seen, load = [[0] * steps for _ in range(tiles)], [0] * pairs
            for u in range(n):
                pair, tile, kb0, kb1 = buf[4 * u:4 * u + 4]
                assert 0 <= pair < pairs and 0 <= kb0 < kb1 <= steps
                load[pair] += kb1 - kb0
                for k in range(kb0, kb1):
                    seen[tile][k] += 1
            assert all(c == 1 for row in seen for c in row), (tiles, steps)
            whole_rounds = -(-tiles // pairs) * steps
            assert max(load) <= whole_rounds, (tiles, steps)
    assert pairs <= 2 or shared > 50
