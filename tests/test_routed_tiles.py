"""Room for the routed experts' tiles of pairs (no GPU needed: the library's answers, and what its entry points refuse before they launch)."""

import ctypes

import pytest

from inference_engine_b200.kernels.build import build_part_library


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(str(build_part_library("routed")))


def _tiles(counts, most, align):
    """The pairs of the tiles that `routed_sort` makes of the experts' pairs."""
    out = []
    for c in counts:
        k, units = -(-c // most), -(-c // align)
        at = 0
        for j in range(k):
            size = units // k + (j < units % k)
            out.append(min(size * align, c - at * align))
            at += size
    return out


def test_tiles_of_experts_that_tokens_name_more_than_once_fit(lib):
    for tokens in [1, 7, 16, 17, 20, 62, 63, 64, 65, 66, 96, 97, 100, 128, 129, 255, 256, 257, 300, 2048]:
        most, align = lib.ie_routed_tiled_most(tokens), lib.ie_routed_tiled_align()
        few = tokens <= lib.ie_routed_tiled_few()
        for top in (1, 2, 4, 8):
            for experts in (1, 5, 32):
                pairs = tokens * top
                for counts in ([pairs], [pairs - 1, 1], [tokens] * top, [pairs // 2, pairs - pairs // 2]):
                    if len(counts) > experts:
                        continue
                    tiles = _tiles(counts, most, align)
                    assert sum(tiles) == pairs and max(tiles) <= most
                    assert len(tiles) <= lib.ie_routed_tc5_max_tiles(pairs, experts, most)
                    # a slot of the ring holds a tile's columns in halves of whole 32s (up to 320), an accumulator of the other kernel 64
                    assert most <= (64 if few else 320) and (tokens > 256 or most <= max(64, -(-tokens // 32) * 32))
        # an expert that no token names twice is one tile, as long as it fits
        assert _tiles([min(tokens, 320)], most, align) == [min(tokens, 320)]


def test_more_pairs_than_there_is_room_for_are_refused(lib):
    p, f = ctypes.c_void_p(16), ctypes.c_float
    invalid = 1  # cudaErrorInvalidValue
    for few, most, tokens in ((1, 65, 8), (1, 320, 64), (1, 64, 65), (0, 321, 300), (0, 0, 300)):
        assert lib.ie_routed_tiled_gate_up(p, p, p, p, p, p, 1, 4, few, most, 4, tokens, 640, 64, 64, f(0), 0, f(1), f(0), None, None) == invalid
        assert lib.ie_routed_tiled_down(p, p, p, p, p, p, p, 1, 4, few, most, 4, tokens, 640, 64, 64, None, None) == invalid
