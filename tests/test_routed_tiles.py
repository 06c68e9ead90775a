"""Room for the routed experts' tiles of pairs (no GPU needed: the library's answers, and what its entry points refuse before they launch)."""

import ctypes

import pytest
import torch

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


@pytest.mark.parametrize("experts,ff,hidden", [(3, 64, 128), (2, 72, 200), (1, 8, 8), (2, 128, 64)])
def test_where_an_experts_entries_lie(experts, ff, hidden):
    from inference_engine_b200.parts.routed import ExpertTiles

    g = torch.Generator().manual_seed(ff)
    gate_up, down = (torch.randn(*s, generator=g).bfloat16() for s in ((experts, 2, ff, hidden), (experts, hidden, ff)))
    tiles = ExpertTiles.of(gate_up, down)
    f, h, rows = -(-ff // 64), -(-hidden // 64), -(-hidden // 128)
    assert tiles.gate_up.shape == (experts, f, h, 128, 64) and tiles.down.shape == (experts, rows, f, 128, 64)
    plain = torch.zeros(experts, f, 64, 2, h * 64).bfloat16()  # [feature, gate or up, k]
    plain.view(experts, f * 64, 2, h * 64)[:, :ff, :, :hidden] = gate_up.transpose(1, 2)
    other = torch.zeros(experts, rows * 128, f * 64).bfloat16()
    other[:, :hidden, :ff] = down
    for r in range(128):
        for k in range(64):
            place = (k // 8 ^ r % 8) * 8 + k % 8
            assert torch.equal(tiles.gate_up[:, :, :, r, place], plain[:, :, r // 16 * 8 + r % 8, r // 8 % 2, k::64])
            assert torch.equal(tiles.down[:, :, :, r, place], other[:, r::128, k::64])


@pytest.mark.gpu
def test_loading_holds_one_experts_matrices_beside_the_tiles():
    from inference_engine_b200.parts.routed import RoutedExperts

    experts, ff, hidden = 24, 512, 1024
    part = RoutedExperts(router="r", expert_prefix="e", experts=experts, top=2, groups=1, keep_groups=1, hidden_size=hidden, intermediate_size=ff,
                         limit=None, alpha=1.0, up_offset=0.0, dtype=torch.bfloat16)
    tensors = {"r": torch.randn(experts, hidden, device="cuda").bfloat16()}
    for e in range(experts):
        tensors.update({f"e{e}.gate": torch.randn(ff, hidden, device="cuda").bfloat16(), f"e{e}.up": torch.randn(ff, hidden, device="cuda").bfloat16(),
                        f"e{e}.down": torch.randn(hidden, ff, device="cuda").bfloat16()})
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before, one = torch.cuda.memory_allocated(), 3 * ff * hidden * 2
    part.bind(tensors, None)
    assert part.tiles is not None and part.w_down is None
    # (the order of the pieces is as large as two thirds of an expert's matrices while it is made)
    assert torch.cuda.max_memory_allocated() - before < (experts + 3) * one
