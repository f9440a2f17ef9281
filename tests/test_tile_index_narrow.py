"""The CPU check of the x-pair tile's index arithmetic (test_tile_index) for the
shape that only single grids use: 16x32."""
import test_tile_index as t


def test_halo_builds_cover_every_read_once():
    t.test_halo_builds_cover_every_read_once(16, 32)


def test_tma_boxes_start_on_16_bytes():
    t.test_tma_boxes_start_on_16_bytes(16, 32)
