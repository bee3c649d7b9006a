"""The bytes that bench.py charges each pass are no more than the kernels move (CPU only)."""
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench


def test_bytes_of_the_record_are_charged_where_they_move():
    fi = {"near_pass": 900, "visible": 500, "sorted_count": 7000, "tiles_x": 10, "tiles_y": 6}
    b = bench.algorithmic_bytes(fi, 1000, 160 * 90, 4)
    # positions and counts of all, the other 56 attributes and 48 B of the record of those in front of the near
    # plane; its last 16 B (the cull extents) and the tile rectangle only of the visible ones
    assert b["preprocess"] == 1000 * (12 + 4) + 900 * (224 + 48) + 500 * (16 + 16)
    # every instance's index, centre and extents; the rest of a record only where a block is met
    assert b["raster"] == 7000 * (4 + 8 + 16) + 60 * 16 + 160 * 90 * 4
