"""The benchmark prints counters of a capture only beside the launch shape they were captured on."""
import bench


def test_counters_belong_to_a_shape():
    for (n, variant, rows), c in bench.NCU_CAPTURES.items():
        assert bench.captured(n, (variant, rows)) is c
        assert bench.captured(n, (variant, rows + 1)) == {} and bench.captured(n + 1, (variant, rows)) == {}
        assert 2 * c["traffic"] < 1.1 * n * n * bench.BYTES_PER_CELL  # the reads: half the step's bytes
    assert bench.captured(1024, (3, 16)) == {}
