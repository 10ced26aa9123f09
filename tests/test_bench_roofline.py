"""The benchmark's roofline entry: bytes that one kernel reads for many queries count once, so the share
of the HBM rate stays a share; without a batched Start the per-query scan is the kernel named."""
import bench

STATS = {"bytes_by_phase": {"top_level": 20_495_728_000, "start": 12_893_805_568, "warmup": 4_895_000_000,
                            "survivor_horizontal": 80_000_000, "survivor_vertical": 1_000_000, "probe": 0}}
# a batch of 10,000 queries that start in 860 of 1,000 clusters of about 1,000 x 1024 bytes
UNIQUE = {"start_rows": 1_020_000_000, "first_checkpoint_rows": 15_900_000}


def test_batched_start_reads_a_cluster_once():
    r = bench.roofline(STATS, UNIQUE, {"start": 0.29, "search_kernel": 0.344}, 1024, 1, 6537.3, "measured")
    assert r["algorithmic_bytes_per_launch"] == 1_020_000_000 + 12_893_805_568 // 1024 * 4
    assert 0.5 < r["frac"] < 0.6 and "start_dist" in r["kernel"] and r["kernel_ms"] == 0.29
    assert r["per_query_bytes"]["start"] == 12_893_805_568


def test_f32_distances_are_counted_per_vector():
    r = bench.roofline(STATS, UNIQUE, {"start": 0.29, "search_kernel": 0.344}, 1024, 4, 6537.3, "measured")
    assert r["algorithmic_bytes_per_launch"] == 1_020_000_000 + 12_893_805_568 // 4096 * 4


def test_without_a_batched_start():
    r = bench.roofline(STATS, None, {"start": 0.0, "search_kernel": 3.7}, 1024, 1, 6537.3, "measured")
    assert r["kernel"] == "search_kernel" and r["algorithmic_bytes_per_launch"] == 17_869_805_568
