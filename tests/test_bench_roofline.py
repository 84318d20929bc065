"""CPU: the launches and traffic of the bench's roofline entries."""
import bench


def test_roofline_counts_no_launches_it_does_not_know():
    r = bench.roofline("stage", 1.0, 1000, 10.0, 1, 1, 6545.3, 34.0, 72.0, 100.0)
    assert r["launches_per_step"] is None and r["traffic"] == 100000 and r["traffic_scope"] == "step"
    r = bench.roofline("evaluation", 1.0, 1000, 10.0, 1, 1, 6545.3, 34.0, 72.0, 100.0, 75)
    assert r["launches_per_step"] == 75 and r["traffic"] == 100000
